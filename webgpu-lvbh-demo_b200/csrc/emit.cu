// emit.cu - K3: radix tree emission, leaf gather, triangle rearrange and bottom-up refit
// (sm_100a).
//
// Produces what the reference computes in three kernels: compute_radix_tree_pointers
// (scripts/bvh/kernels/radix-tree.js:137-238, parent links), bvh_upward_pass
// (scripts/bvh/kernels/bvh-up-pass.js:200-280, node boxes and child links) and
// rearrange_triangles (scripts/bvh/kernels/rearrange.js:162-169).
//
// Tree.  With d[k] = delta(k, k+1) (common-prefix length of adjacent sorted keys, index
// tie-break, -1 past either end), the Karras radix tree is the Cartesian tree of d: the node
// whose split is s covers [L, R], where L-1 and R are the nearest positions left and right of
// s with a smaller d.  A node [L, R] is the LEFT child of split R when d[R] > d[L-1], else the
// RIGHT child of split L-1 (adjacent d values always differ), so its Karras index is R or L
// (0 for the root) - exactly the numbering compute_child_index produces - and its parent
// follows from its own range alone; its parent is the node of the larger of the two separators
// around it.  So every node is found on its own thread from the separators, with its box as the
// union of a range of leaves: no per-node binary search and no climb from child to parent.
//
// Passes.
//   K3b (k_tree_climb)   blocks of 256 sorted leaves in shared memory, a persistent grid that
//                        prefetches the next blocks: leaf k's triangle perm[k] arrives with
//                        three others by one TMA gather of four 48-byte rows, goes to the
//                        output soup at k and is reduced to its box (exact-zero components
//                        nudged by 1e-8 as bvh-up-pass.js:209-210 does).  Then the nodes that lie
//                        in the block, one thread each.  A subtree whose parent crosses the
//                        block's edge leaves as an "open item" (at most 2 x 64 per block: they
//                        hang off the two boundary paths of a tree at most 64 deep).
//   K3c (k_top_group)    the nodes that straddle blocks (~3 % of them), from the open items: per
//                        group of blocks in shared memory, each node on its own thread, then per
//                        group of groups, up to the root (see below).
#include <cstddef>
#include <cstring>
#include <cuda.h>  // CUtensorMap
#include <cudaTypedefs.h>
#include <type_traits>

#include "lvbh_device.cuh"
#include "lvbh_internal.h"

namespace lvbh {

namespace {

// Tree-pass geometry: blocks of 2^LOG sorted leaves (one thread each), resident CTAs per SM
// of the persistent grid.  The plain build uses LOG = 8; a batched build may pick LOG = 7.
template <int LOG>
struct TreeGeo {
    static constexpr int EB = 1 << LOG;
    static constexpr int kCtasPerSm = LOG == 8 ? 4 : 8;
};

// Where a block of EB sorted leaves lives.  A batched build is a list of segments (meshes)
// laid end to end; every block lies inside one segment and every index a kernel works with
// is local to that segment (the plain build is the one-segment case).
struct Span {
    size_t start;  // the segment's first position in the batch
    int n;         // the segment's triangle count
    int b0;        // the block's first leaf within the segment
};

template <int LOG>
struct OneSeg {
    static constexpr int EB = 1 << LOG;
    int n;
    __device__ __forceinline__ int blocks() const { return (n + EB - 1) / EB; }
    __device__ __forceinline__ Span span(int blk) const { return Span{0, n, blk * EB}; }
};

template <int LOG>
struct ManySegs {
    static constexpr int EB = 1 << LOG;
    const SegRow *rows;       // num_segs + 1 rows
    const uint32_t *blk_seg;  // segment of each block
    int nblk;
    __device__ __forceinline__ int blocks() const { return nblk; }
    __device__ __forceinline__ Span span(int blk) const {
        const uint32_t sg = __ldg(blk_seg + blk);
        const uint32_t t0 = __ldg(&rows[sg].tri), t1 = __ldg(&rows[sg + 1].tri);
        const int first = (int)__ldg(&rows[sg].blk);
        return Span{t0, (int)(t1 - t0), (blk - first) * EB};
    }
};

// Where the tree pass gets its leaves.  SoupLeaves: leaf t of a block is triangle perm[b0 + t]
// of the 48-byte soup, copied to the output soup.  MeshLeaves (the indexed leaf format): leaf t
// is the sorted triangle b0 + t, whose three vertex indices are already in sorted order
// (sidx, written by the leaf-index pass) and whose vertices are 16-byte rows of a vertex
// buffer; nothing is copied.
struct SoupLeaves {
    static constexpr bool kMesh = false;
    const float4 *tri;
    const uint32_t *perm;
    float4 *otri;
};
struct MeshLeaves {
    static constexpr bool kMesh = true;
    const float4 *verts;
    const uint32_t *sidx;
    uint32_t nverts;
};

// K3b shared memory.
//
// slot: the gathered triangles of this block and the next: buffer b holds leaves 4g .. 4g + 3 in
// slot[b][g], four 48-byte rows (float4 0..11, one tensor gather each) in a 256-byte slot, so that
// every gather's destination starts on a 128-byte boundary.  Once a block's rows are read, its
// buffer holds the block's boxes of 16 leaves, until the copies of the block two ahead go there.
// pool: the boxes of 1 and of 4 leaves from each leaf on ([0 .. EB) and [EB .. 2 EB) mins and maxes
// of one, then of four); when every node has its box, the records: node of separator j at
// [4 j .. 4 j + 3] (rec_at).
// key, perm: the keys of this block's leaves and the next's, the permutation entries (mesh: the
// vertex indices) of the leaves two and three blocks ahead, all by 4-byte cp.async: held in registers
// from one block to the next they spilled, and a spilled load waits for its value at once.
template <int EB, bool MESH>
struct TreeSmem {
    static constexpr int kRow = MESH ? 3 : 4;      // float4 per leaf in a slot
    static constexpr int kIdx = MESH ? 3 : 1;      // index words per leaf
    float4 slot[2][EB * kRow];
    float4 pool[4 * EB];
    __align__(16) uint32_t plane[EB / 32][8];  // (16-byte loads) bit b of the separators before leaves
                                               // 32 w .. 32 w + 31, at [w][b]
    uint32_t key[2][EB + 2];      // keys of leaves b0-1 .. b0+EB, by buffer parity
    uint32_t perm[2][kIdx * EB];  // as above: two blocks ahead of a block on buffer b at [b]
    int P[EB];                    // separator j's node: its index less b0 (-1: not in this block)
    Span ring[8];                 // spans of this CTA's blocks it .. it + 4 at [it % 8], several segments
    uint64_t bar[2];              // completion of the gathers into slot[0] / slot[1]
    uint8_t wmin[EB / 32];        // smallest separator of each warp's
    uint8_t sep[EB + 1];          // separators (before each leaf and after the last; -1 as 0)
    int open[2];                  // open items emitted, by buffer parity (a block's and the next's)
};

// The lanes whose 6-bit value, given bit by bit in planes, is below v.
__device__ __forceinline__ uint32_t lanes_below(const uint32_t (&plane)[6], uint32_t v) {
    uint32_t lt = 0, eq = 0xFFFFFFFFu;
#pragma unroll
    for (int b = 5; b >= 0; --b) {
        const uint32_t m = (uint32_t)((int32_t)(v << (31 - b)) >> 31);  // all ones when v has bit b
        lt |= eq & m & ~plane[b];
        eq &= ~(plane[b] ^ m);
    }
    return lt;
}

__device__ __forceinline__ void box_join(float4 &lo, float4 &hi, const float4 &l, const float4 &h) {
    lo.x = fminf(lo.x, l.x); lo.y = fminf(lo.y, l.y); lo.z = fminf(lo.z, l.z);
    hi.x = fmaxf(hi.x, h.x); hi.y = fmaxf(hi.y, h.y); hi.z = fmaxf(hi.z, h.z);
}

// The separators of up to 32 W consecutive leaves or items as bit planes: bit b of those before
// 32 w .. 32 w + 31 at plane[w][b], each warp's smallest at wmin[w], each one at sep[i] (6 bits: -1,
// past a segment's ends, as 0; other separators are 2 or more).
//
// The nearest smaller separators of sv, the one before this thread's leaf or item, among the m + 1
// around and between m of them: na before it (-1: none), nb after it (m + 1: none).
template <int W>
__device__ __forceinline__ void nearest_smaller(const uint32_t (*plane)[8], const uint8_t *wmin, const uint8_t *sep,
                                                const uint32_t (&own)[6], uint32_t sv, int m, int &na, int &nb) {
    const int warp = threadIdx.x >> 5;
    const uint32_t below = lanes_below(own, sv), lt = lanemask_lt();
    const uint32_t ml = below & lt, mr = below & ~lt;  // (this lane's own bit is never set)
    uint32_t wb = 0;  // the warps with a separator below this one
#pragma unroll
    for (int w = 0; w < W; ++w) wb |= (uint32_t)(wmin[w] < sv) << w;
    auto search = [&](int w) {
        const uint4 x = *reinterpret_cast<const uint4 *>(&plane[w][0]);
        const uint2 y = *reinterpret_cast<const uint2 *>(&plane[w][4]);
        const uint32_t p6[6] = {x.x, x.y, x.z, x.w, y.x, y.y};
        return lanes_below(p6, sv);
    };
    na = -1;
    nb = m + 1;
    if (ml) {
        na = 32 * warp + 31 - __clz(ml);
    } else {
        const uint32_t wl = wb & ((1u << warp) - 1u);
        if (wl) {
            const int w = 31 - __clz(wl);
            na = 32 * w + 31 - __clz(search(w));
        }
    }
    if (mr) {
        nb = 32 * warp + __ffs(mr) - 1;
    } else {
        const uint32_t wr = wb & ~((2u << warp) - 1u);
        if (wr) {
            const int w = __ffs(wr) - 1;
            nb = 32 * w + __ffs(search(w)) - 1;
        } else if (sep[m] < sv) {
            nb = m;
        }
    }
}

// This thread's bit-plane words (all lanes call it) and what the block sees of them.
__device__ __forceinline__ void put_planes(uint32_t sv, uint32_t (&own)[6], uint32_t (*plane)[8], uint8_t *wmin) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t mine = 0;
#pragma unroll
    for (int b = 0; b < 6; ++b) {
        own[b] = __ballot_sync(0xFFFFFFFFu, (sv >> b) & 1u);
        mine = lane == b ? own[b] : mine;
    }
    if (lane < 6) plane[warp][lane] = mine;
    const uint32_t smallest = __reduce_min_sync(0xFFFFFFFFu, sv);
    if (lane == 0) wmin[warp] = (uint8_t)smallest;
}

// Boxes of 1, 4 and 16 consecutive leaves or items from each one on, cut at the warp's end.
struct Windows {
    float4 *lo1, *hi1, *lo4, *hi4, *lo16, *hi16;
    // this thread's 4 and 16 (all lanes call it; lo, hi: its own box)
    __device__ __forceinline__ void put(float4 lo, float4 hi) const {
        const int t = threadIdx.x;
        auto widen = [&](int d) {  // (past the warp's end a lane meets itself)
            box_join(lo, hi, make_float4(__shfl_down_sync(0xFFFFFFFFu, lo.x, d), __shfl_down_sync(0xFFFFFFFFu, lo.y, d),
                                         __shfl_down_sync(0xFFFFFFFFu, lo.z, d), 0.f),
                     make_float4(__shfl_down_sync(0xFFFFFFFFu, hi.x, d), __shfl_down_sync(0xFFFFFFFFu, hi.y, d),
                                 __shfl_down_sync(0xFFFFFFFFu, hi.z, d), 0.f));
        };
        widen(1);
        widen(2);
        lo4[t] = lo;
        hi4[t] = hi;
        widen(4);
        widen(8);
        lo16[t] = lo;
        hi16[t] = hi;
    }
    // The union of a .. b - 1 (at least two), warp by warp: a range that goes on past its first warp
    // takes that warp's part as one cut window of 16 (two from 17 on); any other piece is at most
    // four windows, the last one ending with it.
    __device__ __forceinline__ void get(int a, int b, float4 &lo, float4 &hi) const {
        int u = a, e = min(b, (a | 31) + 1);
        if (e < b) {
            lo = lo16[a];
            hi = hi16[a];
            if (e - a > 16) box_join(lo, hi, lo16[e - 16], hi16[e - 16]);
            u = e;
            e = min(b, u + 32);
        } else {
            lo = lo1[a];
            hi = hi1[a];
            u = a + 1;
        }
        for (;;) {
            const int len = e - u, step = len >= 16 ? 16 : len >= 4 ? 4 : 1, z = e - step;
            const float4 *slo = len >= 16 ? lo16 : len >= 4 ? lo4 : lo1, *shi = len >= 16 ? hi16 : len >= 4 ? hi4 : hi1;
            box_join(lo, hi, slo[z], shi[z]);
            for (int i = u; i < z; i += step) box_join(lo, hi, slo[i], shi[i]);
            if (e == b) break;
            u = e;
            e = min(b, e + 32);
        }
    }
};

// Word `part` of the record of separator j in a pool of records, each record's four words rotated
// so that the scattered writes of its two halves spread over the banks.
__device__ __forceinline__ int rec_at(int j, int part) { return 4 * j + (part ^ ((j >> 1) & 3)); }
// Box and link of a child into its parent's record: side 0 in words 0 and 1, side 1 in 2 and 3
// (f_1 = 2, f_2 = 0).
__device__ __forceinline__ void hand_over(float4 *pool, int j, bool left, float4 lo, float4 hi) {
    hi.w = __int_as_float(left ? 2 : 0);
    pool[rec_at(j, left ? 0 : 2)] = lo;
    pool[rec_at(j, left ? 1 : 3)] = hi;
}

// K3b: leaf gather, rearrange and the tree over blocks of EB sorted leaves (see the pass list
// above).  Leaf t of a block gathers triangle perm[b0 + t]: its index is loaded three blocks
// ahead, its 48-byte row is copied into shared memory two blocks ahead (with those of leaves
// t+1..t+3 by one tile::gather4 copy through `soup_map`, the soup as a tensor of 12-float
// rows, completing on the buffer's mbarrier; no registers held meanwhile), then written to the
// output soup and reduced to the leaf box.  A mesh leaf's three 16-byte vertex rows (mostly L2
// hits) come by cp.async instead (soup_map unused).
//
// Separator j of the block (the split before leaf j, j >= 1) has its node on thread j.  The node
// covers leaves a .. b - 1 between the nearest smaller separators on either side; its parent is
// the node of the larger of those two, its index follows from its range, its box is the union of
// its leaves.  The nearest smaller separators come from bit planes (six ballots per warp: the
// lanes below a value are a few bit operations on them; the warp to look in from the warps'
// minima), the box from windows of 1, 4 and 16 leaves made by shuffles.  Node and leaf then hand
// box and link to their parent's record in shared memory, and each record goes out by four
// neighbouring threads.  A node with no smaller separator on one side within the block lies across
// its edge; what hangs below such nodes leaves as open items.
//
// What bounds it: shared-memory wavefronts (65 % of the LSU pipe), four block barriers a block
// and DRAM (220 B per triangle at 2^24, 50 %); issue slots are half used.  Leaves that climb from
// child to parent instead wait in dependent chains (13,000 cycles of a block's 19,000).  The pass,
// climb -> this (B200): 2^24 clustered triangles 847 -> 803 us, 1,000,003 59 -> 53, the 2 M mesh
// 118 -> 94, a 1,024-mesh batch of 33 M triangles 1,806 -> 1,476.
template <int LOG, class Segs, class Leaves = SoupLeaves>
__global__ void __launch_bounds__(TreeGeo<LOG>::EB, TreeGeo<LOG>::kCtasPerSm) k_tree_climb(Segs segs,
                                                    const uint32_t *__restrict__ keys_all,
                                                    Leaves lv,
                                                    float4 *nodes_all, int32_t *parents_all,
                                                    OpenItem *out_items, uint32_t *out_counts,
                                                    Control *ctl, const __grid_constant__ CUtensorMap soup_map) {
    constexpr int EB = TreeGeo<LOG>::EB, W = EB / 32;
    constexpr bool kOne = std::is_same<Segs, OneSeg<LOG>>::value;
    // When a block's buffer is refilled: beside the hand-over, by two warps (one soup: its scattered
    // rows come late enough as it is, 2^24 triangles 803 us against 842-867 at the end), or at the
    // end, by every warp (meshes of a batch and mesh leaves, whose rows mostly hit L2: the copies'
    // queueing holds up no barrier, a 33 M triangle batch 1,573 -> 1,475 us, the 2 M mesh 96 -> 94)
    constexpr bool kLate = !kOne || Leaves::kMesh;
    using Smem = TreeSmem<EB, Leaves::kMesh>;
    static_assert(offsetof(Smem, plane) % 16 == 0 && offsetof(Smem, pool) % 16 == 0 && offsetof(Smem, bar) % 8 == 0, "aligned loads");
    extern __shared__ __align__(16) unsigned char smem[];
    // the layout from the first 128-byte boundary (the launch adds 128 bytes of slack)
    Smem &S = *reinterpret_cast<Smem *>(smem + ((128u - (smem_addr(smem) & 127u)) & 127u));
    // leaf t's three rows in buffer b
    auto tri_row = [&](int b, int x) -> float4 * { return &S.slot[b][Leaves::kMesh ? 3 * x : (x >> 2) * 16 + (x & 3) * 3]; };
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    chain_wait();
    // a sort whose look-back gave up left unsorted keys: build nothing from them (uniform)
    if (ld_relaxed_gpu(&ctl->err) & ERR_LOOKBACK_TIMEOUT) return;
    const int nblk = segs.blocks();

    // Leaves come in three steps ahead of their block: the permutation entry (its three vertex
    // indices for a mesh) three blocks ahead, its triangle copied into slot[] two blocks ahead, its
    // key one block ahead.  Two buffers, slot[0] and slot[1], serve the copies two blocks ahead: a
    // block's buffer is refilled once its boxes are used, so the copies of two blocks are in flight
    // for most of a block.
    const int grid = (int)gridDim.x;
    // the span of this CTA's block `it` (a batch's, loads in a chain, by thread 0 an iteration before
    // anyone needs it)
    auto span_of = [&](int it) -> Span {
        if constexpr (kOne) return segs.span(blockIdx.x + it * grid);
        else return S.ring[it & 7];
    };
    auto find_span = [&](int it) {
        if constexpr (!kOne)
            if ((int)blockIdx.x + it * grid < nblk) S.ring[it & 7] = segs.span(blockIdx.x + it * grid);
    };
    auto fetch_perm = [&](const Span &sp, int b) {
        if constexpr (Leaves::kMesh) {
            const int words = 3 * min(EB, sp.n - sp.b0);
            const uint32_t *r = lv.sidx + 3ull * (sp.start + sp.b0);
#pragma unroll
            for (int q = 0; q < 3; ++q)
                if (t + q * EB < words) cp_async4(&S.perm[b][t + q * EB], r + t + q * EB);
        } else if (sp.b0 + t < sp.n) {
            cp_async4(&S.perm[b][t], lv.perm + sp.start + sp.b0 + t);
        }
    };
    bool bad_perm = false;
    // Mesh: the block's vertex rows (mostly in L2) by cp.async, one commit group per thread and block.
    auto fetch_mesh = [&](const Span &sp, int buf) {
        if constexpr (Leaves::kMesh) {
            if (sp.b0 + t < sp.n) {
                // an index past the vertex buffer was reported by the Morton pass; read row 0
                const uint32_t nv = lv.nverts;
                const uint32_t *p = &S.perm[buf][3 * t];
                float4 *d = tri_row(buf, t);
#pragma unroll
                for (int q = 0; q < 3; ++q) cp_async16(d + q, lv.verts + (p[q] < nv ? p[q] : 0u));
            }
            cp_async_commit();
        }
    };
    // Soup: group g of a block's gathers into slot[buf] (leaves 4g .. 4g+3) as one tile::gather4 copy
    // on the buffer's mbarrier, whose phase expects 192 bytes per group (group 0's arrival is its
    // only one); a leaf past the segment repeats its group's first row (read, never used).  The copy
    // engine takes about one small copy per 11 to 17 cycles per SM, which one 48-byte copy per leaf
    // kept saturated; with four rows a copy and the tensor map's 64-byte L2 fills a random gather of
    // 16.7 M rows takes 0.55 ms against 0.67 (B200; DRAM reads 154 -> 98 B per row).
    auto gather_rows = [&](const Span &sp, int buf, int g) {
        const int m2 = min(EB, sp.n - sp.b0), ng = (m2 + 3) / 4;
        if (g == 0) mbar_arrive_tx(&S.bar[buf], 192u * (uint32_t)ng);
        if (g < ng) {
            uint32_t row[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t ti = S.perm[buf][4 * g + (4 * g + q < m2 ? q : 0)];
                if (ti >= (uint32_t)sp.n) { bad_perm = true; ti = 0; }
                row[q] = (uint32_t)(sp.start + ti);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // reads and writes above, copies below
            gather4_g2s(&S.slot[buf][16 * g], &soup_map, row[0], row[1], row[2], row[3], &S.bar[buf]);
        }
    };
    // one block ahead: the keys of its leaves and on either side of it
    auto fetch_keys = [&](const Span &sp, int b) {
        const uint32_t *keys = keys_all + sp.start;
        const int b0 = sp.b0, n = sp.n, k = b0 + t;
        if (k < n) cp_async4(&S.key[b][t + 1], keys + k);
        if (t == 0 && b0 > 0) cp_async4(&S.key[b][0], keys + b0 - 1);
        if (t == EB - 1 && b0 + EB < n) cp_async4(&S.key[b][EB + 1], keys + b0 + EB);
    };
    // The block two ahead's leaves into slot[buf], which no thread reads any more.
    auto refill = [&](int blk, int it, int buf) {
        if (blk + 2 * grid >= nblk) return;
        if constexpr (Leaves::kMesh) {
            fetch_mesh(span_of(it + 2), buf);
        } else {
            const int g = kLate ? 8 * warp + lane : t - EB / 2;
            if (kLate ? lane < 8 : g >= 0 && g < EB / 4) gather_rows(span_of(it + 2), buf, g);
        }
    };
    int buf = 0;
    uint32_t phase = 0;  // bit b: parity of the next phase of S.bar[b] (uniform over the block)
    bool copy_timeout = false;
    if (t < 2) mbar_init(&S.bar[t], 1);
    if (t < 2) S.open[t] = 0;
    if (t < 4) find_span(t);
    mbar_init_fence();
    __syncthreads();
    if ((int)blockIdx.x < nblk) {
        // the first two blocks' leaves (uniform branches)
        for (int k = 0; k < 2 && (int)blockIdx.x + k * grid < nblk; ++k) fetch_perm(span_of(k), k);
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
        for (int k = 0; k < 2 && (int)blockIdx.x + k * grid < nblk; ++k) {
            const Span sp = span_of(k);
            if constexpr (Leaves::kMesh) fetch_mesh(sp, k);
            else if (t < EB / 4) gather_rows(sp, k, t);
        }
        __syncthreads();  // perm is read
        fetch_keys(span_of(0), 0);
        if ((int)blockIdx.x + 2 * grid < nblk) fetch_perm(span_of(2), 0);
        cp_async_commit();
    }

    // Thread 0, after a barrier that follows the previous block's emissions: that block's count
    // of open items, and its counter cleared for the next block (the counters alternate with the
    // buffers).
    auto settle_prev = [&](int blk, int buf) {
        if (blk - grid >= (int)blockIdx.x) {
            const int o = S.open[buf ^ 1];
            out_counts[blk - grid] = (uint32_t)min(o, kOpenCap);
            out_counts[nblk + blk - grid] = 0u;  // a counter of the straddling pass
            if (o > kOpenCap) atomicOr(&ctl->err, ERR_TREE);
        }
        S.open[buf ^ 1] = 0;
    };
    // after the barrier that ends a block's use of the other buffer's keys and indices: the next
    // block's keys and the permutation three blocks ahead
    auto fetch_next = [&](int blk, int it, int buf) {
        if (blk + grid < nblk) fetch_keys(span_of(it + 1), buf ^ 1);
        if (blk + 3 * grid < nblk) fetch_perm(span_of(it + 3), buf ^ 1);
        cp_async_commit();
    };
    int last = -1, last_buf = 0;
    for (int blk = blockIdx.x, it = 0; blk < nblk; blk += grid, ++it, buf ^= 1) {
        last = blk;
        last_buf = buf;
        const Span sp = span_of(it);
        const int b0 = sp.b0, n = sp.n;
        float4 *nodes = nodes_all + 4ull * sp.start;
        int32_t *parents = parents_all + 2ull * sp.start;
        const int m = min(EB, n - b0);
        const int k = b0 + t;
        const bool active = t < m;
        // this leaf's triangle: to the output soup, and its box (exact-zero components nudged
        // by 1e-8 as bvh-up-pass.js:209-210 does)
        if constexpr (Leaves::kMesh) {
            // the rows of the next block may still be in flight (the newest group), not this one's; in
            // the first turn the keys came last
            if (blk + grid < nblk && blk != (int)blockIdx.x) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else cp_async_wait_all();
        } else {
            cp_async_wait_all();
            if (!mbar_wait(&S.bar[buf], (phase >> buf) & 1u)) copy_timeout = true;
            phase ^= 1u << buf;
        }
        float4 leaf_lo = make_float4(0.f, 0.f, 0.f, __int_as_float(-(k + 1)));
        float4 leaf_hi = make_float4(0.f, 0.f, 0.f, 0.f);
        if (active) {
            const float4 *tr = tri_row(buf, t);
            const float4 a = tr[0], b = tr[1], c = tr[2];
            if constexpr (!Leaves::kMesh) {
                float4 *dst = lv.otri + 3ull * (sp.start + k);
                st_stream(dst, a);
                st_stream(dst + 1, b);
                st_stream(dst + 2, c);
            }
            float nx = fminf(a.x, fminf(b.x, c.x)), ny = fminf(a.y, fminf(b.y, c.y)), nz = fminf(a.z, fminf(b.z, c.z));
            float xx = fmaxf(a.x, fmaxf(b.x, c.x)), xy = fmaxf(a.y, fmaxf(b.y, c.y)), xz = fmaxf(a.z, fmaxf(b.z, c.z));
            nx = nx == 0.0f ? -1e-8f : nx; ny = ny == 0.0f ? -1e-8f : ny; nz = nz == 0.0f ? -1e-8f : nz;
            xx = xx == 0.0f ? 1e-8f : xx;  xy = xy == 0.0f ? 1e-8f : xy;  xz = xz == 0.0f ? 1e-8f : xz;
            leaf_lo = make_float4(nx, ny, nz, __int_as_float(-(k + 1)));
            leaf_hi = make_float4(xx, xy, xz, 0.f);
        }
        if (n == 1) {  // one leaf, one arrival at node 0: left slot only, f_1 = 1
            if (t == 0) {
                nodes[0] = make_float4(leaf_lo.x, leaf_lo.y, leaf_lo.z, __int_as_float(-1));
                nodes[1] = make_float4(leaf_hi.x, leaf_hi.y, leaf_hi.z, __int_as_float(1));
                nodes[2] = make_float4(0.f, 0.f, 0.f, 0.f);
                nodes[3] = make_float4(0.f, 0.f, 0.f, 0.f);
                parents[0] = 0;
                parents[1] = 0;
            }
            // uniform across the block.  The barrier keeps every thread's wait on this buffer's
            // phase and its reads ahead of the refill.
            __syncthreads();
            if (t == 0) {
                settle_prev(blk, buf);
                find_span(it + 4);
            }
            fetch_next(blk, it, buf);
            refill(blk, it, buf);
            __syncthreads();  // perm is read
            continue;
        }
        if (k == 0) {  // the root has no parent; slot N-1 and record N-1 stay zero
            parents[0] = 0;
            parents[n - 1] = 0;
            const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            float4 *last = nodes + 4ull * (n - 1);
            last[0] = z; last[1] = z; last[2] = z; last[3] = z;
        }
        __syncthreads();  // rows read, keys written; the block before is done with the pool
        if (t == 0) {
            settle_prev(blk, buf);
            find_span(it + 4);
        }
        fetch_next(blk, it, buf);
        // the separator before leaf t, as 6 bits: d of a split is 2 or more (keys below 2^30, indices
        // below 2^30), -1 past the segment's ends is kept as 0; past the block's leaves 63
        auto dval = [&](int x) -> uint32_t {  // separator after leaf b0 + x, x in [-1, EB - 1]
            const int g = b0 + x;
            if (g < 0 || g >= n - 1) return 0u;
            const uint32_t a = S.key[buf][x + 1], b = S.key[buf][x + 2];
            return (uint32_t)(a != b ? __clz(a ^ b) : 32 + __clz(g ^ (g + 1)));
        };
        const uint32_t sv = active ? dval(t - 1) : 63u;
        uint32_t pl[6];
        put_planes(sv, pl, S.plane, S.wmin);
        if (active) S.sep[t] = (uint8_t)sv;
        if (t == m - 1) S.sep[m] = (uint8_t)dval(m - 1);
        S.P[t] = -1;
        const Windows win{S.pool, S.pool + EB, S.pool + 2 * EB, S.pool + 3 * EB, S.slot[buf], S.slot[buf] + EB};
        win.lo1[t] = leaf_lo;
        win.hi1[t] = leaf_hi;
        win.put(leaf_lo, leaf_hi);
        __syncthreads();
        int na = -1, nb = m + 1;  // separator t's node: leaves na .. nb - 1 (-1, m + 1: none in the block)
        if (t >= 1 && active) nearest_smaller<W>(S.plane, S.wmin, S.sep, pl, sv, m, na, nb);
        // the node: index, box, and the record its parent has (separator np, 0 and m: not here)
        const bool in = na >= 0 && nb <= m && t >= 1 && active;
        float4 nlo, nhi;
        int np = 0, P = 0;
        bool nleft = false, root = false;
        if (in) {
            nleft = S.sep[nb] > S.sep[na];
            root = b0 + na == 0 && b0 + nb == n;
            P = root ? 0 : nleft ? nb - 1 : na;  // (the root's block begins the segment: b0 == 0)
            np = nleft ? nb : na;
            S.P[t] = P;
            win.get(na, nb, nlo, nhi);
            nlo.w = __int_as_float(b0 + P);
        }
        const bool lleft = active && S.sep[t + 1] > sv;  // the leaf is its parent's left child
        const int ip = lleft ? t + 1 : t;
        leaf_lo = win.lo1[t];  // (read back rather than held through the search)
        leaf_hi = win.hi1[t];
        __syncthreads();
        if (in && !root && np > 0 && np < m) hand_over(S.pool, np, nleft, nlo, nhi);
        if (active && ip > 0 && ip < m) hand_over(S.pool, ip, lleft, leaf_lo, leaf_hi);
        if (!kLate) refill(blk, it, buf);
        __syncthreads();
        // parent links, and what leaves the block for K3c
        OpenItem *out = out_items + (size_t)blk * kOpenCap;
        auto emit = [&](float4 lo, float4 hi, int a, int b) {
            const int dl = S.sep[a], dr = S.sep[b];
            OpenItem it;
            it.lo = lo;
            it.hi = make_float4(hi.x, hi.y, hi.z, __int_as_float(dr ? dr : -1));
            it.xl = b0 + a;
            it.xr = b0 + b - 1;
            it.pad0 = dl ? dl : -1;
            it.pad1 = 0;
            const int at = atomicAdd(&S.open[buf], 1);
            if (at < kOpenCap) out[at] = it;
            else atomicOr(&ctl->err, ERR_TREE);
        };
        if (active) {
            const int q = ip > 0 && ip < m ? S.P[ip] : -1;
            if (q >= 0) parents[n + k] = b0 + q;
            else emit(leaf_lo, leaf_hi, t, t + 1);
        }
        if (in && !root) {
            const int q = np > 0 && np < m ? S.P[np] : -1;
            if (q >= 0) parents[b0 + P] = b0 + q;
            else emit(nlo, nhi, na, nb);
        }
        // the records, four threads each
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int j = r * (EB / 4) + (t >> 2), part = t & 3;
            const int q = S.P[j];
            if (q >= 0) nodes[4ull * (b0 + q) + part] = S.pool[rec_at(j, part)];
        }
        if (kLate) refill(blk, it, buf);
    }
    __syncthreads();  // the last block's open items are counted
    if (t == 0 && last >= 0) {
        const int o = S.open[last_buf];
        out_counts[last] = (uint32_t)min(o, kOpenCap);
        out_counts[nblk + last] = 0u;
        if (o > kOpenCap) atomicOr(&ctl->err, ERR_TREE);
    }
    if (bad_perm) atomicOr(&ctl->err, ERR_TREE);
    if (copy_timeout) atomicOr(&ctl->err, ERR_COPY_TIMEOUT);
}

// K3c: the nodes that straddle tree blocks, without a climb.  The open items of consecutive
// blocks, in leaf order, partition those blocks' leaves; with the separators between and around
// them they are a shorter instance of the same problem: the node of the separator at split s
// covers the items between the nearest smaller separators on either side, its parent is the node
// of the larger of those two, its index follows from its own range, and its box is the union of a
// range of items.  So every node of such a run is found on its own thread (reduce_run).  A node
// with no smaller separator on one side within the run extends past it; the maximal subtrees
// below such nodes (at most 2 x 64: they hang off the run's two boundary paths) are the run's own
// open items.
//
// One block reduces a group of kGroupBlocks tree blocks; the last of kFan neighbouring groups to
// finish (a counter per parent, nothing waits) goes on with what those groups left as one run,
// and so on up to the root: three levels at 2^20 triangles, four at 2^24.  Latency bounds it: a level
// is six block barriers and four dependent L2 accesses, about 4 us (an item that climbs pays 0.5 to
// 2.6 us for each of up to 31 levels of the tree).  The pass, climbs -> runs (B200): 4,098 triangles
// 19 -> 5 us, 65,536 uniform 35 -> 10, 1,000,003 clustered 63 -> 22, the 2 M sphere 65 -> 27, 2^24
// clustered 130 -> 70, 1,024 meshes of 33 M triangles 203 -> 117.
//
// Sizes: a run holds at most 256 items, one per thread: a child's open items (<= kOpenCap) always
// fit beside what the children before it left (<= kOpenCap), so a run that would be longer is
// reduced a few children at a time.  A tree block leaves 8.1 items on average (uniform and
// clustered triangles), so a group of 24 blocks leaves 60 of 256 threads idle and rarely needs a
// second turn.  16 blocks (more levels, more idle threads) take 89 us at 2^24 and 142 for the
// batch, 28 blocks and 14 groups 68 and 109 but 23.1 (22.0) at 1,000,003 and 29.5 (27.3) for the
// sphere.
constexpr int kRunCap = 256;
constexpr int kRunWarps = kRunCap / 32;
static_assert(kRunCap >= 2 * kOpenCap && kGroupBlocks <= 32 && kFan <= 32, "a run takes two children; one warp counts them");

struct RunSmem {
    float4 lo[3][kRunCap], hi[3][kRunCap];  // Windows; when every node has its box, [1] holds those of
                                            // the nodes that leave (box, link and end item)
    float4 rec[4 * kRunCap];                // the separators' records (rec_at)
    __align__(16) uint32_t plane[kRunWarps][8];
    int xl[kRunCap + 1];     // first leaf of each item, then the end of the last one
    int P[kRunCap];          // the separators' nodes (-1: not in this run)
    int out[kRunCap];        // what leaves the run from item i on: -1 nothing, 0 the item, else the node
                             // of separator out[i]
    int cstart[33];          // the children's first items among those loaded together
    int warp[kRunWarps];
    int take, last;
    uint8_t wmin[kRunWarps];
    uint8_t sep[kRunCap + 1];  // the separators around and between the items (-1 as 0)
};

// The open item of leaves [xl, xr]; dl, dr: the separators before and after it.
__device__ __forceinline__ OpenItem open_item(float4 lo, float4 hi, int ref, int xl, int xr, int dl, int dr) {
    OpenItem o;
    o.lo = make_float4(lo.x, lo.y, lo.z, __int_as_float(ref));
    o.hi = make_float4(hi.x, hi.y, hi.z, __int_as_float(dr));
    o.xl = xl;
    o.xr = xr;
    o.pad0 = dl;
    o.pad1 = 0;
    return o;
}

// Every node of the run of M items in S (lo[0] with the links, hi[0], xl[0 .. M], sep[0 .. M]
// set, a barrier since): records and parent links to memory; the run's own open items, in leaf
// order, to dst (at most kOpenCap of them) or, when dst is null, back to S as the next run.
// Returns their number (uniform).  ok: false when an index lies outside the segment (nothing is
// written for it).  Thread t has item t and the node of separator t, as in the tree pass.
__device__ __forceinline__ int reduce_run(RunSmem &S, int M, int n, float4 *nodes, int32_t *parents, OpenItem *dst,
                                          bool &ok) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool active = t < M;
    const Windows win{S.lo[0], S.hi[0], S.lo[1], S.hi[1], S.lo[2], S.hi[2]};
    const uint32_t sv = active ? S.sep[t] : 63u;
    uint32_t pl[6];
    put_planes(sv, pl, S.plane, S.wmin);
    const float4 ilo = S.lo[0][t], ihi = S.hi[0][t];  // (past the run's end: not used)
    win.put(ilo, ihi);
    S.out[t] = -1;
    S.P[t] = -1;
    __syncthreads();
    int na = -1, nb = M + 1, P = 0, np = 0;
    float4 nlo, nhi;
    bool in = false, root = false;
    const int ref = __float_as_int(ilo.w);
    if (active && (ref < -n || ref >= n - 1)) ok = false;
    if (t >= 1 && active) {
        nearest_smaller<kRunWarps>(S.plane, S.wmin, S.sep, pl, sv, M, na, nb);
        in = na >= 0 && nb <= M;
    }
    if (in) {
        const int L = S.xl[na], R = S.xl[nb] - 1;
        const bool left = S.sep[nb] > S.sep[na];
        root = L == 0 && R == n - 1;
        P = root ? 0 : left ? R : L;
        np = left ? nb : na;
        if ((uint32_t)P >= (uint32_t)(n - 1)) {
            ok = false;
            in = false;
        } else {
            S.P[t] = P;
            win.get(na, nb, nlo, nhi);
            nlo.w = __int_as_float(P);
            if (!root && np > 0 && np < M) hand_over(S.rec, np, left, nlo, nhi);
        }
    }
    const bool ileft = active && S.sep[t + 1] > sv;
    const int ip = ileft ? t + 1 : t;
    if (active && ip > 0 && ip < M) hand_over(S.rec, ip, ileft, ilo, ihi);
    __syncthreads();
    // parent links; what leaves: items and nodes of the run whose parent's node does not lie in it
    if (active) {
        const int q = ip > 0 && ip < M ? S.P[ip] : -1;
        if (q < 0) S.out[t] = 0;
        else if (ref >= -n && ref < n - 1) parents[ref >= 0 ? ref : n - (ref + 1)] = q;
    }
    if (in && !root) {
        const int q = np > 0 && np < M ? S.P[np] : -1;
        if (q >= 0) {
            parents[P] = q;
        } else {
            S.out[na] = t;
            nhi.w = __int_as_float(nb);
            S.lo[1][t] = nlo;  // the windows are read
            S.hi[1][t] = nhi;
        }
    }
    // the records, four threads each
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int j = r * (kRunCap / 4) + (t >> 2), part = t & 3;
        if (r * (kRunCap / 4) >= M) break;  // uniform
        const int q = S.P[j];
        if (q >= 0) nodes[4ull * q + part] = S.rec[rec_at(j, part)];
    }
    __syncthreads();
    const int o = S.out[t];
    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, o >= 0);
    if (lane == 0) S.warp[warp] = __popc(bal);
    float4 lo, hi;
    int oref = 0, xl = 0, xr = 0, dl = 0, dr = 0;
    if (o >= 0) {
        lo = S.lo[o ? 1 : 0][o ? o : t];
        hi = S.hi[o ? 1 : 0][o ? o : t];
        const int b = o ? __float_as_int(hi.w) : t + 1;
        oref = __float_as_int(lo.w);
        xl = S.xl[t];
        xr = S.xl[b] - 1;
        dl = S.sep[t];
        dr = S.sep[b];
    }
    const int end_xl = S.xl[M], end_sep = S.sep[M];
    __syncthreads();
    int at = __popc(bal & lanemask_lt()), total = 0;
#pragma unroll
    for (int w = 0; w < kRunWarps; ++w) {
        const int c = S.warp[w];
        at += w < warp ? c : 0;
        total += c;
    }
    if (dst) {
        if (o >= 0 && at < kOpenCap) dst[at] = open_item(lo, hi, oref, xl, xr, dl ? dl : -1, dr ? dr : -1);
        return total;
    }
    if (o >= 0) {
        S.lo[0][at] = lo;
        S.hi[0][at] = hi;
        S.xl[at] = xl;
        S.sep[at] = (uint8_t)dl;
    }
    if (t == 0) { S.xl[total] = end_xl; S.sep[total] = (uint8_t)end_sep; }
    __syncthreads();
    return total;
}

// The tree blocks of one segment as the straddling pass sees them: its first triangle and size,
// its tree blocks [blk0, blk1) as global block numbers and the group's number within it.
struct GroupSpan {
    size_t start;
    int n, blk0, blk1, grp;
};
template <int LOG>
struct OneSegGroups {
    static constexpr int kCtas = 3;  // 80 registers: 70 us at 2^24 either way, 22.0 against 23.3 at 1,000,003
    int n;
    __device__ __forceinline__ GroupSpan group(int g) const {
        return GroupSpan{0, n, 0, (n + (1 << LOG) - 1) >> LOG, g};
    }
};
struct ManySegGroups {  // groups never cross a segment; each starts at its segment's first group
    static constexpr int kCtas = 4;  // many runs at once: 117 us at 4 against 122 at 3
    const SegRow *rows;
    const uint32_t *grp_seg;
    __device__ __forceinline__ GroupSpan group(int g) const {
        const uint32_t sg = __ldg(grp_seg + g);
        const uint32_t t0 = __ldg(&rows[sg].tri), t1 = __ldg(&rows[sg + 1].tri);
        return GroupSpan{t0, (int)(t1 - t0), (int)__ldg(&rows[sg].blk), (int)__ldg(&rows[sg + 1].blk),
                         g - (int)__ldg(&rows[sg].grp)};
    }
};

// counts: per tree block its open items, then (n_counts words on) the counters of the units that
// start there, cleared by the tree pass.  A unit's open items are in its first block's slots.
template <class Groups>
__global__ void __launch_bounds__(kRunCap, Groups::kCtas) k_top_group(Groups groups, OpenItem *items, uint32_t *counts,
                                                           uint32_t n_counts, float4 *nodes_all, int32_t *parents_all,
                                                           Control *ctl) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RunSmem &S = *reinterpret_cast<RunSmem *>(smem_raw);
    const int t = threadIdx.x;
    chain_wait();
    if (ld_relaxed_gpu(&ctl->err) & ERR_LOOKBACK_TIMEOUT) return;  // unsorted keys: nothing to build
    const GroupSpan gs = groups.group(blockIdx.x);
    const int n = gs.n, nblk = gs.blk1 - gs.blk0;
    if (nblk < 2) return;  // one tree block: its root is complete
    float4 *nodes = nodes_all + 4ull * gs.start;
    int32_t *parents = parents_all + 2ull * gs.start;
    bool ok = true;
    // level 1: unit = group, children = tree blocks; each later level kFan times as wide
    int unit = gs.grp;
    long long stride = 1;  // tree blocks per child
    for (int level = 1, fan = kGroupBlocks;; ++level, stride *= fan, fan = kFan, unit /= fan) {
        const int first = (int)(unit * stride * fan);  // the unit's first block within the segment
        const int nchild = (int)min((long long)fan, (nblk - first + stride - 1) / stride);
        const size_t blk0 = (size_t)gs.blk0 + first;
        if (level > 1) {
            // the last child to come goes on with all of them; a single child is the unit
            if (nchild > 1) {
                __syncthreads();  // this block's items and count are written
                if (t == 0) {
                    uint32_t *tally = counts + n_counts + blk0 + (level - 1);
                    S.last = atom_add_acq_rel_gpu(tally, 1u) == (uint32_t)(nchild - 1);
                }
                __syncthreads();
                if (!S.last) break;
            }
        }
        if (nchild > 1 || level == 1) {
            // the children's items, as many children at a time as fit beside what is left of those
            // before; a run of what came so far is reduced in between
            int M = 0, c = 0;
            while (c < nchild) {
                if (t < 32) {
                    const bool child = c + t < nchild;  // at most 32
                    int incl = child ? (int)min(__ldcg(counts + blk0 + (c + t) * stride), (uint32_t)kOpenCap) : 0;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                        if (t >= o) incl += y;
                    }
                    S.cstart[t + 1] = incl;
                    if (t == 0) S.cstart[0] = 0;
                    const uint32_t fits = __ballot_sync(0xFFFFFFFFu, child && M + incl <= kRunCap);
                    if (t == 0) S.take = max(1, __popc(fits));
                }
                __syncthreads();
                const int take = S.take, add = min(S.cstart[take], kRunCap - M);
                // item t of them: child b's (a tree block's items are unordered: their place is their
                // rank by first leaf)
                OpenItem it;
                int at = t, b0 = 0, b1 = 0;
                if (t < add) {
                    int b = 0;  // the last child that starts at or before t
#pragma unroll
                    for (int h = 16; h > 0; h >>= 1) b += b + h < take && S.cstart[b + h] <= t ? h : 0;
                    b0 = S.cstart[b];
                    b1 = min(S.cstart[b + 1], add);
                    const OpenItem *src = items + (blk0 + (c + b) * stride) * kOpenCap + (t - b0);
                    it.lo = __ldcg(&src->lo);
                    it.hi = __ldcg(&src->hi);
                    const int4 x = __ldcg(reinterpret_cast<const int4 *>(&src->xl));
                    it.xl = x.x;
                    it.xr = x.y;
                    it.pad0 = x.z;
                    S.out[t] = x.x;
                    // every first leaf inside the segment: what is derived from it then is too
                    if (x.x < 0 || x.y < x.x || x.y >= n) ok = false;
                }
                if (level == 1) {  // uniform
                    __syncthreads();
                    if (t < add) {
                        at = b0;
#pragma unroll 4
                        for (int k = b0; k < b1; ++k) at += S.out[k] < it.xl;
                    }
                }
                if (t < add) {
                    const int x = M + at;
                    S.lo[0][x] = it.lo;
                    S.hi[0][x] = it.hi;
                    S.xl[x] = it.xl;
                    S.sep[x] = (uint8_t)min(max(it.pad0, 0), 63);
                    if (at == add - 1) {  // the run's end
                        S.xl[x + 1] = it.xr + 1;
                        S.sep[x + 1] = (uint8_t)min(max(__float_as_int(it.hi.w), 0), 63);
                    }
                }
                M += add;
                c += take;
                if (__syncthreads_or(!ok)) { M = 0; ok = false; break; }  // inconsistent items: build nothing from them
                if (M > 0) M = reduce_run(S, M, n, nodes, parents, c < nchild ? nullptr : items + blk0 * kOpenCap, ok);
                if (M > kOpenCap) { ok = false; M = kOpenCap; }
            }
            if (t == 0) counts[blk0] = (uint32_t)M;
            if (first == 0 && stride * fan >= nblk) {  // the whole segment: nothing may be left
                if (M != 0) ok = false;
                break;
            }
        }
    }
    if (!ok) atomicOr(&ctl->err, ERR_TREE);
}

// the layout plus the slack that puts it on a 128-byte boundary
template <int LOG, class Segs, class Leaves>
inline size_t leaves_smem_bytes() { return sizeof(TreeSmem<(1 << LOG), Leaves::kMesh>) + 128; }

// The soup as a 2-D tensor of `rows` rows of 12 floats, 48 bytes apart, for the tree pass's
// tile::gather4 copies: one-row boxes of a whole row, the L2 filling 64 bytes per DRAM request
// (most of a randomly gathered row's 128-byte line is never used).  The base is 16-byte
// aligned (every entry point checks it) and 1 <= rows <= LVBH_MAX_TRIS.
cudaError_t soup_tensor_map(CUtensorMap *m, const float4 *tri, uint32_t rows) {
    static const PFN_cuTensorMapEncodeTiled_v12000 enc = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    }();
    if (!enc) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {12, rows}, strides[1] = {48};
    const cuuint32_t box[2] = {12, 1}, elem[2] = {1, 1};
    const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float4 *>(tri), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_64B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int LOG, class Segs, class Leaves>
void launch_emit_impl(Segs segs, int groups, Leaves lv, const CUtensorMap &soup_map, const uint32_t *keys,
                      float4 *nodes, int32_t *parents, OpenItem *items, uint32_t *counts, Control *ctl,
                      cudaStream_t s, cudaEvent_t *ev, int ctas_per_sm, const uint32_t *grp_seg = nullptr,
                      int ngroups = 0) {
    if (ev) cudaEventRecord(ev[0], s);  // the leaf gather runs inside the tree pass
    const int per_sm = ctas_per_sm > 0 && ctas_per_sm < TreeGeo<LOG>::kCtasPerSm ? ctas_per_sm
                                                                                : TreeGeo<LOG>::kCtasPerSm;
    const int grid = min(groups, sm_count() * per_sm);
    // batched builds always chain; a one-mesh build by its size
    bool chain = true;
    if constexpr (std::is_same<Segs, OneSeg<LOG>>::value) chain = chain_build((uint32_t)segs.n);
    launch_chained(chain, k_tree_climb<LOG, Segs, Leaves>, grid, TreeGeo<LOG>::EB, leaves_smem_bytes<LOG, Segs, Leaves>(), s,
                   segs, keys, lv, nodes, parents, items, counts, ctl, soup_map);
    if (ev) cudaEventRecord(ev[1], s);
    if constexpr (std::is_same<Segs, OneSeg<LOG>>::value) {
        if (groups > 1)
            launch_chained(chain, k_top_group<OneSegGroups<LOG>>, straddle_groups((uint32_t)groups), kRunCap,
                           sizeof(RunSmem), s, OneSegGroups<LOG>{segs.n}, items, counts, (uint32_t)groups, nodes,
                           parents, ctl);
    } else if (ngroups > 0) {
        launch_chained(chain, k_top_group<ManySegGroups>, ngroups, kRunCap, sizeof(RunSmem), s,
                       ManySegGroups{segs.rows, grp_seg}, items, counts, (uint32_t)groups, nodes, parents, ctl);
    }
    if (ev) cudaEventRecord(ev[2], s);
}

template <class K>
cudaError_t prefer_shared(K kernel, size_t bytes) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                (int)cudaSharedmemCarveoutMaxShared);
}

}  // namespace

size_t emit_groups(uint32_t n, int log_eb) { return (n + (1u << log_eb) - 1) >> log_eb; }

cudaError_t emit_init() {
    constexpr int L = kLogEmitBlock;
    cudaError_t e = prefer_shared(k_tree_climb<L, OneSeg<L>>, leaves_smem_bytes<L, OneSeg<L>, SoupLeaves>());
    if (e == cudaSuccess) e = prefer_shared(k_tree_climb<8, ManySegs<8>>, leaves_smem_bytes<8, ManySegs<8>, SoupLeaves>());
    if (e == cudaSuccess) e = prefer_shared(k_tree_climb<7, ManySegs<7>>, leaves_smem_bytes<7, ManySegs<7>, SoupLeaves>());
    if (e == cudaSuccess)
        e = prefer_shared(k_tree_climb<L, OneSeg<L>, MeshLeaves>, leaves_smem_bytes<L, OneSeg<L>, MeshLeaves>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_top_group<OneSegGroups<L>>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(RunSmem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_top_group<ManySegGroups>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(RunSmem));
    return e;
}

cudaError_t launch_emit(const float4 *tri, const uint32_t *perm, const uint32_t *keys, uint32_t n,
                        float4 *otri, float4 *nodes, int32_t *parents, OpenItem *items,
                        uint32_t *counts, Control *ctl, cudaStream_t s, cudaEvent_t *ev) {
    if (n == 0) return cudaSuccess;
    CUtensorMap map;
    const cudaError_t e = soup_tensor_map(&map, tri, n);
    if (e != cudaSuccess) return e;
    const int groups = (int)emit_groups(n, kLogEmitBlock);
    launch_emit_impl<kLogEmitBlock>(OneSeg<kLogEmitBlock>{(int)n}, groups, SoupLeaves{tri, perm, otri}, map, keys,
                                    nodes, parents, items, counts, ctl, s, ev, 0);
    return cudaSuccess;
}

void launch_emit_mesh(const float4 *verts, uint32_t num_verts, const uint32_t *sidx, const uint32_t *keys,
                      uint32_t n, float4 *nodes, int32_t *parents, OpenItem *items, uint32_t *counts,
                      Control *ctl, cudaStream_t s, cudaEvent_t *ev) {
    if (n == 0) return;
    const int groups = (int)emit_groups(n, kLogEmitBlock);
    CUtensorMap unused;  // mesh leaves come by cp.async
    std::memset(&unused, 0, sizeof unused);
    launch_emit_impl<kLogEmitBlock>(OneSeg<kLogEmitBlock>{(int)n}, groups, MeshLeaves{verts, sidx, num_verts},
                                    unused, keys, nodes, parents, items, counts, ctl, s, ev, 0);
}

cudaError_t launch_emit_batch(const BatchPlan &bp, const float4 *tri, const uint32_t *perm,
                              const uint32_t *keys, float4 *otri, float4 *nodes, int32_t *parents,
                              OpenItem *items, uint32_t *counts, Control *ctl, cudaStream_t s,
                              cudaEvent_t *ev) {
    if (bp.blocks == 0) return cudaSuccess;
    CUtensorMap map;
    const cudaError_t e = soup_tensor_map(&map, tri, bp.total);
    if (e != cudaSuccess) return e;
    if (bp.log_block == 7)
        launch_emit_impl<7>(ManySegs<7>{bp.rows, bp.blk_seg, (int)bp.blocks}, (int)bp.blocks,
                            SoupLeaves{tri, perm, otri}, map, keys, nodes, parents, items, counts, ctl, s, ev,
                            bp.tree_ctas_per_sm, bp.grp_seg, (int)bp.groups);
    else
        launch_emit_impl<8>(ManySegs<8>{bp.rows, bp.blk_seg, (int)bp.blocks}, (int)bp.blocks,
                            SoupLeaves{tri, perm, otri}, map, keys, nodes, parents, items, counts, ctl, s, ev,
                            bp.tree_ctas_per_sm, bp.grp_seg, (int)bp.groups);
    return cudaSuccess;
}

}  // namespace lvbh
