// small.cu - K1 + K2 of a small build in one kernel: scene box, Morton keys and the whole sort on
// one thread-block cluster (sm_100a).
//
// A build of up to kSmallMax triangles leaves most of the chip idle whatever its kernels do; its
// time is their number.  The general path runs eleven launches before the tree pass (control-block
// clear, box and centroids, keys, three sort passes of two or three kernels), each 2.5 to 9 us for
// a few thousand keys.  Here one cluster of up to 16 blocks goes from the triangles to the sorted
// arrays: the keys stay in registers, the blocks exchange the box and their digit counts through
// distributed shared memory and the keys through L2, with two cluster barriers per pass.  Results
// are those of the general path (morton.cu, sort.cu).
//
// What bounds it: 16 SMs.  Of 61,000 cycles at 65,536 triangles (4 keys a thread) ranking by ballots
// took 21,000 (integer pipe: about 150 cycles a warp, key and scheduler), moving the keys 18,000,
// the rest was reading triangles, quantising and barriers; with three rows in four ranked by words
// (k_onesweep's mix, sort.cu) the kernel takes 29 us instead of 32, 17 at 4,098 triangles.  Whole
// calls in kept buffers, general path -> this one (B200, clustered): 1,000 triangles 81 -> 55 us,
// 4,098 83 -> 62, 20,000 93 -> 74, 50,000 95 -> 86, 65,536 95 -> 86 (uniform 93 -> 79), 81,920 98 ->
// 100, 131,072 106 -> 122 (eight keys a thread); so kSmallMax is 65,536.  Measured on it: keys
// scattered through distributed shared memory instead of L2 8,700 cycles a pass instead of 4,300
// (two cycles a store either way until the keys are put in digit order first), three 10-bit passes
// 35 us instead of 32, __match_any_sync for the ballots 40 us.
#include <atomic>
#include <cooperative_groups.h>

#include "lvbh_device.cuh"
#include "lvbh_internal.h"

namespace cg = cooperative_groups;

namespace lvbh {

namespace {

constexpr int T = 1024;
constexpr int W = T / 32;
constexpr int kMaxBlocks = 16;
constexpr int kSoup = 0, kMesh = 1;
// Digits: four passes of 8 bits over the 30-bit keys.  With 10-bit digits (three passes) the 32
// warps' counters of 1,024 digits were most of a pass.
constexpr int D = kDigits32, kPasses = kSortPasses32, kBits = kDigitBits32;
// A warp's counters: two digits to a word.  Rows 129 words apart: the prefix phase's lanes (four
// words of eight rows, every fourth row) then meet 32 different banks.
constexpr int kRow = D / 2 + 1;
constexpr int kParts = T / (D / 2), kPartRows = W / kParts;
constexpr int kCrowd = 8;  // peers in a ballot row above which the next three rows use ballots too
static_assert(kParts == 8 && kPartRows == 4, "one thread per word and group of four warps");

// IPT keys per thread.
template <int IPT>
struct SmallSmem {
    union {
        float cen[3][IPT * T];     // centroids, before the sort
        struct {
            uint2 kv[IPT * T];     // keys and values: staged in digit order (several blocks), or
                                   // between the passes (one block)
            uint32_t whist[W][kRow];  // per-warp digit counts, then per-warp offsets within the
                                      // block's digit
        };
    };
    uint32_t peers[IPT > 1 ? W : 1][IPT > 1 ? D : 4];  // the lanes of a warp's row that hold a digit (zero
                                                       // between rows)
    uint32_t cnt[D / 2];    // the block's digit counts, two to a word ...
    uint32_t all[kMaxBlocks][D / 2];  // ... and every block's (each writes its row in all blocks: reading
                                      // the other blocks' rows took 4,200 cycles a pass instead)
    uint32_t start[D];      // output position of the block's first key of each digit ...
    uint32_t tile[D];       // ... and its position among the block's keys in digit order
    uint2 warp[D / 64];
    float red[W][6];
    uint32_t ord[7];        // the block's box as ordered words, and its error bits ...
    uint32_t ords[kMaxBlocks][8];  // ... and every block's
    uint32_t box[7];        // the cluster's
    uint32_t stamp[3];      // profiled: the clock at the start, with the box and with the keys
};

// A cluster barrier in two halves, the triangles' loads in between.
__device__ __forceinline__ void cluster_started_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_started_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }

// Key i of a thread is key (block IPT T) + warp 32 IPT + 32 i + lane: input order is (block, warp,
// i, lane), the order the stable ranks count in.
// STAMPS (a profiled build): the first block's first thread reads the clock between the stages.
template <int SRC, int IPT, bool STAMPS>
__global__ void __launch_bounds__(T) k_small_sort(const float4 *__restrict__ rows, const uint32_t *__restrict__ idx3,
                                                  uint32_t nverts, uint32_t n, HostBounds hb,
                                                  Control *__restrict__ ctl, uint2 *kv,
                                                  uint32_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmallSmem<IPT> &S = *reinterpret_cast<SmallSmem<IPT> *>(smem_raw);
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), blocks = cluster.num_blocks();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t lt = lanemask_lt();
    const uint32_t local = warp * (32 * IPT) + lane, base = rank * (IPT * T) + local;
    const bool stamps = STAMPS && rank == 0 && tid == 0;
    if (stamps) S.stamp[0] = (uint32_t)clock();

    cluster_started_arrive();
    // boxes and centroids (aabb-z-idx.js:186-191)
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    uint32_t err = 0;
#pragma unroll 2
    for (int i = 0; i < IPT; ++i) {
        const uint32_t t = base + 32 * i;
        if (t >= n) continue;
        float4 v0, v1, v2;
        bool in0 = true, in1 = true, in2 = true;  // mesh: an index past the buffer reads row 0
        if constexpr (SRC == kMesh) {
            const uint32_t i0 = __ldg(idx3 + 3ull * t), i1 = __ldg(idx3 + 3ull * t + 1), i2 = __ldg(idx3 + 3ull * t + 2);
            in0 = i0 < nverts; in1 = i1 < nverts; in2 = i2 < nverts;
            v0 = __ldg(rows + (in0 ? i0 : 0u));
            v1 = __ldg(rows + (in1 ? i1 : 0u));
            v2 = __ldg(rows + (in2 ? i2 : 0u));
            if (!(in0 && in1 && in2)) err |= ERR_BAD_INDEX;
        } else {
            v0 = __ldg(rows + 3ull * t);
            v1 = __ldg(rows + 3ull * t + 1);
            v2 = __ldg(rows + 3ull * t + 2);
        }
        if (!(finite3(v0) && finite3(v1) && finite3(v2))) err |= ERR_NONFINITE;
        const float nx = fminf(v0.x, fminf(v1.x, v2.x)), ny = fminf(v0.y, fminf(v1.y, v2.y)), nz = fminf(v0.z, fminf(v1.z, v2.z));
        const float xx = fmaxf(v0.x, fmaxf(v1.x, v2.x)), xy = fmaxf(v0.y, fmaxf(v1.y, v2.y)), xz = fmaxf(v0.z, fmaxf(v1.z, v2.z));
        S.cen[0][local + 32 * i] = centroid(nx, xx);
        S.cen[1][local + 32 * i] = centroid(ny, xy);
        S.cen[2][local + 32 * i] = centroid(nz, xz);
        if (SRC == kSoup || (in0 && in1 && in2)) {
            mn[0] = fminf(mn[0], nx); mn[1] = fminf(mn[1], ny); mn[2] = fminf(mn[2], nz);
            mx[0] = fmaxf(mx[0], xx); mx[1] = fmaxf(mx[1], xy); mx[2] = fmaxf(mx[2], xz);
        }
    }
    // the scene box and the error bits: warp, block, cluster
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            mn[a] = fminf(mn[a], __shfl_xor_sync(0xFFFFFFFFu, mn[a], o));
            mx[a] = fmaxf(mx[a], __shfl_xor_sync(0xFFFFFFFFu, mx[a], o));
        }
    }
    err = __reduce_or_sync(0xFFFFFFFFu, err);
    if (tid < 7) S.ord[tid] = 0u;
    if (lane == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) { S.red[warp][a] = mn[a]; S.red[warp][3 + a] = mx[a]; }
    }
    __syncthreads();
    if (lane == 0 && err) atomicOr(&S.ord[6], err);
    if (warp < 6) {  // warp a: word a (min as ~ord_lo, max as ord_lo: the largest wins)
        const float v = S.red[lane][warp];
        S.ord[warp] = __reduce_max_sync(0xFFFFFFFFu, warp < 3 ? ~ord_lo(v) : ord_lo(v));
    }
    cluster_started_wait();  // every block runs: its shared memory may be written
    __syncthreads();
    if (lane < 7 && warp < (int)blocks) cluster.map_shared_rank(S.ords[rank], warp)[lane] = S.ord[lane];
    cluster.sync();
    if (tid < 7) {
        uint32_t w = 0;
#pragma unroll
        for (int q = 0; q < kMaxBlocks; ++q) {
            const uint32_t x = q < (int)blocks ? S.ords[q][tid] : 0u;
            w = tid < 6 ? max(w, x) : w | x;
        }
        S.box[tid] = w;
        if (rank == 0) {  // the control block's head: this kernel is the build's first
            if (tid < 6) ctl->bounds_ord[tid] = w;
            else ctl->err = w;
        }
    }
    __syncthreads();
    if (stamps) S.stamp[1] = (uint32_t)clock();
    float umin[3], umax[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        umin[a] = hb.use ? hb.v[a] : ord_lo_inv(~S.box[a]);
        umax[a] = hb.use ? hb.v[3 + a] : ord_lo_inv(S.box[3 + a]);
    }
    uint32_t k[IPT], v[IPT];
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
        v[i] = base + 32 * i;
        k[i] = 0;
        if (v[i] < n)
            k[i] = morton3(quantise_cen(S.cen[0][local + 32 * i], umin[0], umax[0]),
                           quantise_cen(S.cen[1][local + 32 * i], umin[1], umax[1]),
                           quantise_cen(S.cen[2][local + 32 * i], umin[2], umax[2]));
    }
    __syncthreads();  // the centroids are read; keys and counts take their place
    if (stamps) S.stamp[2] = (uint32_t)clock();

    if constexpr (IPT > 1) {
#pragma unroll
        for (int i = 0; i < D / 32; ++i) S.peers[warp][32 * i + lane] = 0u;
    }
    uint16_t *own = reinterpret_cast<uint16_t *>(S.whist[warp]);  // digit d at own[d]
    const uint32_t mine = min((uint32_t)(IPT * T), n - min(n, rank * (IPT * T)));  // the block's keys
    for (int pass = 0; pass < kPasses; ++pass) {
        const int shift = pass * kBits;
#pragma unroll
        for (int i = 0; i < D / 64; ++i) S.whist[warp][32 * i + lane] = 0u;
        __syncwarp();
        // stable ranks within the warp, as in k_onesweep: after a ballot row, up to three by words
        bool words = false;
        uint32_t rk[(IPT + 1) / 2];
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const bool valid = base + 32 * i < n;
            const uint32_t d = (k[i] >> shift) & (D - 1);
            const uint32_t c = own[d];  // (of digit 0 for a lane past the end: not used)
            uint32_t peers = 0;
            if (IPT > 1 && i % 4 != 0 && words) {
                uint32_t *w = &S.peers[IPT > 1 ? warp : 0][IPT > 1 ? d : 0];
                if (valid) atomicOr(w, 1u << lane);
                __syncwarp();
                if (valid) peers = *w;
                __syncwarp();
                if (peers >> lane == 1u) *w = 0u;
            } else {
                peers = __ballot_sync(0xFFFFFFFFu, valid);
#pragma unroll
                for (int b = 0; b < kBits; ++b) {
                    const uint32_t bit = (d >> b) & 1u;
                    const uint32_t vote = __ballot_sync(0xFFFFFFFFu, bit);
                    peers &= bit ? vote : ~vote;
                }
                if (!valid) peers = 0;
                if (IPT > 1 && i % 4 == 0) words = !__any_sync(0xFFFFFFFFu, __popc(peers) > kCrowd);
                __syncwarp();
            }
            if (peers >> lane == 1u) own[d] = (uint16_t)(c + __popc(peers));
            __syncwarp();
            const uint32_t x = c + __popc(peers & lt);
            if (i & 1) rk[i / 2] |= x << 16; else rk[i / 2] = x;
        }
        __syncthreads();
        // digits over the warps, two to a word (a block's counts stay below 2^16): thread 8 j + p has
        // word j of rows 4 p .. 4 p + 3
        {
            const int word = tid / kParts, part = tid % kParts;
            uint32_t x[kPartRows], sum = 0;
#pragma unroll
            for (int w = 0; w < kPartRows; ++w) { x[w] = S.whist[part * kPartRows + w][word]; sum += x[w]; }
            uint32_t incl = sum;
#pragma unroll
            for (int o = 1; o < kParts; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o, kParts);
                if (part >= o) incl += y;
            }
            uint32_t c = incl - sum;
#pragma unroll
            for (int w = 0; w < kPartRows; ++w) { S.whist[part * kPartRows + w][word] = c; c += x[w]; }
            if (part == kParts - 1) S.cnt[word] = c;
        }
        __syncthreads();
        for (uint32_t q = warp / (D / 64); q < blocks; q += W / (D / 64)) {
            const int word = 32 * (warp % (D / 64)) + lane;
            cluster.map_shared_rank(S.all[rank], q)[word] = S.cnt[word];
        }
        cluster.sync();  // every block's counts; every block has its keys in registers
        // thread tid: digits 2 tid and 2 tid + 1 over the cluster's blocks, then over the digits
        uint32_t pre0 = 0, pre1 = 0, tot0 = 0, tot1 = 0, own0 = 0, own1 = 0;
        uint2 incl = make_uint2(0u, 0u);
        if (tid < D / 2) {
#pragma unroll
            for (uint32_t q = 0; q < kMaxBlocks; ++q) {
                const uint32_t x = q < blocks ? S.all[q][tid] : 0u;
                if (q == rank) { pre0 = tot0; pre1 = tot1; own0 = x & 0xFFFFu; own1 = x >> 16; }
                tot0 += x & 0xFFFFu;
                tot1 += x >> 16;
            }
            incl = make_uint2(tot0 + tot1, own0 + own1);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl.x, o), z = __shfl_up_sync(0xFFFFFFFFu, incl.y, o);
                if (lane >= o) { incl.x += y; incl.y += z; }
            }
            if (lane == 31) S.warp[warp] = incl;
        }
        __syncthreads();
        if (tid < D / 2) {
            uint32_t off = incl.x - tot0 - tot1, loc = incl.y - own0 - own1;
#pragma unroll
            for (int w = 0; w < D / 64; ++w) {
                off += w < warp ? S.warp[w].x : 0u;
                loc += w < warp ? S.warp[w].y : 0u;
            }
            *reinterpret_cast<uint2 *>(&S.start[2 * tid]) = make_uint2(off + pre0, off + tot0 + pre1);
            *reinterpret_cast<uint2 *>(&S.tile[2 * tid]) = make_uint2(loc, loc + own0);
        }
        __syncthreads();
        // the block's keys in digit order (of one block: in sorted order)
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            if (base + 32 * i >= n) continue;
            const uint32_t d = (k[i] >> shift) & (D - 1);
            const uint32_t at = S.tile[d] + own[d] + ((rk[i / 2] >> (16 * (i & 1))) & 0xFFFFu);
            if (at < mine) S.kv[at] = make_uint2(k[i], v[i]);  // always, for consistent counts
        }
        __syncthreads();
        if (blocks > 1) {  // to their places, neighbours of one digit to neighbouring addresses
#pragma unroll
            for (int i = 0; i < IPT; ++i) {
                const uint32_t at = tid + T * i;
                if (at >= mine) continue;
                const uint2 x = S.kv[at];
                const uint32_t d = (x.x >> shift) & (D - 1), pos = S.start[d] + at - S.tile[d];
                if (pos < n) __stcg(kv + pos, x);
            }
            cluster.sync();  // every block's keys have arrived
        }
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            if (base + 32 * i >= n) continue;
            const uint2 x = blocks == 1 ? S.kv[local + 32 * i] : __ldcg(kv + base + 32 * i);
            k[i] = x.x;
            v[i] = x.y;
        }
    }
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
        const uint32_t t = base + 32 * i;
        if (t < n) {
            keys_out[t] = k[i];
            vals_out[t] = v[i];
        }
    }
    if (stamps) {
        const float all = (float)((uint32_t)clock() - S.stamp[0]);
        ctl->front[0] = (uint32_t)((float)(S.stamp[1] - S.stamp[0]) / all * 65536.0f);
        ctl->front[1] = (uint32_t)((float)(S.stamp[2] - S.stamp[0]) / all * 65536.0f);
    }
}

template <int SRC, int IPT, bool STAMPS>
cudaError_t allow_cluster() {
    auto k = k_small_sort<SRC, IPT, STAMPS>;
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallSmem<IPT>));
    return e == cudaSuccess ? cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : e;
}

template <int SRC, int IPT>
cudaError_t small_attrs(int *clusters) {
    cudaError_t e = allow_cluster<SRC, IPT, false>();
    if (e == cudaSuccess) e = allow_cluster<SRC, IPT, true>();
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kMaxBlocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = kMaxBlocks;
    cfg.blockDim = T;
    cfg.dynamicSmemBytes = sizeof(SmallSmem<IPT>);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int c = 0;
    e = cudaOccupancyMaxActiveClusters(&c, k_small_sort<SRC, IPT, false>, &cfg);
    if (c < *clusters) *clusters = c;
    return e;
}

template <int SRC, int IPT>
cudaError_t launch_ipt(const float4 *rows, const uint32_t *idx3, uint32_t nverts, uint32_t n, const HostBounds &hb,
                       Control *ctl, uint32_t *kv, uint32_t *keys, uint32_t *vals, bool stamps, cudaStream_t s) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (n + IPT * T - 1) / (IPT * T);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = attr[0].val.clusterDim.x;
    cfg.blockDim = T;
    cfg.dynamicSmemBytes = sizeof(SmallSmem<IPT>);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto k = stamps ? k_small_sort<SRC, IPT, true> : k_small_sort<SRC, IPT, false>;
    return cudaLaunchKernelEx(&cfg, k, rows, idx3, nverts, n, hb, ctl, reinterpret_cast<uint2 *>(kv), keys, vals);
}

// The fewest keys per thread with which at most 16 blocks hold n.
template <int SRC>
cudaError_t launch_src(const float4 *rows, const uint32_t *idx3, uint32_t nverts, uint32_t n, const HostBounds &hb,
                       Control *ctl, uint32_t *kv, uint32_t *keys, uint32_t *vals, bool stamps, cudaStream_t s) {
    const uint32_t per = (n + kMaxBlocks * T - 1) / (kMaxBlocks * T);
    if (per <= 1) return launch_ipt<SRC, 1>(rows, idx3, nverts, n, hb, ctl, kv, keys, vals, stamps, s);
    if (per <= 2) return launch_ipt<SRC, 2>(rows, idx3, nverts, n, hb, ctl, kv, keys, vals, stamps, s);
    static_assert(kSmallMax <= 4 * kMaxBlocks * T, "four keys per thread are enough");
    return launch_ipt<SRC, 4>(rows, idx3, nverts, n, hb, ctl, kv, keys, vals, stamps, s);
}

std::atomic<int> g_small_ok[64];  // per device: 1 when a full cluster of every form fits

}  // namespace

bool small_build(uint32_t n) {
    int dev = 0;
    cudaGetDevice(&dev);
    return n <= kSmallMax && dev >= 0 && dev < 64 && g_small_ok[dev].load(std::memory_order_relaxed);
}

// A device (or part of one) on which clusters of 16 such blocks cannot run answers the query with zero or
// with an error; either way its small builds take the general path.
void small_init() {
    int dev = 0, c = 1;
    cudaGetDevice(&dev);
    cudaError_t e = small_attrs<kSoup, 1>(&c);
    if (e == cudaSuccess) e = small_attrs<kSoup, 2>(&c);
    if (e == cudaSuccess) e = small_attrs<kSoup, 4>(&c);
    if (e == cudaSuccess) e = small_attrs<kMesh, 1>(&c);
    if (e == cudaSuccess) e = small_attrs<kMesh, 2>(&c);
    if (e == cudaSuccess) e = small_attrs<kMesh, 4>(&c);
    if (e != cudaSuccess) cudaGetLastError();
    if (dev >= 0 && dev < 64) g_small_ok[dev].store(e == cudaSuccess && c > 0, std::memory_order_relaxed);
}

cudaError_t launch_small_sort(const float4 *tri, uint32_t n, const HostBounds &hb, Control *ctl, uint32_t *kv,
                              uint32_t *keys, uint32_t *vals, bool stamps, cudaStream_t s) {
    return launch_src<kSoup>(tri, nullptr, 0u, n, hb, ctl, kv, keys, vals, stamps, s);
}

cudaError_t launch_small_sort_mesh(const float4 *verts, uint32_t nverts, const uint32_t *idx3, uint32_t n,
                                   const HostBounds &hb, Control *ctl, uint32_t *kv, uint32_t *keys, uint32_t *vals,
                                   bool stamps, cudaStream_t s) {
    return launch_src<kMesh>(verts, idx3, nverts, n, hb, ctl, kv, keys, vals, stamps, s);
}

}  // namespace lvbh
