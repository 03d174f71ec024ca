// obj.cu - OBJ text -> the build's 48-byte triangle soup and MODEL_BOUNDS, on the device.
//
// Replaces parseObj(file) (scripts/obj/parse-obj.js:3-88) and the OBJFile parser it calls
// (scripts/obj/obj-file-parser.js:19-193), which the demo runs on the main thread before every
// build (main.js:72-73).  The text is parsed in parallel, one thread per line, with the
// reference's semantics:
//   * lines split on '\n' and cut at the first '#'; tokens separated by runs of JavaScript
//     whitespace (`\s`: ASCII \t \n \v \f \r and space, and the UTF-8 forms of U+00A0, U+1680,
//     U+2000-200A, U+2028, U+2029, U+202F, U+205F, U+3000, U+FEFF); keyword lower-cased;
//   * the statements the parser checks fail the parse where the reference throws: g and s with
//     other than one argument (:101-105, :196-201), l with fewer than two vertices or a vertex
//     of more than two '/'-parts (:132-151), f with fewer than three vertices, a vertex of more
//     than three parts or a vertex index parseInt()s to 0 (:153-186);
//   * only model 0 counts (parse-obj.js:17-60): the default model when a v / vt / vn / l / f
//     statement precedes the first `o` (_currentModel, :82-91), else the model the first `o`
//     opens; negative face indices count back from that model's vertices so far, and every
//     index must name one of its vertices (else the reference's array read throws);
//   * vertices are parsed as JavaScript's parseFloat does (longest decimal prefix, correctly
//     rounded), exactly on the device for every decimal exponent within 10^+-27 (see
//     dec_to_double); the rare rest is re-parsed on the host by the C library's correctly
//     rounded strtod;
//   * faces are fan-triangulated from their first vertex, y and z swapped, stored as float32
//     (round to nearest even, the Float32Array of build-bvh.js:14-21), pad 3.1415; bounds are
//     Math.min / Math.max over the faces' vertices in double (NaN absorbs, -0 below +0) from
//     +-1e30, and two floor triangles lie at z_min + .01 (parse-obj.js:62-76).
// Passes: newlines per 16 KB chunk -> scan -> line starts; per-line classify and check with a
// (vertex | triangle) count per block of 256 lines; one block that finds model 0's line range
// and scans those counts over it; vertices; faces -> soup; bounds over the vertices that faces
// used, and the floor.  The per-line passes are bound by instructions per text byte, so the
// forms that exporters write (single spaces, plain decimals, indices that start with 1 to 9) have
// short loops of their own (fast_*), which leave every other line to the general scanners.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "lvbh.h"
#include "lvbh_device.cuh"
#include "lvbh_internal.h"

namespace lvbh {

namespace {

typedef unsigned __int128 u128;

constexpr int kT = 256;
constexpr int kChunk = kT * 64;  // text bytes per newline-count block (64 per thread)
constexpr uint32_t kNone = 0xFFFFFFFFu;

enum : uint8_t { LT_NONE = 0, LT_O, LT_G, LT_V, LT_VT, LT_VN, LT_L, LT_S, LT_F };

// Device state of one parse (set to its initial values by k_nl_count).
struct ObjCtl {
    uint32_t err_line;    // smallest 0-based line whose statement throws (kNone: none)
    uint32_t bad_index;   // a model-0 face names no vertex
    uint32_t num_hard;    // vertex lines left to the host parser
    uint32_t newlines;
    uint32_t m0a, m0b;    // model 0's lines [m0a, m0b)
    uint32_t no_model;    // the text defines no model (output.models[0] is undefined)
    uint32_t done;        // blocks of the bounds pass that have finished
    unsigned long long totals;  // model-0 vertices (low 32 bits) and triangles (high 32 bits)
    unsigned long long bmin[3], bmax[3];  // ordered doubles (ord64)
    uint32_t nan_min[3], nan_max[3];
};

// A vertex line the device leaves to the host: its text [start, end) (up to its comment, or
// further when the device stopped reading before it) and vertex rank.  The same
// slot then carries the host's exact coordinates back (HardFix).
struct HardLine {
    unsigned long long start, end;
    uint32_t vi, pad0;
    uint32_t pad1, pad2;
};
struct HardFix {
    double xyz[3];
    uint32_t vi, pad;
};
static_assert(sizeof(HardLine) == sizeof(HardFix), "hard-line slot");

// Length in bytes of the JavaScript whitespace character at s[i] (0: none), the line ending
// at e.  A UTF-8 lead byte always starts a new character for the decoder of readAsText (an
// unfinished sequence before it becomes U+FFFD), so checking every byte position finds exactly
// the whitespace characters the decoded string holds.
template <typename S>
__host__ __device__ __forceinline__ int ws_len(const S &s, uint64_t i, uint64_t e) {
    const uint8_t c = s[i];
    if (c == ' ' || (c >= 9 && c <= 13)) return 1;
    if (c < 0xC2) return 0;
    if (c == 0xC2) return (i + 1 < e && s[i + 1] == 0xA0) ? 2 : 0;
    if (i + 2 >= e) return 0;
    const uint8_t c1 = s[i + 1], c2 = s[i + 2];
    switch (c) {
        case 0xE1: return (c1 == 0x9A && c2 == 0x80) ? 3 : 0;
        case 0xE2:
            if (c1 == 0x80) return ((c2 >= 0x80 && c2 <= 0x8A) || c2 == 0xA8 || c2 == 0xA9 || c2 == 0xAF) ? 3 : 0;
            return (c1 == 0x81 && c2 == 0x9F) ? 3 : 0;
        case 0xE3: return (c1 == 0x80 && c2 == 0x80) ? 3 : 0;
        case 0xEF: return (c1 == 0xBB && c2 == 0xBF) ? 3 : 0;
    }
    return 0;
}

// Next token of s[i, e): false when none is left; else [a, b).
template <typename S>
__host__ __device__ __forceinline__ bool next_token(const S &s, uint64_t &i, uint64_t e, uint64_t &a,
                                                    uint64_t &b) {
    while (i < e) {
        const int w = ws_len(s, i, e);
        if (!w) break;
        i += w;
    }
    if (i >= e) return false;
    a = i;
    while (i < e && !ws_len(s, i, e)) ++i;
    b = i;
    return true;
}

// Order-preserving map of doubles (-0 below +0) for 64-bit atomic min / max.
__device__ __forceinline__ unsigned long long ord64(double d) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(d);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

__constant__ double kPow10[23] = {1e0,  1e1,  1e2,  1e3,  1e4,  1e5,  1e6,  1e7,
                                  1e8,  1e9,  1e10, 1e11, 1e12, 1e13, 1e14, 1e15,
                                  1e16, 1e17, 1e18, 1e19, 1e20, 1e21, 1e22};

__device__ __forceinline__ int bitlen128(u128 x) {
    const unsigned long long hi = (unsigned long long)(x >> 64), lo = (unsigned long long)x;
    return hi ? 128 - __clzll((long long)hi) : 64 - __clzll((long long)lo);
}

// (x + f) * 2^e2 rounded to the nearest double, ties to even; x has more than 53 bits or
// f == 0, f in [0, 1) is represented by `sticky` = (f != 0).  The result is a normal double.
__device__ double round_scaled(u128 x, int e2, bool sticky) {
    const int nb = bitlen128(x);
    unsigned long long mant;
    int shift = 0;
    if (nb <= 53) {
        mant = (unsigned long long)x;
    } else {
        shift = nb - 53;
        mant = (unsigned long long)(x >> shift);
        const u128 rem = x & (((u128)1 << shift) - 1), half = (u128)1 << (shift - 1);
        if (rem > half || (rem == half && (sticky || (mant & 1)))) ++mant;
        if (mant == (1ull << 53)) { mant >>= 1; ++shift; }
    }
    const double p2 = __longlong_as_double((long long)(e2 + shift + 1023) << 52);
    return __dmul_rn(__ull2double_rn(mant), p2);  // both exact
}

// w * 10^q correctly rounded (w >= 1): false when q lies outside the device's exact range.
// |q| <= 22 with w <= 2^53 is one IEEE multiply or divide of exact doubles (Clinger, "How to
// read floating point numbers accurately", 1990).  Otherwise, for |q| <= 27 (5^27 < 2^63): the
// exact integer w * 5^q scaled by 2^q, or the 128-bit quotient (w * 2^(64 + lz)) / 5^-q with
// its remainder as the sticky bit, rounded once.
__device__ bool dec_to_double(unsigned long long w, int q, double &out) {
    if (w <= (1ull << 53) && q >= -22 && q <= 22) {
        out = q >= 0 ? __dmul_rn((double)w, kPow10[q]) : __ddiv_rn((double)w, kPow10[-q]);
        return true;
    }
    if (q < -27 || q > 27) return false;
    unsigned long long p5 = 1;
    for (int k = 0; k < (q >= 0 ? q : -q); ++k) p5 *= 5;
    if (q >= 0) {
        out = round_scaled((u128)w * p5, q, false);
        return true;
    }
    const int lz = __clzll((long long)w);
    const u128 n = (u128)(w << lz) << 64;
    const u128 quo = n / p5;
    const u128 rem = n - quo * p5;
    out = round_scaled(quo, q - 64 - lz, rem != 0);  // 2^-(64 + lz) * 2^q * 5^q = 10^q / 2^(64+lz)
    return true;
}

// ---- Line scanning on the device.  A line is b[0, e): b is its first byte in a block's
// shared-memory window or in global memory (each kernel inlines the scan once per case, so the
// window case compiles to shared-memory loads), positions are 32-bit, and the first '#' ends the
// line (cut when the scan reaches it).

// Bytes of the JavaScript whitespace character at b[i] (0: none).
__device__ __forceinline__ uint32_t ws32(const uint8_t *b, uint32_t i, uint32_t e) {
    const uint32_t c = b[i];
    if (c <= 32) return (c == 32 || c - 9u <= 4u) ? 1u : 0u;
    if (c < 0xC2) return 0;
    return (uint32_t)ws_len(b, (uint64_t)i, (uint64_t)e);  // the multi-byte forms
}

// Skips whitespace from i: false at the end of the content (the line's end, or a '#', which
// then becomes the end).
__device__ __forceinline__ bool skip_ws(const uint8_t *b, uint32_t &i, uint32_t &e) {
    while (i < e) {
        if (b[i] == '#') {
            e = i;
            return false;
        }
        const uint32_t w = ws32(b, i, e);
        if (!w) return true;
        i += w;
    }
    return false;
}

// Moves i to the end of the token it is in (whitespace, '#' or the end); returns the number of
// '/' bytes passed.
__device__ __forceinline__ uint32_t skip_token(const uint8_t *b, uint32_t &i, uint32_t &e) {
    uint32_t slashes = 0;
    while (i < e) {
        const uint32_t c = b[i];
        if (c == '#') {
            e = i;
            break;
        }
        if ((c <= 32 || c >= 0xC2) && ws32(b, i, e)) break;
        slashes += c == '/';
        ++i;
    }
    return slashes;
}

constexpr long long kIdxNaN = -0x7FFFFFFFFFFFFFFFll - 1;  // parseInt found no digit
constexpr long long kIdxHuge = kIdxNaN + 1;               // |value| >= 2^53: names no vertex

// parseInt (radix undefined) from b[i]: sign, optional 0x / 0X, the longest digit run (what
// parseInt makes of a face vertex's first '/'-part, which ends where the digits do); i is left
// after the digits.  Values of 2^53 and more name no vertex and are not 0, so they collapse to
// kIdxHuge.
__device__ __forceinline__ long long parse_index(const uint8_t *b, uint32_t &i, uint32_t e) {
    bool neg = false;
    if (i < e && (b[i] == '+' || b[i] == '-')) {
        neg = b[i] == '-';
        ++i;
    }
    uint32_t radix = 10;
    if (i + 1 < e && b[i] == '0' && (b[i + 1] | 0x20u) == 'x') {
        radix = 16;
        i += 2;
    }
    unsigned long long v = 0;
    uint32_t digits = 0;
    while (i < e) {
        const uint32_t c = b[i];
        uint32_t d;
        if (c - '0' <= 9u) d = c - '0';
        else if (radix == 16 && (c | 0x20u) - 'a' <= 5u) d = (c | 0x20u) - 'a' + 10;
        else break;
        v = v < (1ull << 53) ? v * radix + d : v;
        ++digits;
        ++i;
    }
    if (!digits) return kIdxNaN;
    if (v >= (1ull << 53)) return kIdxHuge;
    return neg ? -(long long)v : (long long)v;
}

__constant__ uint32_t kPow10u[10] = {1u, 10u, 100u, 1000u, 10000u, 100000u, 1000000u, 10000000u,
                                     100000000u, 1000000000u};

// parseFloat from b[i], a token's first byte: true with the double in out, false when the host
// parses it (decimal exponent beyond +-27, or more than 19 significant digits whose dropped
// tail could change the rounding); i is left where the literal ends.  Significant digits
// accumulate nine at a time in 32 bits.
__device__ __forceinline__ bool parse_number(const uint8_t *b, uint32_t &i, uint32_t e, double &out) {
    bool neg = false;
    if (i < e && (b[i] == '+' || b[i] == '-')) {
        neg = b[i] == '-';
        ++i;
    }
    if (i + 8 <= e && b[i] == 'I' && b[i + 1] == 'n' && b[i + 2] == 'f' && b[i + 3] == 'i' &&
        b[i + 4] == 'n' && b[i + 5] == 'i' && b[i + 6] == 't' && b[i + 7] == 'y') {
        i += 8;
        out = neg ? -INFINITY : INFINITY;
        return true;
    }
    unsigned long long m = 0;  // folded significant digits
    uint32_t acc = 0, na = 0;  // digits not folded yet (at most 9)
    uint32_t nd = 0;           // significant digits kept (at most 19)
    long long dexp = 0;
    bool any = false, inexact = false, frac = false;
    while (i < e) {
        const uint32_t c = b[i];
        const uint32_t d = c - '0';
        if (d > 9u) {
            if (c == '.' && !frac) {
                frac = true;
                ++i;
                continue;
            }
            break;
        }
        any = true;
        if (nd < 19) {
            if (nd | d) {
                acc = acc * 10 + d;
                ++nd;
                if (++na == 9) {
                    m = m * 1000000000ull + acc;
                    acc = 0;
                    na = 0;
                }
            }
            dexp -= frac;
        } else {
            dexp += !frac;
            inexact |= d != 0;
        }
        ++i;
    }
    if (!any) {
        out = NAN;
        return true;
    }
    m = m * kPow10u[na] + acc;
    long long e10 = 0;
    if (i < e && (b[i] | 0x20u) == 'e') {
        uint32_t j = i + 1;
        bool eneg = false;
        if (j < e && (b[j] == '+' || b[j] == '-')) {
            eneg = b[j] == '-';
            ++j;
        }
        long long ev = 0;
        uint32_t ed = 0;
        while (j < e && b[j] - '0' <= 9u) {
            if (ev < 1000000000ll) ev = ev * 10 + (b[j] - '0');
            ++j;
            ++ed;
        }
        if (ed) {
            e10 = eneg ? -ev : ev;
            i = j;
        }
    }
    if (m == 0) {
        out = neg ? -0.0 : 0.0;
        return true;
    }
    const long long q = e10 + dexp;
    if (q < -27 || q > 27) return false;
    double v;
    if (!dec_to_double(m, (int)q, v)) return false;
    if (inexact) {  // the value lies strictly between m * 10^q and (m + 1) * 10^q
        double hi;
        if (!dec_to_double(m + 1, (int)q, hi) || hi != v) return false;
    }
    out = neg ? -v : v;
    return true;
}

constexpr int kLineBlock = 256;     // lines per block of the per-line kernels
constexpr int kWindow = 16 * 1024;  // text bytes a block stages in shared memory

// A thread's line l of a block's lines [l0, l0 + kLineBlock), and the text the block stages:
// positions fit 32 bits (LVBH_OBJ_MAX_BYTES).  Their loads depend on nothing but the line number,
// so they are in flight together with a kernel's other first loads.
struct LineText {
    uint32_t p, q;    // the line's bytes [p, q) (without the '\n'; nothing past the last line)
    uint32_t w0, w1;  // the window: from the 16-byte boundary at or below the first line's start, as
                      // much of the block's text as fits
    __device__ __forceinline__ LineText(const uint32_t *__restrict__ line_start, uint32_t L, uint32_t l0, uint64_t n) {
        const uint32_t l = l0 + threadIdx.x, last = min(L, l0 + kLineBlock);
        p = l < L ? line_start[l] : 0u;
        q = l + 1 < L ? line_start[l + 1] - 1u : l < L ? (uint32_t)n : 0u;
        w0 = line_start[l0] & ~15u;
        const uint32_t z = last < L ? line_start[last] : (uint32_t)n;
        w1 = w0 + min(z - w0, (uint32_t)kWindow);
    }
    // [w0, w1) of the text into win, all 16-byte copies in flight together.  Every thread calls it.
    __device__ __forceinline__ void stage(const uint8_t *__restrict__ text, uint64_t n, uint8_t *win) const {
        const uint32_t len = w1 - w0, rest = (uint32_t)n - w0;
        for (uint32_t o = 16u * threadIdx.x; o < len; o += 16u * kLineBlock) {
            if (o + 16u <= rest) {
                cp_async16(win + o, text + w0 + o);
            } else {
                for (uint32_t k = 0; k < 16; ++k)
                    if (o + k < rest) win[o + k] = text[w0 + o + k];
            }
        }
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
    }
    __device__ __forceinline__ uint32_t len() const { return q - p; }
    __device__ __forceinline__ bool whole() const { return p >= w0 && q < w1; }  // the line and its newline
    __device__ __forceinline__ bool body() const { return p >= w0 && q <= w1; }  // the line
};

__device__ __forceinline__ uint8_t lower(uint8_t c) { return (c >= 'A' && c <= 'Z') ? c + 32 : c; }

__device__ __forceinline__ uint8_t keyword(const uint8_t *b, uint32_t a, uint32_t z) {
    const uint32_t n = z - a;
    if (n == 1) {
        switch (lower(b[a])) {
            case 'o': return LT_O;
            case 'g': return LT_G;
            case 'v': return LT_V;
            case 'l': return LT_L;
            case 's': return LT_S;
            case 'f': return LT_F;
        }
    } else if (n == 2 && lower(b[a]) == 'v') {
        if (lower(b[a + 1]) == 't') return LT_VT;
        if (lower(b[a + 1]) == 'n') return LT_VN;
    }
    return LT_NONE;
}

// Exclusive scan of one value per thread across the block (blockDim.x a multiple of 32).
template <typename U>
__device__ __forceinline__ U block_scan(U x, U *s_warp, U *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    U incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const U y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    U off = 0, all = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
        off += i < warp ? s_warp[i] : (U)0;
        all += s_warp[i];
    }
    __syncthreads();
    if (total) *total = all;
    return off + incl - x;
}

// Smallest value over the warp into *dst (atomically), skipping kNone and values that cannot
// lower it, so that one word shared by the grid sees few atomics.
__device__ __forceinline__ void warp_min_into(uint32_t v, uint32_t *dst) {
    v = __reduce_min_sync(0xFFFFFFFFu, v);
    if ((threadIdx.x & 31) == 0 && v != kNone && v < *(volatile uint32_t *)dst) atomicMin(dst, v);
}

// The 64 text bytes of thread threadIdx.x of chunk blockIdx.x (zero past the end): four
// 16-byte loads; newline count by a SWAR zero-byte test on each word.
__device__ __forceinline__ void load64(const uint8_t *__restrict__ s, uint64_t n, uint64_t p, uint4 (&v)[4]) {
    if (p + 64 <= n) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = __ldg(reinterpret_cast<const uint4 *>(s + p) + j);  // read again: keep it in L2
    } else {
        uint8_t *b = reinterpret_cast<uint8_t *>(v);
        for (int k = 0; k < 64; ++k) b[k] = p + k < n ? s[p + k] : 0;
    }
}

__device__ __forceinline__ uint32_t newlines_in(uint32_t w) {
    const uint32_t x = w ^ 0x0A0A0A0Au;  // zero bytes where '\n' was
    return __popc(~(((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x | 0x7F7F7F7Fu));
}

// The newline bytes of w as four bits.
__device__ __forceinline__ uint32_t newline_nibble(uint32_t w) {
    const uint32_t x = w ^ 0x0A0A0A0Au, y = ~(((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x | 0x7F7F7F7Fu);
    return ((y >> 7) * 0x10204080u) >> 28;  // bits 7, 15, 23, 31 -> 0, 1, 2, 3
}

__device__ __forceinline__ uint32_t newlines64(const uint4 (&v)[4]) {
    uint32_t c = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) c += newlines_in(v[j].x) + newlines_in(v[j].y) + newlines_in(v[j].z) + newlines_in(v[j].w);
    return c;
}

// Newlines per kChunk bytes (64 per thread); the control block's initial values.
__global__ void __launch_bounds__(kT) k_nl_count(const uint8_t *__restrict__ s, uint64_t n,
                                                 uint32_t *__restrict__ cnt, ObjCtl *__restrict__ ctl) {
    __shared__ uint32_t w[kT / 32];
    if (blockIdx.x == 0) {
        for (uint32_t i = threadIdx.x; i < sizeof(ObjCtl) / 4; i += kT) reinterpret_cast<uint32_t *>(ctl)[i] = 0u;
        __syncthreads();
        if (threadIdx.x == 0) ctl->err_line = kNone;
        if (threadIdx.x < 3) ctl->bmin[threadIdx.x] = ~0ull;
    }
    uint4 v[4];
    load64(s, n, (uint64_t)blockIdx.x * kChunk + threadIdx.x * 64ull, v);
    const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, newlines64(v));
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int i = 0; i < kT / 32; ++i) t += w[i];
        cnt[blockIdx.x] = t;
    }
}

// Exclusive scan of v[0, n) in place by one block, each thread over a run of consecutive
// entries; *total = the sum.
template <typename U>
__global__ void __launch_bounds__(1024) k_scan_small(U *v, uint32_t n, U *total) {
    __shared__ U s_warp[32];
    chain_wait();
    const uint32_t per = (n + 1023) / 1024, b = threadIdx.x * per, e = min(n, b + per);
    U sum = 0;
    for (uint32_t i = b; i < e; ++i) sum += v[i];
    U all;
    U run = block_scan<U>(sum, s_warp, &all);
    for (uint32_t i = b; i < e; ++i) {
        const U x = v[i];
        v[i] = run;
        run += x;
    }
    if (threadIdx.x == 0) *total = all;
}

// Line starts: the newline at byte k (rank r over the text) starts line r + 1 at k + 1.  At most
// `cap` lines are written (the caller sees from the count that there are more).  Before chain_wait it
// reads the text only, complete before k_nl_count began, for which k_scan_small has waited.
__global__ void __launch_bounds__(kT) k_nl_write(const uint8_t *__restrict__ s, uint64_t n,
                                                 const uint32_t *__restrict__ base, uint32_t cap,
                                                 uint32_t *__restrict__ line_start) {
    __shared__ uint32_t s_warp[kT / 32];
    const uint64_t p = (uint64_t)blockIdx.x * kChunk + threadIdx.x * 64ull;
    uint4 v[4];
    load64(s, n, p, v);
    // bit k: byte k is a newline
    unsigned long long m = 0;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(v);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t bits = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) bits |= newline_nibble(w[8 * h + j]) << (4 * j);
        m |= (unsigned long long)bits << (32 * h);
    }
    const uint32_t before = block_scan<uint32_t>((uint32_t)__popcll((long long)m), s_warp, nullptr);
    chain_wait();
    uint32_t r = base[blockIdx.x] + before;
    while (m) {
        const int k = __ffsll((long long)m) - 1;
        if (++r < cap) line_start[r] = (uint32_t)p + k + 1;
        m &= m - 1;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) line_start[0] = 0;
}

struct LineClass {
    uint8_t type;
    bool bad;
    uint32_t fan;
};

// Statement type of the line b[0, len), whether the reference's parser throws on it (g / s
// with other than one argument, l with fewer than two vertices or a vertex of more than two
// '/'-parts, f with fewer than three vertices, a vertex of more than three parts or a first
// part parseInt()s to 0 or -0), and the triangles a face fans into.
__device__ __forceinline__ LineClass classify(const uint8_t *b, uint32_t len) {
    uint32_t i = 0, e = len;
    if (!skip_ws(b, i, e)) return {LT_NONE, false, 0};
    const uint32_t a = i;
    skip_token(b, i, e);
    const uint8_t t = keyword(b, a, i);
    if (t == LT_NONE || t == LT_V || t == LT_VT || t == LT_VN || t == LT_O) return {t, false, 0};  // no checks
    uint32_t ntok = 1;
    bool bad = false;
    while (skip_ws(b, i, e)) {
        ++ntok;
        if (t == LT_F) {
            bad |= parse_index(b, i, e) == 0;
            bad |= skip_token(b, i, e) > 2;
        } else if (t == LT_L) {
            bad |= skip_token(b, i, e) > 1;
        } else {
            skip_token(b, i, e);
        }
    }
    if ((t == LT_G || t == LT_S) && ntok != 2) bad = true;
    if (t == LT_L && ntok < 3) bad = true;
    uint32_t fan = 0;
    if (t == LT_F) {
        if (ntok < 4) bad = true;
        else fan = ntok - 3;
    }
    return {t, bad, fan};
}

// The class of a line in its common forms: empty, comment, `v ` / `vt ` / `vn ` (no checks), and
// `f` with tokens apart by spaces that start with 1 to 9 (an index that parseInt makes neither 0
// nor NaN) and hold ASCII without '#'.  b[len] is the line's '\n'.  False: classify() decides.
__device__ __forceinline__ bool fast_class(const uint8_t *b, LineClass &r) {
    r = LineClass{LT_NONE, false, 0};
    const uint32_t c0 = b[0];
    if (c0 == '\n' || c0 == '#') return true;
    const uint32_t c1 = b[1];  // at most the '\n'
    if (c0 == 'v') {
        if (c1 == ' ') { r.type = LT_V; return true; }
        if ((c1 == 't' || c1 == 'n') && b[2] == ' ') { r.type = c1 == 't' ? LT_VT : LT_VN; return true; }
        return false;
    }
    if (c0 != 'f' || c1 != ' ') return false;
    r.type = LT_F;
    uint32_t i = 1, ntok = 0, c = ' ';
    for (;;) {
        while (c == ' ') c = b[++i];
        if (c == '\n') break;
        if (c == '\r' && b[i + 1] == '\n') break;
        if (c - '1' > 8u) return false;
        ++ntok;
        do c = b[++i];
        while (c - '0' <= 9u);
        if (c == '/') {
            uint32_t slashes = 1;
            do {
                c = b[++i];
                slashes += c == '/';
            } while (c > ' ' && c < 0x80 && c != '#');
            r.bad |= slashes > 2;
        }
        if (c != ' ' && c != '\n' && c != '\r') return false;
    }
    if (ntok < 3) r.bad = true;
    else r.fan = ntok - 2;
    return true;
}

// What k_lines leaves per block of kLineBlock lines (an array each): packed counts of all its
// lines (vertices in the low, triangles in the high 32 bits), its first two `o` lines and its
// first model-creating one (kNone: none).
struct LineBlocks {
    unsigned long long *count;
    uint32_t *o1, *o2, *need;
};

// Per line: its class.  One block per kLineBlock lines, their text staged in shared memory.
__global__ void __launch_bounds__(kLineBlock, 8) k_lines(const uint8_t *__restrict__ text, uint64_t n,
                                                      const uint32_t *__restrict__ line_start, uint32_t cap,
                                                      uint8_t *__restrict__ type, uint32_t *__restrict__ fans,
                                                      LineBlocks blocks, ObjCtl *__restrict__ ctl) {
    __shared__ __align__(16) uint8_t win[kWindow];
    __shared__ unsigned long long s_count[kLineBlock / 32];
    __shared__ uint32_t s_o[kLineBlock / 32], s_need[kLineBlock / 32];
    chain_wait();
    const uint32_t L = ctl->newlines + 1u, l0 = blockIdx.x * kLineBlock, l = l0 + threadIdx.x;
    if (L > cap || l0 >= L) return;  // more lines than there is room for: the caller comes again
    const LineText lt(line_start, L, l0, n);
    lt.stage(text, n, win);
    LineClass c{LT_NONE, false, 0};
    if (l < L) {
        if (lt.whole()) {
            if (!fast_class(win + (lt.p - lt.w0), c)) c = classify(win + (lt.p - lt.w0), lt.len());
        } else {
            c = classify(text + lt.p, lt.len());
        }
        type[l] = c.type;
        fans[l] = c.fan;
    }
    warp_min_into(c.bad ? l : kNone, &ctl->err_line);
    const bool need = c.type == LT_V || c.type == LT_VT || c.type == LT_VN || c.type == LT_L || c.type == LT_F;
    const uint32_t nv = __popc(__ballot_sync(0xFFFFFFFFu, c.type == LT_V));
    const uint32_t nt = __reduce_add_sync(0xFFFFFFFFu, c.type == LT_F ? c.fan : 0u);
    const uint32_t no = __ballot_sync(0xFFFFFFFFu, c.type == LT_O), nn = __ballot_sync(0xFFFFFFFFu, need);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        s_count[warp] = (unsigned long long)nt << 32 | nv;
        s_o[warp] = no;
        s_need[warp] = nn;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long count = 0;
        uint32_t o1 = kNone, o2 = kNone, first_need = kNone;
        for (int w = kLineBlock / 32 - 1; w >= 0; --w) {
            count += s_count[w];
            const uint32_t at = l0 + 32 * w, o = s_o[w];
            if (s_need[w]) first_need = at + __ffs(s_need[w]) - 1;
            if (o) {
                const uint32_t rest = o & (o - 1);
                o2 = rest ? at + __ffs(rest) - 1 : o1;
                o1 = at + __ffs(o) - 1;
            }
        }
        blocks.count[blockIdx.x] = count;
        blocks.o1[blockIdx.x] = o1;
        blocks.o2[blockIdx.x] = o2;
        blocks.need[blockIdx.x] = first_need;
    }
}

// Packed count of a model-0 line: one vertex (low 32 bits) or a face's triangles (high).
__device__ __forceinline__ unsigned long long line_count(uint8_t t, uint32_t fan) {
    return t == LT_V ? 1ull : t == LT_F ? (unsigned long long)fan << 32 : 0ull;
}

// Model 0's lines [a, b): the default model when a model-creating statement precedes the first `o`
// (_currentModel, obj-file-parser.js:82-91), else the model that `o` opens, up to the next `o`.
// Then pre[block]: the packed counts of model 0's lines before the block.  One block of threads;
// a line block that a or b cuts is counted line by line.
__global__ void __launch_bounds__(1024) k_model(LineBlocks blocks, const uint8_t *__restrict__ type,
                                                const uint32_t *__restrict__ fans, uint32_t cap,
                                                unsigned long long *__restrict__ pre, ObjCtl *__restrict__ ctl) {
    __shared__ uint32_t s_min[3][32];
    __shared__ unsigned long long s_warp[32];
    chain_wait();
    const uint32_t L = ctl->newlines + 1u;
    if (L > cap) return;
    const uint32_t nb = (L + (kLineBlock - 1)) / kLineBlock;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto block_min = [&](uint32_t v, int slot) {
        v = __reduce_min_sync(0xFFFFFFFFu, v);
        if (lane == 0) s_min[slot][warp] = v;
        __syncthreads();
        return __reduce_min_sync(0xFFFFFFFFu, s_min[slot][lane]);
    };
    // a thread's two smallest first-`o` lines and its smallest model-creating line
    uint32_t o1 = kNone, o2 = kNone, need = kNone;
#pragma unroll 8
    for (uint32_t i = threadIdx.x; i < nb; i += 1024) {
        const uint32_t o = blocks.o1[i];
        o2 = min(o2, max(o1, o));
        o1 = min(o1, o);
        need = min(need, blocks.need[i]);
    }
    const uint32_t fo = block_min(o1, 0), fn = block_min(need, 1);
    uint32_t so = o1 == fo ? o2 : o1;
    if (threadIdx.x == 0 && fo != kNone) so = min(so, blocks.o2[fo / kLineBlock]);
    so = block_min(so, 2);
    uint32_t a = 0, b = 0, none = 0;
    if (fn != kNone && (fo == kNone || fn < fo)) {
        b = fo == kNone ? L : fo;
    } else if (fo != kNone) {
        a = fo;
        b = so == kNone ? L : so;
    } else {
        none = 1;
    }
    // the line blocks that a and b lie in (the same one, or a is at its block's start, at times)
    const uint32_t ba = a / kLineBlock, bb = b / kLineBlock;
    // threads 0 .. 255 count block ba's lines of model 0, threads 256 .. 511 block bb's
    const uint32_t half = threadIdx.x / kLineBlock, l = (half ? bb : ba) * kLineBlock + threadIdx.x % kLineBlock;
    unsigned long long c = 0, ca = 0, cb = 0;
    if (half < 2 && l >= a && l < b) c = line_count(type[l], fans[l]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    if (lane == 0) s_warp[warp] = c;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kLineBlock / 32; ++w) {
        ca += s_warp[w];
        cb += s_warp[kLineBlock / 32 + w];
    }
    __syncthreads();
    // a warp's 512 line blocks in four rows of 128, four consecutive ones per lane (whole lines per
    // access: with 16 consecutive ones per thread the one SM's requests took 16 us of the kernel's
    // 21 for 12,300 line blocks)
    constexpr int kRows = 4;
    unsigned long long all = 0;
    for (uint32_t base = 0; base < nb; base += 1024u * 4 * kRows) {
        unsigned long long x[kRows][4], run[kRows], sum = 0;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const uint32_t i = base + (warp * kRows + r) * 128u + 4u * lane;
#pragma unroll
            for (int k = 0; k < 4; k += 2) {
                ulonglong2 v = make_ulonglong2(0ull, 0ull);
                if (i + k + 1 < nb) v = *reinterpret_cast<const ulonglong2 *>(blocks.count + i + k);
                else if (i + k < nb) v.x = blocks.count[i + k];
                x[r][k] = v.x;
                x[r][k + 1] = v.y;
            }
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            unsigned long long four = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t i = base + (warp * kRows + r) * 128u + 4u * lane + k;
                if (i < ba || i > bb) x[r][k] = 0ull;
                if (i == bb) x[r][k] = cb;
                if (i == ba) x[r][k] = ca;
                four += x[r][k];
            }
            unsigned long long incl = four;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += y;
            }
            run[r] = sum + incl - four;  // before this lane's four, within the warp
            sum += __shfl_sync(0xFFFFFFFFu, incl, 31);
        }
        if (lane == 0) s_warp[warp] = sum;
        __syncthreads();
        unsigned long long off = all;
        for (int w = 0; w < 32; ++w) {
            off += w < warp ? s_warp[w] : 0ull;
            all += s_warp[w];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const uint32_t i = base + (warp * kRows + r) * 128u + 4u * lane;
            unsigned long long p4[4], c4 = off + run[r];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                p4[k] = c4;
                c4 += x[r][k];
            }
#pragma unroll
            for (int k = 0; k < 4; k += 2) {
                if (i + k + 1 < nb) *reinterpret_cast<ulonglong2 *>(pre + i + k) = make_ulonglong2(p4[k], p4[k + 1]);
                else if (i + k < nb) pre[i + k] = p4[k];
            }
        }
    }
    if (threadIdx.x == 0) {
        ctl->m0a = a;
        ctl->m0b = b;
        ctl->no_model = none;
        ctl->totals = all;
    }
}

struct VertexParse {
    double x, y, z;
    uint32_t end;  // where the scan stopped (the content's end when a number was left over)
    bool ok;
};

// The coordinates of the vertex line b[0, len) (missing ones 0, as _parseVertexCoords has it).
__device__ __forceinline__ VertexParse parse_vertex(const uint8_t *b, uint32_t len) {
    VertexParse r{0.0, 0.0, 0.0, len, true};
    uint32_t i = 0, e = len;
    skip_ws(b, i, e);
    skip_token(b, i, e);  // the keyword
    if (skip_ws(b, i, e)) {
        r.ok &= parse_number(b, i, e, r.x);
        skip_token(b, i, e);
        if (skip_ws(b, i, e)) {
            r.ok &= parse_number(b, i, e, r.y);
            skip_token(b, i, e);
            if (skip_ws(b, i, e)) {
                r.ok &= parse_number(b, i, e, r.z);
                skip_token(b, i, e);
            }
        }
    }
    r.end = e;
    return r;
}

// The coordinates of a vertex line in its common form: `v`, then three plain decimals of at most
// nine digits apart by spaces (value = digits / 10^k, one IEEE division of exact doubles, as
// dec_to_double has it).  b[len] is the line's '\n'.  False: parse_vertex() decides.
__device__ __forceinline__ bool fast_vertex(const uint8_t *b, double (&out)[3]) {
    if (b[0] != 'v' || b[1] != ' ') return false;
    uint32_t i = 1, c = ' ';
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (c != ' ') return false;
        while (c == ' ') c = b[++i];
        const bool neg = c == '-';
        if (neg) c = b[++i];
        uint32_t m = 0, d, at = i;  // (m wraps past nine digits: not used then)
        while ((d = c - '0') <= 9u) {
            m = m * 10 + d;
            c = b[++i];
        }
        uint32_t nd = i - at, k = 0;
        if (c == '.') {
            c = b[at = ++i];
            while ((d = c - '0') <= 9u) {
                m = m * 10 + d;
                c = b[++i];
            }
            k = i - at;
            nd += k;
        }
        if (nd - 1u > 8u || (c != ' ' && c != '\n' && c != '\r')) return false;
        const double v = k ? __ddiv_rn((double)m, kPow10[k]) : (double)m;
        out[a] = neg ? -v : v;
    }
    return true;
}

// float32 of a coordinate as Float32Array stores it (NaN as the quiet NaN 0x7FC00000).
__device__ __forceinline__ float to_f32(double d) {
    return isnan(d) ? __int_as_float(0x7FC00000) : __double2float_rn(d);
}

// A vertex as the soup holds it: x, the file's z as y and y as z, and the pad.
__device__ __forceinline__ float4 soup_row(double x, double y, double z) {
    return make_float4(to_f32(x), to_f32(z), to_f32(y), __double2float_rn(3.1415));
}

// Model 0's vertices by rank: their doubles, their soup rows, and whether a face names them.
struct Verts {
    double *xyz;
    float4 *row;
    uint8_t *used;
};

// Model-0 vertex lines -> doubles and soup rows at their rank; numbers outside the device's
// exact range are listed for the host.  Block i has the lines of line block blk0 + i, its text
// staged when it holds a vertex line of model 0's lines [a, b).
__global__ void __launch_bounds__(kLineBlock, 8) k_vertices(const uint8_t *__restrict__ text, uint64_t n,
                                                         const uint32_t *__restrict__ line_start, uint32_t L,
                                                         const uint8_t *__restrict__ type, uint32_t blk0, uint32_t a,
                                                         uint32_t b, const unsigned long long *__restrict__ pre,
                                                         Verts vs, HardLine *__restrict__ hard,
                                                         ObjCtl *__restrict__ ctl) {
    __shared__ __align__(16) uint8_t win[kWindow];
    __shared__ uint32_t s_v[kLineBlock / 32];
    const uint32_t blk = blk0 + blockIdx.x, l0 = blk * kLineBlock, l = l0 + threadIdx.x;
    const LineText lt(line_start, L, l0, n);
    uint32_t vi = (uint32_t)pre[blk];
    const bool mine = l >= a && l < b && type[l] == LT_V;
    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, mine);
    if ((threadIdx.x & 31) == 0) s_v[threadIdx.x >> 5] = __popc(bal);
    if (!__syncthreads_or(mine)) return;
    lt.stage(text, n, win);
    if (!mine) return;
    vi += __popc(bal & lanemask_lt());
    for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) vi += s_v[w];
    double c[3];
    if (!(lt.whole() && fast_vertex(win + (lt.p - lt.w0), c))) {
        VertexParse r;
        if (lt.body()) r = parse_vertex(win + (lt.p - lt.w0), lt.len());
        else r = parse_vertex(text + lt.p, lt.len());
        c[0] = r.x;
        c[1] = r.y;
        c[2] = r.z;
        if (!r.ok) {
            const uint32_t h = atomicAdd(&ctl->num_hard, 1u);
            hard[h] = HardLine{lt.p, (unsigned long long)lt.p + r.end, vi, 0u, 0u, 0u};
        }
    }
    vs.xyz[3ull * vi] = c[0];
    vs.xyz[3ull * vi + 1] = c[1];
    vs.xyz[3ull * vi + 2] = c[2];
    vs.row[vi] = soup_row(c[0], c[1], c[2]);
    vs.used[vi] = 0;
}

__global__ void __launch_bounds__(kT) k_patch(const HardFix *__restrict__ fix, uint32_t count, Verts vs) {
    const uint32_t i = blockIdx.x * kT + threadIdx.x;
    if (i >= count) return;
    const HardFix f = fix[i];
    vs.xyz[3ull * f.vi] = f.xyz[0];
    vs.xyz[3ull * f.vi + 1] = f.xyz[1];
    vs.xyz[3ull * f.vi + 2] = f.xyz[2];
    vs.row[f.vi] = soup_row(f.xyz[0], f.xyz[1], f.xyz[2]);
}

// A face's fan, one vertex after the other: stores triangles (first, previous, current).
struct Fan {
    float4 first, prev;
    float4 *tri;
    uint32_t nv = 0;
    // vertex vk (0-based, the model's): false when the model has no such vertex
    __device__ __forceinline__ bool add(uint32_t vk, uint32_t nverts, const Verts &vs) {
        if (vk >= nverts) return false;
        vs.used[vk] = 1;
        const float4 cur = vs.row[vk];
        if (nv == 0) {
            first = cur;
        } else if (nv >= 2) {
            tri[0] = first;
            tri[1] = prev;
            tri[2] = cur;
            tri += 3;
        }
        prev = cur;
        ++nv;
        return true;
    }
};

// The face line b[0, len): its vertices resolved (negative indices against `before`, the
// model's vertices so far) and fanned; false when an index names no vertex.
__device__ __forceinline__ bool emit_face(const uint8_t *b, uint32_t len, long long before, uint32_t nverts,
                                          const Verts &vs, float4 *tri) {
    uint32_t i = 0, e = len;
    skip_ws(b, i, e);
    skip_token(b, i, e);  // the keyword
    Fan fan;
    fan.tri = tri;
    while (skip_ws(b, i, e)) {
        long long v = parse_index(b, i, e);
        skip_token(b, i, e);
        if (v == kIdxNaN || v == kIdxHuge) return false;
        if (v < 0) v = before + 1 + v;  // vertices.length + 1 + vertexIndex
        const long long vk = v - 1;
        if (vk < 0 || vk >= (long long)nverts) return false;
        fan.add((uint32_t)vk, nverts, vs);
    }
    return true;
}

// The same for the common form (as fast_class has it, indices of at most nine digits); done:
// false when emit_face has to do the line (again from its start: it stores the same triangles).
__device__ __forceinline__ bool fast_face(const uint8_t *b, uint32_t nverts, const Verts &vs, float4 *tri, bool &done) {
    done = false;
    if (b[0] != 'f' || b[1] != ' ') return true;
    Fan fan;
    fan.tri = tri;
    uint32_t i = 1, c = ' ';
    for (;;) {
        while (c == ' ') c = b[++i];
        if (c == '\n') break;
        if (c == '\r' && b[i + 1] == '\n') break;
        uint32_t v = c - '0', d;
        const uint32_t at = i;
        if (v - 1u > 8u) return true;
        while ((d = (c = b[++i]) - '0') <= 9u) v = v * 10 + d;
        if (i - at > 9) return true;  // v may have wrapped
        if (c == '/') {
            do c = b[++i];
            while (c > ' ' && c < 0x80 && c != '#');
        }
        if (c != ' ' && c != '\n' && c != '\r') return true;
        if (!fan.add(v - 1u, nverts, vs)) {
            done = true;
            return false;
        }
    }
    done = true;
    return true;
}

// Model-0 faces -> fan triangles (y and z swapped, float32, pad 3.1415), their vertices marked.
// Blocks as k_vertices.  Before chain_wait it reads the text and what obj_scan's kernels wrote (lines,
// types, fans, prefixes): the host has waited for those before it launched k_vertices, which writes
// none of them.
__global__ void __launch_bounds__(kLineBlock, 8) k_faces(const uint8_t *__restrict__ text, uint64_t n,
                                                      const uint32_t *__restrict__ line_start, uint32_t L,
                                                      const uint8_t *__restrict__ type,
                                                      const uint32_t *__restrict__ fans, uint32_t blk0, uint32_t a,
                                                      uint32_t b, const unsigned long long *__restrict__ pre,
                                                      uint32_t nverts, Verts vs, float4 *__restrict__ tri,
                                                      ObjCtl *__restrict__ ctl) {
    __shared__ __align__(16) uint8_t win[kWindow];
    __shared__ uint32_t s_warp[kLineBlock / 32], s_v[kLineBlock / 32];
    const uint32_t blk = blk0 + blockIdx.x, l0 = blk * kLineBlock, l = l0 + threadIdx.x;
    const LineText lt(line_start, L, l0, n);
    const unsigned long long first = pre[blk];
    const bool in = l >= a && l < b;
    const uint8_t ty = in ? type[l] : (uint8_t)LT_NONE;
    const uint32_t fan = in ? fans[l] : 0u;
    const bool mine = ty == LT_F;
    const uint32_t vbal = __ballot_sync(0xFFFFFFFFu, ty == LT_V);
    if ((threadIdx.x & 31) == 0) s_v[threadIdx.x >> 5] = __popc(vbal);
    uint32_t at = 0;
    if (__syncthreads_or(mine)) {
        at = (uint32_t)(first >> 32) + block_scan<uint32_t>(mine ? fan : 0u, s_warp, nullptr);
        lt.stage(text, n, win);
    }
    chain_wait();  // the vertices; every block's, so that k_bounds_floor's wait stands for k_vertices too
    if (!mine) return;
    float4 *out = tri + 3ull * at;
    bool ok = true, done = false;
    if (lt.whole()) ok = fast_face(win + (lt.p - lt.w0), nverts, vs, out, done);
    if (!done) {
        uint32_t before = (uint32_t)first + __popc(vbal & lanemask_lt());  // model-0 vertices so far
        for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) before += s_v[w];
        if (lt.body()) ok = emit_face(win + (lt.p - lt.w0), lt.len(), before, nverts, vs, out);
        else ok = emit_face(text + lt.p, lt.len(), before, nverts, vs, out);
    }
    if (!ok) atomicOr(&ctl->bad_index, 1u);
}

// Math.min / Math.max over the vertices that faces name (x, the file's z, y; -0 below +0, NaN
// absorbs), and, in the last block to finish, the floor (parse-obj.js:62-76): two triangles at
// z_min + .01, 10000 out in x and y, after the model's triangles; z_min = Math.min from 1e30.
__global__ void __launch_bounds__(kT) k_bounds_floor(Verts vs, uint32_t nverts, float4 *__restrict__ tri_floor,
                                                     ObjCtl *__restrict__ ctl) {
    __shared__ unsigned long long s_mn[3][kT / 32], s_mx[3][kT / 32];
    __shared__ int s_nan[3][kT / 32];
    __shared__ bool s_last;
    chain_wait();
    unsigned long long mn[3] = {~0ull, ~0ull, ~0ull}, mx[3] = {0ull, 0ull, 0ull};
    bool nan[3] = {false, false, false};
    for (uint32_t v = blockIdx.x * kT + threadIdx.x; v < nverts; v += gridDim.x * kT) {
        const bool used = vs.used[v] != 0;  // (read with the coordinates: one wait)
        const double *p = vs.xyz + 3ull * v;
        const double c[3] = {p[0], p[2], p[1]};
        if (!used) continue;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            if (isnan(c[ax])) {
                nan[ax] = true;
                continue;
            }
            const unsigned long long o = ord64(c[ax]);
            mn[ax] = o < mn[ax] ? o : mn[ax];
            mx[ax] = o > mx[ax] ? o : mx[ax];
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        unsigned long long lo = mn[ax], hi = mx[ax];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long lo2 = __shfl_xor_sync(0xFFFFFFFFu, lo, o);
            const unsigned long long hi2 = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
            lo = lo2 < lo ? lo2 : lo;
            hi = hi2 > hi ? hi2 : hi;
        }
        const int nan_any = __any_sync(0xFFFFFFFFu, nan[ax]);
        if (lane == 0) { s_mn[ax][warp] = lo; s_mx[ax][warp] = hi; s_nan[ax][warp] = nan_any; }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int ax = threadIdx.x;
        unsigned long long lo = ~0ull, hi = 0ull;
        int nan_any = 0;
        for (int w = 0; w < kT / 32; ++w) {
            lo = s_mn[ax][w] < lo ? s_mn[ax][w] : lo;
            hi = s_mx[ax][w] > hi ? s_mx[ax][w] : hi;
            nan_any |= s_nan[ax][w];
        }
        // (few blocks still move the words that all of them would queue on)
        if (lo != ~0ull && lo < *(volatile unsigned long long *)&ctl->bmin[ax]) atomicMin(&ctl->bmin[ax], lo);
        if (hi != 0ull && hi > *(volatile unsigned long long *)&ctl->bmax[ax]) atomicMax(&ctl->bmax[ax], hi);
        if (nan_any) {
            atomicOr(&ctl->nan_min[ax], 1u);
            atomicOr(&ctl->nan_max[ax], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atom_add_acq_rel_gpu(&ctl->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    const int v = threadIdx.x;  // 6 vertices
    if (v == 0) ctl->done = 0u;
    if (v >= 6) return;
    const unsigned long long zo = __ldcg(&ctl->bmin[2]);
    double zmin = 1e30;
    if (__ldcg(&ctl->nan_min[2])) {
        zmin = NAN;
    } else if (zo != ~0ull) {
        const double d = __longlong_as_double((long long)((zo >> 63) ? (zo & 0x7FFFFFFFFFFFFFFFull) : ~zo));
        zmin = d < 1e30 ? d : 1e30;
    }
    const float h = to_f32(__dadd_rn(zmin, .01)), f = 10000.0f, pad = __double2float_rn(3.1415);
    const float xs[6] = {-f, f, -f, f, f, -f}, ys[6] = {-f, -f, f, -f, f, f};
    tri_floor[v] = make_float4(xs[v], ys[v], h, pad);
}

// parseFloat of a whitespace-free token on the host, for the numbers the device leaves to it:
// the C library's correctly rounded strtod on the longest decimal prefix.
double host_parse_float(const uint8_t *t, size_t len) {
    size_t i = 0;
    bool neg = false;
    if (i < len && (t[i] == '+' || t[i] == '-')) { neg = t[i] == '-'; ++i; }
    if (len - i >= 8 && std::memcmp(t + i, "Infinity", 8) == 0) return neg ? -INFINITY : INFINITY;
    const size_t st = i;
    size_t digits = 0;
    while (i < len && t[i] >= '0' && t[i] <= '9') { ++i; ++digits; }
    if (i < len && t[i] == '.') {
        ++i;
        while (i < len && t[i] >= '0' && t[i] <= '9') { ++i; ++digits; }
    }
    if (!digits) return NAN;
    size_t end = i;
    if (i < len && (t[i] == 'e' || t[i] == 'E')) {
        size_t j = i + 1;
        if (j < len && (t[j] == '+' || t[j] == '-')) ++j;
        size_t ed = 0;
        while (j < len && t[j] >= '0' && t[j] <= '9') { ++j; ++ed; }
        if (ed) end = j;
    }
    const std::string lit(reinterpret_cast<const char *>(t) + st, end - st);
    const double v = std::strtod(lit.c_str(), nullptr);
    return neg ? -v : v;
}

double ord64_inv(unsigned long long o) {
    const unsigned long long u = (o >> 63) ? (o & 0x7FFFFFFFFFFFFFFFull) : ~o;
    double d;
    std::memcpy(&d, &u, 8);
    return d;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Grow one scratch block to at least `need` bytes (contents are not kept).
cudaError_t grow(void *&p, size_t &have, size_t need) {
    if (need <= have) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    have = 0;
    const cudaError_t e = cudaMalloc(&p, need);
    if (e == cudaSuccess) have = need;
    return e;
}

}  // namespace

#define OBJ_CUDA(call, what)                          \
    do {                                              \
        if (int rc_ = cuda((call), what)) return rc_; \
    } while (0)

namespace {

int obj_cuda(cudaError_t e, const char *what, std::string &err) {
    if (e == cudaSuccess) return LVBH_OK;
    cudaGetLastError();
    err = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? LVBH_ENOMEM : LVBH_ECUDA;
}

}  // namespace

int obj_scan(ObjScratch &sc, const char *text, uint64_t bytes, bool host_text, uint32_t *num_tris, uint64_t *err_line,
             cudaStream_t s, std::string &err) {
    auto cuda = [&](cudaError_t e, const char *what) { return obj_cuda(e, what, err); };
    auto reject = [&](uint64_t line, const std::string &msg) {
        *err_line = line;
        err = msg;
        return LVBH_EPARSE;
    };
    *err_line = 0;
    sc.scanned = false;
    if (!sc.host) OBJ_CUDA(cudaMallocHost(&sc.host, sizeof(ObjCtl)), "cudaMallocHost");
    ObjCtl *hc = static_cast<ObjCtl *>(sc.host);
    // text (staged when it is host memory or not 16-byte aligned), control block, newline
    // counts per chunk
    const uint32_t chunks = bytes ? (uint32_t)((bytes + kChunk - 1) / kChunk) : 1u;
    const bool stage = host_text || (reinterpret_cast<uintptr_t>(text) & 15u);
    const size_t text_part = stage ? align256(bytes) : 0;
    OBJ_CUDA(grow(sc.text, sc.text_bytes, text_part + align256(sizeof(ObjCtl)) + align256((chunks + 1) * 4ull)),
             "cudaMalloc(obj text)");
    const uint8_t *d_text = reinterpret_cast<const uint8_t *>(text);
    char *c = static_cast<char *>(sc.text);
    if (stage) {
        if (bytes) OBJ_CUDA(cudaMemcpyAsync(c, text, bytes, host_text ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, s),
                            "cudaMemcpyAsync(text)");
        d_text = reinterpret_cast<const uint8_t *>(c);
        c += text_part;
    }
    ObjCtl *ctl = reinterpret_cast<ObjCtl *>(c);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(c + align256(sizeof(ObjCtl)));
    k_nl_count<<<chunks, kT, 0, s>>>(d_text, bytes, cnt, ctl);
    launch_chained(true, k_scan_small<uint32_t>, 1, 1024, 0, s, cnt, chunks, &ctl->newlines);
    // lines, model 0 and the vertex / triangle prefixes in one stream-ordered run, for as many lines
    // as a text of this size usually has at most; one with more of them (seen from the count)
    // runs again.  Whole calls on device text (B200): 16.5 MB in lines of 11 bytes 250 us so, 224 with
    // room for its lines at once, 1.3 MB 106 and 87; at bytes / 8, 47 MB in lines of 32 bytes 199 us
    // instead of 189 (empty blocks of k_lines), 28 MB of 19 bytes 160 instead of 158
    uint32_t cap = (uint32_t)std::min<uint64_t>(bytes / 16 + 4096, 0xFFFFFFFEull);
    for (;;) {
        const uint32_t nb = cap / kLineBlock + 1;
        const size_t starts = align256((cap + 1ull) * 4), types = align256(cap), fan_part = align256(cap * 4ull);
        const size_t b8 = align256(nb * 8ull), b4 = align256(nb * 4ull);
        OBJ_CUDA(grow(sc.lines, sc.lines_bytes, starts + types + fan_part + 2 * b8 + 3 * b4),
                 "cudaMalloc(obj lines)");
        char *cl = static_cast<char *>(sc.lines);
        sc.line_start = reinterpret_cast<uint32_t *>(cl);
        sc.type = reinterpret_cast<uint8_t *>(cl + starts);
        sc.fans = reinterpret_cast<uint32_t *>(cl + starts + types);
        cl += starts + types + fan_part;
        sc.pre = reinterpret_cast<unsigned long long *>(cl);
        const LineBlocks blocks{reinterpret_cast<unsigned long long *>(cl + b8), reinterpret_cast<uint32_t *>(cl + 2 * b8),
                                reinterpret_cast<uint32_t *>(cl + 2 * b8 + b4),
                                reinterpret_cast<uint32_t *>(cl + 2 * b8 + 2 * b4)};
        launch_chained(true, k_nl_write, chunks, kT, 0, s, d_text, bytes, cnt, cap, sc.line_start);
        launch_chained(true, k_lines, (cap + kLineBlock - 1) / kLineBlock, kLineBlock, 0, s, d_text, bytes, sc.line_start,
                       cap, sc.type, sc.fans, blocks, ctl);
        launch_chained(true, k_model, 1, 1024, 0, s, blocks, sc.type, sc.fans, cap, sc.pre, ctl);
        OBJ_CUDA(cudaGetLastError(), "k_lines");
        OBJ_CUDA(cudaMemcpyAsync(hc, ctl, sizeof(ObjCtl), cudaMemcpyDeviceToHost, s), "readback");
        OBJ_CUDA(cudaStreamSynchronize(s), "cudaStreamSynchronize");
        if (hc->newlines + 1ull <= cap) break;
        cap = hc->newlines + 1u;  // at most LVBH_OBJ_MAX_BYTES + 1
    }
    if (hc->err_line != kNone)
        return reject(hc->err_line + 1ull, "line " + std::to_string(hc->err_line + 1ull) +
                                                ": a statement the OBJ parser rejects");
    if (hc->no_model) return reject(0, "the OBJ text defines no model");
    const uint64_t nfan = hc->totals >> 32;
    if (nfan + 2 > LVBH_MAX_TRIS) return reject(0, "the OBJ text makes more than LVBH_MAX_TRIS triangles");
    *num_tris = (uint32_t)nfan + 2;
    sc.scanned = true;
    sc.src = text;
    sc.d_text = d_text;
    sc.src_bytes = bytes;
    sc.host_text = host_text;
    sc.ctl = ctl;
    return LVBH_OK;
}

int obj_emit(ObjScratch &sc, float *dst, uint32_t max_tris, const float **tri_out, double *bounds6, uint64_t *err_line,
             cudaStream_t s, std::string &err) {
    auto cuda = [&](cudaError_t e, const char *what) { return obj_cuda(e, what, err); };
    *err_line = 0;
    if (!sc.scanned) {
        err = "no scanned OBJ text";
        return LVBH_EINVAL;
    }
    ObjCtl *hc = static_cast<ObjCtl *>(sc.host), *ctl = static_cast<ObjCtl *>(sc.ctl);
    const uint32_t L = hc->newlines + 1u, a = hc->m0a, b = hc->m0b;
    const uint32_t nverts = (uint32_t)(hc->totals & 0xFFFFFFFFull), nfan = (uint32_t)(hc->totals >> 32);
    if (dst && nfan + 2u > max_tris) {  // the scan stays: the caller may come again with more room
        err = "the soup has " + std::to_string(nfan + 2u) + " triangles, the caller's memory holds " + std::to_string(max_tris);
        return LVBH_EINVAL;
    }
    sc.scanned = false;
    const uint32_t blk0 = a / kLineBlock, nblk = b > a ? (b - 1) / kLineBlock - blk0 + 1 : 0;
    const size_t xyz = align256(nverts * 24ull), rows = align256(nverts * 16ull), used = align256(nverts);
    OBJ_CUDA(grow(sc.verts, sc.verts_bytes, xyz + rows + used + align256(nverts * (size_t)sizeof(HardLine))),
             "cudaMalloc(obj vertices)");
    if (!dst) {
        OBJ_CUDA(grow(sc.soup, sc.soup_bytes, align256((nfan + 2ull) * 48)), "cudaMalloc(obj soup)");
        dst = static_cast<float *>(sc.soup);
    }
    char *cv = static_cast<char *>(sc.verts);
    float4 *tri = reinterpret_cast<float4 *>(dst);
    const Verts vs{reinterpret_cast<double *>(cv), reinterpret_cast<float4 *>(cv + xyz),
                   reinterpret_cast<uint8_t *>(cv + xyz + rows)};
    HardLine *hard = reinterpret_cast<HardLine *>(cv + xyz + rows + used);
    const uint8_t *d_text = sc.d_text;
    const uint64_t bytes = sc.src_bytes;
    // vertices, faces, bounds and floor, then one read-back; numbers the device left to the host
    // (rare) are patched in and the faces, bounds and floor run again
    auto faces_bounds_floor = [&](bool chain) {
        if (nfan)
            launch_chained(chain && nverts, k_faces, nblk, kLineBlock, 0, s, d_text, bytes, sc.line_start, L, sc.type, sc.fans,
                           blk0, a, b, sc.pre, nverts, vs, tri, ctl);
        const uint32_t want = (nverts + kT - 1) / kT, most = (uint32_t)sm_count() * 8u;
        const uint32_t grid = want < 1 ? 1 : want < most ? want : most;
        launch_chained(true, k_bounds_floor, grid, kT, 0, s, vs, nverts, tri + 3ull * nfan, ctl);
    };
    if (nverts)
        k_vertices<<<nblk, kLineBlock, 0, s>>>(d_text, bytes, sc.line_start, L, sc.type, blk0, a, b, sc.pre, vs, hard, ctl);
    faces_bounds_floor(true);
    OBJ_CUDA(cudaGetLastError(), "k_faces");
    OBJ_CUDA(cudaMemcpyAsync(hc, ctl, sizeof(ObjCtl), cudaMemcpyDeviceToHost, s), "readback");
    OBJ_CUDA(cudaStreamSynchronize(s), "cudaStreamSynchronize");
    const uint32_t nh = nverts ? hc->num_hard : 0;
    if (nh) {
        std::vector<HardLine> hl(nh);
        OBJ_CUDA(cudaMemcpyAsync(hl.data(), hard, nh * sizeof(HardLine), cudaMemcpyDeviceToHost, s), "readback");
        OBJ_CUDA(cudaStreamSynchronize(s), "cudaStreamSynchronize");
        std::vector<HardFix> fix(nh);
        std::vector<uint8_t> buf;
        for (uint32_t h = 0; h < nh; ++h) {
            uint64_t len = hl[h].end - hl[h].start;
            const uint8_t *ln = reinterpret_cast<const uint8_t *>(sc.src) + hl[h].start;
            if (!sc.host_text) {
                buf.resize(len);
                if (len) OBJ_CUDA(cudaMemcpy(buf.data(), d_text + hl[h].start, len, cudaMemcpyDeviceToHost), "readback");
                ln = buf.data();
            }
            const void *hash = len ? std::memchr(ln, '#', len) : nullptr;  // the comment cut
            if (hash) len = static_cast<const uint8_t *>(hash) - ln;
            uint64_t k = 0, ta = 0, tb = 0;
            next_token(ln, k, len, ta, tb);  // the keyword
            HardFix f{{0.0, 0.0, 0.0}, hl[h].vi, 0u};
            for (int ax = 0; ax < 3; ++ax) {
                if (!next_token(ln, k, len, ta, tb)) break;
                f.xyz[ax] = host_parse_float(ln + ta, tb - ta);
            }
            fix[h] = f;
        }
        HardFix *dfix = reinterpret_cast<HardFix *>(hard);
        OBJ_CUDA(cudaMemcpyAsync(dfix, fix.data(), nh * sizeof(HardFix), cudaMemcpyHostToDevice, s),
                 "cudaMemcpyAsync(fix)");
        k_patch<<<(nh + kT - 1) / kT, kT, 0, s>>>(dfix, nh, vs);
        // the bounds and the index check start over
        for (int ax = 0; ax < 3; ++ax) {
            hc->bmin[ax] = ~0ull;
            hc->bmax[ax] = 0ull;
            hc->nan_min[ax] = hc->nan_max[ax] = 0u;
        }
        hc->bad_index = 0u;
        OBJ_CUDA(cudaMemcpyAsync(ctl, hc, sizeof(ObjCtl), cudaMemcpyHostToDevice, s), "cudaMemcpyAsync(ctl)");
        faces_bounds_floor(false);
        OBJ_CUDA(cudaGetLastError(), "k_faces");
        OBJ_CUDA(cudaMemcpyAsync(hc, ctl, sizeof(ObjCtl), cudaMemcpyDeviceToHost, s), "readback");
        OBJ_CUDA(cudaStreamSynchronize(s), "cudaStreamSynchronize");  // also: `fix` is pageable
    }
    if (hc->bad_index) {
        err = "a face of model 0 names a vertex the model does not have";
        return LVBH_EPARSE;
    }
    // bounds: Math.min / Math.max from 1e30 / -1e30 over the faces' vertices
    for (int ax = 0; ax < 3; ++ax) {
        const double lo = hc->bmin[ax] == ~0ull ? 1e30 : ord64_inv(hc->bmin[ax]);
        const double hi = hc->bmax[ax] == 0ull ? -1e30 : ord64_inv(hc->bmax[ax]);
        bounds6[ax] = hc->nan_min[ax] ? NAN : (lo < 1e30 ? lo : 1e30);
        bounds6[3 + ax] = hc->nan_max[ax] ? NAN : (hi > -1e30 ? hi : -1e30);
    }
    if (tri_out) *tri_out = dst;
    return LVBH_OK;
}
#undef OBJ_CUDA

void obj_free(ObjScratch &sc) {
    if (sc.text) cudaFree(sc.text);
    if (sc.lines) cudaFree(sc.lines);
    if (sc.soup) cudaFree(sc.soup);
    if (sc.verts) cudaFree(sc.verts);
    if (sc.host) cudaFreeHost(sc.host);
    sc = ObjScratch{};
}

}  // namespace lvbh
