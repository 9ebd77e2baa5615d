// The resident sweeps of small and medium grids: see kernels_sor_cluster.cu for
// one thread-block cluster, kernels_sor_grid.cu for CTAs over the whole device.
#pragma once

#include "engine.hpp"

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <set>
#include <tuple>
#include <type_traits>

namespace vb {
namespace resident {

constexpr int kMaxCtas = 16;
constexpr int kSmemLimit = 227 * 1024;
constexpr int kPollLimit = 1 << 22;
constexpr uint32_t kNever = 0xffffffffu;  // a number that no half sweep has

using pair_t = unsigned long long;  // two floats

struct Args {
    int n, hw, groups;       // groups: 4-slot groups per row (hw rounded up)
    int row, planes;         // shared memory: floats per row, planes per colour
    int plane, colour_stride;  // floats per plane and per colour
    int half;                // threads for the rows of one parity and PZ planes, a multiple of 32
    // GRID: row blocks and plane slabs of the CTAs, and the exchange words in
    // global memory (`region` bytes per CTA, then the reduction words), all
    // zero at launch
    int yblocks, zblocks;
    unsigned char* words;
    int region, half_bytes, y_half;  // bytes: per CTA; between the halves of a z word and of a y word
    float omega;
    // by diagonal: mixed, omega / max(d, floor); else the divisor max(d, floor)
    // with 1 / divisor in two floats for the two-product division
    float w[7], relax[7], zh[7], zl[7];
    int two_product;         // it does for the divisors of d = 3 .. 6
    float* xs;
    const float* bs;
    const uint8_t* diag;     // split-layout solid mask or null
    ProjControl* ctrl;
    int subtract_mean;
    int interval;            // sweeps per check
    int flag_nonfinite;      // mixed: a non-finite measured residual stops the solve
    int wait_probe;          // see ProjectionArgs
};

// Threads per CTA: the registers that PZ planes of iterate, right-hand side
// and diagonals leave without spills.
__host__ __device__ constexpr int max_threads(int pz) { return pz == 1 ? 768 : (pz == 2 ? 640 : (pz == 3 ? 576 : 512)); }

// Weights and divisors: one for every cell, by diagonal, by a solid mask.
enum Kind { kUniform = 0, kGeneral = 1, kMasked = 2 };
enum Mode { kFixed = int(SweepMode::kFixed), kTolerance = int(SweepMode::kTolerance), kMixed = int(SweepMode::kMixed) };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t map_to(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void st_remote(uint32_t addr, unsigned long long value) {
    asm volatile("st.shared::cluster.u64 [%0], %1;\n" ::"r"(addr), "l"(value) : "memory");
}

__device__ __forceinline__ pair_t pack2(float a, float b) {
    pair_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
// send4 (below) through global memory.
__device__ __forceinline__ void send4_global(unsigned char* to, int second, const float (&v)[4], uint32_t epoch) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};\n" ::"l"(to), "l"(pack2(v[0], __uint_as_float(epoch))),
                 "l"(pack2(v[1], __uint_as_float(epoch)))
                 : "memory");
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};\n" ::"l"(to + second),
                 "l"(pack2(v[2], __uint_as_float(epoch))), "l"(pack2(v[3], __uint_as_float(epoch)))
                 : "memory");
}
// The 4 words of such a pair of stores: loads of the width of a word, so that a
// value and the number beside it are one access (elements of a vector access
// are separate ones in the PTX memory model).
struct Words {
    pair_t w[4];
    __device__ __forceinline__ uint4 values() const {
        return make_uint4(uint32_t(w[0]), uint32_t(w[1]), uint32_t(w[2]), uint32_t(w[3]));
    }
    __device__ __forceinline__ bool complete(uint32_t epoch) const {
        return uint32_t(w[0] >> 32) == epoch && uint32_t(w[1] >> 32) == epoch && uint32_t(w[2] >> 32) == epoch &&
               uint32_t(w[3] >> 32) == epoch;
    }
};
__device__ __forceinline__ void load_global(const unsigned char* from, pair_t& a, pair_t& b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];\n" : "=l"(a), "=l"(b) : "l"(from) : "memory");
}
__device__ __forceinline__ void load_shared(uint32_t from, pair_t& a, pair_t& b) {
    asm volatile("ld.relaxed.cluster.shared::cta.v2.b64 {%0, %1}, [%2];\n" : "=l"(a), "=l"(b) : "r"(from) : "memory");
}

__device__ __forceinline__ void ld4(const float* p, float (&o)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
}

// 4 values with the half sweep's number into another CTA's shared memory, two
// 16-byte stores of two 8-byte words each; a word is never torn.
__device__ __forceinline__ void send4(uint32_t addr, uint32_t second, const float (&v)[4], uint32_t epoch) {
    const float e = __uint_as_float(epoch);
    asm volatile("st.relaxed.cluster.shared::cluster.v2.b64 [%0], {%1, %2};\n" ::"r"(addr), "l"(pack2(v[0], e)),
                 "l"(pack2(v[1], e))
                 : "memory");
    asm volatile("st.relaxed.cluster.shared::cluster.v2.b64 [%0], {%1, %2};\n" ::"r"(addr + second),
                 "l"(pack2(v[2], e)), "l"(pack2(v[3], e))
                 : "memory");
}
// Waits (bounded) until the 4 words carry `epoch`, then stores their values;
// false when the wait ran out.
__device__ __forceinline__ bool receive4(uint32_t addr, uint32_t second, float* to, uint32_t epoch,
                                         int limit = kPollLimit) {
    // unrolled, the polls' copies cost registers: a half sweep of a fixed budget
    // 1.02 us at 45^3 and 1.61 at 49^3, with one copy 0.95 and 1.38
#pragma unroll 1
    for (int i = 0; i < limit; ++i) {
        Words w;
        load_shared(addr, w.w[0], w.w[1]);
        load_shared(addr + second, w.w[2], w.w[3]);
        if (w.complete(epoch)) {
            *reinterpret_cast<uint4*>(to) = w.values();
            return true;
        }
    }
    return false;
}

// q[j] = t[j] / max(diag[j], floor), diag = 3, 4, 5 or 6. kUniform: the divisor
// is the same for all four and the two-product division applies. One range
// test for the four cells. A zero (frequent once the iterate stands still)
// passes it: its quotient may come out with the other sign, which the sum with
// an iterate that is not -0 does not show, and no iterate that started at +0
// ever is.
template <int KIND>
__device__ __forceinline__ void divide4(const Args& a, const float (&t)[4], const float (&diag)[4], float (&q)[4]) {
    uint32_t lo = 0xffffffffu;  // twice the bits without the sign, less 1: zero wraps to the top
    float hi = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        lo = min(lo, 2u * __float_as_uint(t[j]) - 1u);
        hi = fmaxf(hi, fabsf(t[j]));
    }
    const bool in_range = lo >= 2u * 0x0f800000u - 1u && hi <= 0x1p127f;  // 2^-96
    float y[4], zh[4], zl[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const bool d5 = KIND != kUniform && diag[j] == 5.f, d4 = KIND != kUniform && diag[j] == 4.f,
                   d3 = KIND != kUniform && diag[j] == 3.f;
        y[j] = d5 ? a.relax[5] : (d4 ? a.relax[4] : (d3 ? a.relax[3] : a.relax[6]));
        zh[j] = d5 ? a.zh[5] : (d4 ? a.zh[4] : (d3 ? a.zh[3] : a.zh[6]));
        zl[j] = d5 ? a.zl[5] : (d4 ? a.zl[4] : (d3 ? a.zl[3] : a.zl[6]));
    }
    if ((KIND == kUniform || a.two_product) && in_range) {
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = __fmaf_rn(t[j], zh[j], __fmul_rn(t[j], zl[j]));
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = t[j] / y[j];
    }
}

// The fluid-neighbour counts of 4 slots from the solid mask, one byte each; 0
// where there is nothing to update.
__device__ __forceinline__ uint32_t mask_bytes(const Args& a, int c, int y, int z, int i0) {
    const int s = (y + z + c) & 1;
    uint32_t d = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (i0 + j < a.hw && 2 * (i0 + j) + s < a.n)
            d |= uint32_t(a.diag[(size_t(c) * a.n * a.n + size_t(z) * a.n + y) * a.hw + i0 + j]) << (8 * j);
    return d;
}

// GUARD: 0 every slot of every thread is a cell; 1 (PAD) some slots of the
// padded rows are none; 2 (PART) also, some threads own fewer than PZ planes.
// kMasked in mixed mode only. GRID: CTAs over the whole device, each a block of
// rows and a slab of planes, exchanging through global memory; otherwise one
// cluster of z-slabs.
constexpr int kItems = 3;                // GRID: halo items a thread fetches per half sweep
constexpr int kTable = 5 + 2 * kItems;  // ints per thread (odd: no bank conflicts)
template <int PZ, int MODE, int KIND, int GUARD, bool GRID>
__global__ void __launch_bounds__(max_threads(PZ), 1) k_sor_resident(Args a) {
    constexpr bool EXACT = MODE != kMixed, MASK = KIND == kMasked, PAD = GUARD >= 1, PART = GUARD == 2;
    // [colour][planes: halo below, owned, halo above][n + 2 rows][row], then the halo words
    extern __shared__ __align__(16) float s_x[];
    __shared__ unsigned long long s_red[2][kMaxCtas];
    __shared__ unsigned long long s_warp[32];
    __shared__ int s_bad, s_dead;
    ProjControl* const ctrl = a.ctrl;
    int rank, ctas, yb = 0;  // slab and slabs in z; row block
    if (GRID) {
        ctas = a.zblocks;
        rank = int(blockIdx.x) / a.yblocks;
        yb = int(blockIdx.x) - rank * a.yblocks;
    } else {
        asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
        asm volatile("mov.u32 %0, %%cluster_nctaid.x;\n" : "=r"(ctas));
    }
    if (ctrl->done) return;  // the same for every CTA
    // Read before the CTAs' first rendezvous: the first CTA's last writes to the
    // control block come after it, and nothing else orders a short fixed budget's
    // end there against the start of a CTA far away.
    const int max_iterations = ctrl->max_iterations, start_iterations = ctrl->iterations;
    const int n = a.n, row = a.row, G = a.groups;
    const int yblocks = GRID ? a.yblocks : 1;
    const int ybase = n / yblocks, yrem = n - ybase * yblocks;
    const int nr = GRID ? ybase + (yb < yrem ? 1 : 0) : n;             // rows of this CTA
    const int y0 = GRID ? yb * ybase + min(yb, yrem) : 0;
    const int base = n / ctas, rem = n - base * ctas;
    const int np = base + (rank < rem ? 1 : 0), z0 = rank * base + min(rank, rem);
    const int plane = a.plane, colour_stride = a.colour_stride;
    const int tid = threadIdx.x, threads = blockDim.x, lane = tid & 31, warp = tid >> 5;

    // this thread's slots: the even rows' groups, then from the next warp on
    // the odd rows', so that a warp's rows have their colours in the same places
    const int half = a.half, per_block = 2 * half;
    const int zb = tid / per_block, task = tid - zb * per_block;
    const int odd = task >= half ? 1 : 0, group = task - odd * half;
    const int r = group / G, i0 = (group - r * G) * 4, yl = min(2 * r + odd, nr - 1), y = y0 + yl;
    const int pl0 = zb * PZ;
    const int cnt = 2 * r + odd < nr ? min(PZ, np - pl0) : 0;  // <= 0: no planes
    int row0 = (pl0 + 1) * plane + (yl + 1) * row + i0;
    const bool link_lo = cnt > 0 && pl0 == 0 && rank > 0;                // exchanges with the CTA below
    const bool link_hi = cnt > 0 && pl0 + cnt == np && rank + 1 < ctas;  // ... and above
    // Halo words [side][colour][half][task][16 B]: what the CTA below (side 0)
    // and above (side 1) sent; `task` is also the partner's. Same offsets in
    // every CTA.
    const uint32_t half_bytes = uint32_t(a.half_bytes);
    const uint32_t words = smem_u32(s_x) + 8u * uint32_t(colour_stride) + uint32_t(task) * 16u;
    const uint32_t to_lo = !GRID && rank > 0 ? map_to(words + 4u * half_bytes, rank - 1) : 0u;
    const uint32_t to_hi = !GRID && rank + 1 < ctas ? map_to(words, rank + 1) : 0u;
    // GRID: the same words per CTA in global memory, then those of the rows at
    // the block's ends, [side][colour][half][plane][group][16 B]. Per thread a
    // table in shared memory holds the offsets of its words: those it sends
    // to (below, above, before, behind; -1: none), then its share of those the
    // CTA receives with their places in the halo of colour 0.
    const int y_half = a.y_half, y_words = 8 * a.half_bytes;
    const bool link_ylo = GRID && cnt > 0 && yl == 0 && yb > 0, link_yhi = GRID && cnt > 0 && yl == nr - 1 && yb + 1 < yblocks;
    int table_at = 2 * colour_stride + tid * kTable;  // in ints from s_x
    int* const s_i = reinterpret_cast<int*>(s_x);
    if (GRID) {
        const int mine = int(blockIdx.x) * a.region;
        const int y_at = y_words + (pl0 * G + i0 / 4) * 16;
        s_i[table_at] = link_lo ? mine - yblocks * a.region + 4 * int(half_bytes) + task * 16 : -1;
        s_i[table_at + 1] = link_hi ? mine + yblocks * a.region + task * 16 : -1;
        s_i[table_at + 2] = link_ylo ? mine - a.region + 4 * y_half + y_at : -1;
        s_i[table_at + 3] = link_yhi ? mine + a.region + y_at : -1;
        for (int q = 0; q < kItems; ++q) {
            int from = -1, to = 0, i = tid + q * threads;
            if (i < 2 * per_block) {  // planes below and above
                const int side = i / per_block, other = i - side * per_block;
                const int o = other >= half ? 1 : 0, g = other - o * half, rr = g / G, yy = 2 * rr + o;
                if (yy < nr && (side == 0 ? rank > 0 : rank + 1 < ctas)) {
                    from = mine + side * 4 * int(half_bytes) + other * 16;
                    to = (side ? np + 1 : 0) * plane + (yy + 1) * row + (g - rr * G) * 4;
                }
            } else {  // rows before and behind
                i -= 2 * per_block;
                const int side = i / (np * G), pg = i - side * np * G, pl = pg / G;
                if (side < 2 && (side == 0 ? yb > 0 : yb + 1 < yblocks)) {
                    from = mine + y_words + side * 4 * y_half + pg * 16;
                    to = (pl + 1) * plane + (side ? nr + 1 : 0) * row + (pg - pl * G) * 4;
                }
            }
            s_i[table_at + 4 + 2 * q] = from;
            s_i[table_at + 5 + 2 * q] = to;
        }
    }
    if (tid == 0) {
        s_bad = 0;
        s_dead = 0;
    }
    const int total = 2 * colour_stride + (GRID ? 0 : 32 * per_block);
    for (int i = tid; i < total; i += threads) s_x[i] = 0.f;
    __syncthreads();
    // a wait ran out: no further waits, the next check ends the solve and the
    // error is reported at the end
    bool dead = false;
    if (a.wait_probe > 0) {
        if (!GRID) {
            dead = !receive4(words, half_bytes, s_x + row0, kNever, a.wait_probe);
        } else {
            Words w;
            dead = true;
            for (int i = 0; i < a.wait_probe && dead; ++i) {
                load_global(a.words + size_t(blockIdx.x) * a.region, w.w[0], w.w[1]);
                dead = uint32_t(w.w[0] >> 32) != kNever;
            }
        }
    }
    const size_t rows = size_t(n) * n;
    float X[2][PZ][4], B[2][PZ][4];
    uint32_t D[2][PZ];  // mask_bytes
    const float bm = a.subtract_mean ? ctrl->rhs_mean_f : 0.f;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int k = 0; k < PZ; ++k) {
            D[c][k] = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) X[c][k][j] = B[c][k][j] = 0.f;
            if (k >= cnt) continue;
            const int z = z0 + pl0 + k;
            if (MASK) D[c][k] = mask_bytes(a, c, y, z, i0);
            const size_t g = (c * rows + size_t(z) * n + y) * a.hw + i0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i0 + j < a.hw) {
                    X[c][k][j] = a.xs[g + j];
                    B[c][k][j] = a.subtract_mean ? a.bs[g + j] - bm : a.bs[g + j];
                }
            *reinterpret_cast<float4*>(s_x + c * colour_stride + row0 + k * plane) =
                make_float4(X[c][k][0], X[c][k][1], X[c][k][2], X[c][k][3]);
        }
    if (!GRID) cluster_barrier();  // every CTA's halo words are cleared
    // one plane's updated slots to the neighbours that read them
    auto send = [&](int c, int k, bool bottom, bool top, const float (&v)[4], uint32_t epoch) {
        if (!GRID) {
            if (bottom && link_lo) send4(to_lo + uint32_t(c) * 2u * half_bytes, half_bytes, v, epoch);
            if (top && link_hi) send4(to_hi + uint32_t(c) * 2u * half_bytes, half_bytes, v, epoch);
        } else {
            if (bottom && link_lo) send4_global(a.words + s_i[table_at] + c * 2 * int(half_bytes), int(half_bytes), v, epoch);
            if (top && link_hi) send4_global(a.words + s_i[table_at + 1] + c * 2 * int(half_bytes), int(half_bytes), v, epoch);
            if (link_ylo) send4_global(a.words + s_i[table_at + 2] + c * 2 * y_half + k * G * 16, y_half, v, epoch);
            if (link_yhi) send4_global(a.words + s_i[table_at + 3] + c * 2 * y_half + k * G * 16, y_half, v, epoch);
        }
    };
    // GRID: everything the neighbours sent of colour c in the half sweep
    // numbered `epoch`, into the halo
    auto fetch = [&](int c, uint32_t epoch) {
        // one item after the other (two or three in flight would spill)
#pragma unroll 1
        for (int q = 0; q < kItems; ++q) {
            const int from = s_i[table_at + 4 + 2 * q];
            if (from < 0) continue;
            const int second = tid + q * threads < 2 * per_block ? int(half_bytes) : y_half;
            Words w;
#pragma unroll 1  // as in receive4
            for (int i = 0; !dead; ++i) {
                const unsigned char* const at = a.words + from + c * 2 * second;
                load_global(at, w.w[0], w.w[1]);
                load_global(at + second, w.w[2], w.w[3]);
                if (w.complete(epoch)) {
                    *reinterpret_cast<uint4*>(s_x + c * colour_stride + s_i[table_at + 5 + 2 * q]) = w.values();
                    break;
                }
                if (i == kPollLimit) dead = true;
            }
        }
        __syncthreads();
    };
    // colour 1 as half sweep -1, numbered 1; half sweep t is numbered t + 2
#pragma unroll
    for (int k = 0; k < PZ; ++k)
        if (k < cnt) send(1, k, k == 0, k == cnt - 1, X[1][k], 1u);
    uint32_t t = 0;  // half sweeps done
    float rmax = 0.f;
    unsigned int bad = 0u;
    float dyz = 4.f + float(int(y > 0) + int(y + 1 < n));  // diagonal away from walls in x and z
    // bit 0: parity of y + z of plane 0; bit 1: first group of the row; bits 8
    // ..: plane k lies at a wall in z
    uint32_t flags = uint32_t(y + z0 + pl0) & 1u;
    if (i0 == 0) flags |= 2u;
    int last = a.hw - 1 - i0;  // the row's last slot, from this group's first
#pragma unroll
    for (int k = 0; k < PZ; ++k)
        if (z0 + pl0 + k == 0 || z0 + pl0 + k + 1 == n) flags |= 256u << k;
    const bool even = (n & 1) == 0;
    // one colour's update; MEASURE: with the residual of every updated cell
    auto half_sweep = [&](auto colour, auto measure) {
        constexpr int c = decltype(colour)::value;
        constexpr bool MEASURE = decltype(measure)::value;
        // what follows from these is worked out anew each half sweep: kept
        // across them it would not fit the registers
        asm volatile("" : "+r"(flags), "+f"(dyz), "+r"(last));
        if (GRID || MODE == kTolerance) asm volatile("" : "+r"(row0), "+r"(table_at));
        if (GRID) fetch(1 - c, t + 1u);
        const float* __restrict__ so = s_x + (1 - c) * colour_stride + row0;
        float* __restrict__ sc = s_x + c * colour_stride + row0;
        // the neighbour CTAs' planes into this thread's halo slots
        auto receive = [&]() {
            if (!GRID && (link_lo || link_hi) && !dead) {
                const uint32_t from = words + uint32_t(1 - c) * 2u * half_bytes;
                float* const halo = const_cast<float*>(so);
                if (link_lo) dead = !receive4(from, half_bytes, halo - plane, t + 1u);
                if (link_hi) dead = !receive4(from + 4u * half_bytes, half_bytes, halo + cnt * plane, t + 1u) || dead;
            }
        };
        auto update = [&](auto kk, auto parity) {
            constexpr int k = decltype(kk)::value;
            constexpr bool s = ((decltype(parity)::value + k + c) & 1) != 0;
            if (PART && k >= cnt) return;
            const float* __restrict__ me = so + k * plane;
            float ym[4], yp[4], zm[4], zp[4];
            ld4(me - row, ym);
            ld4(me + row, yp);
            const float edge = s ? me[4] : me[-1];
            if (k > 0) {
#pragma unroll
                for (int j = 0; j < 4; ++j) zm[j] = X[1 - c][k > 0 ? k - 1 : 0][j];
            } else {
                ld4(me - plane, zm);
            }
            if (k + 1 < PZ && (!PART || k + 1 < cnt)) {
#pragma unroll
                for (int j = 0; j < 4; ++j) zp[j] = X[1 - c][k + 1 < PZ ? k + 1 : k][j];
            } else {
                ld4(me + plane, zp);
            }
            const float* o = X[1 - c][k];
            // other-colour cells -1 + s .. 3 + s of this row
            const float e[5] = {s ? o[0] : edge, s ? o[1] : o[0], s ? o[2] : o[1], s ? o[3] : o[2], s ? edge : o[3]};
            const float diag0 = (flags & (256u << k)) ? dyz - 1.f : dyz, diag1 = diag0 - 1.f;
            float diag[4], bo[4], v[4], res[4];
            // slots that are cells: up to the row's last; for odd n the last of s = 1 is none
            const int cells = s && !even ? last - 1 : last;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float off = 0.f;
                off += -1.f * e[j];
                off += -1.f * e[j + 1];
                off += -1.f * ym[j];
                off += -1.f * yp[j];
                off += -1.f * zm[j];
                off += -1.f * zp[j];
                bo[j] = B[c][k][j] - off;
                if (MASK) {
                    diag[j] = float(int(D[c][k] >> (8 * j)) & 0xff);
                } else {
                    // the cell at x = 0 (slot 0, s = 0) and the one at x = n - 1
                    // (the last slot, s = 1 for even n, else 0)
                    bool wall = false;
                    if (j == 0 && !s) wall = flags & 2u;
                    if (PAD) wall |= (s == even) && j == last;
                    else if (j == 3 && s) wall = last == 3;
                    diag[j] = wall ? diag1 : diag0;
                }
                v[j] = bo[j] - diag[j] * X[c][k][j];
            }
            if (EXACT) {
                float q[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = a.omega * v[j];
                divide4<KIND>(a, v, diag, q);
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = X[c][k][j] + q[j];
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float d = diag[j];
                    float w = a.w[6];
                    if (KIND == kGeneral) w = d == 6.f ? w : (d == 5.f ? a.w[5] : (d == 4.f ? a.w[4] : a.w[3]));
                    if (MASK)
                        w = d == 6.f ? w : (d == 5.f ? a.w[5] : (d == 4.f ? a.w[4] : (d == 3.f ? a.w[3] : (d == 2.f ? a.w[2] : a.w[1]))));
                    v[j] = X[c][k][j] + v[j] * w;
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool cell = MASK ? diag[j] > 0.f : (!PAD || j <= cells);
                res[j] = cell ? v[j] : X[c][k][j];
                if (MEASURE && cell) {
                    const float rr = bo[j] - diag[j] * v[j];
                    if (!isfinite(rr)) bad = 1u;
                    rmax = fmaxf(rmax, fabsf(rr));
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) X[c][k][j] = res[j];
            send(c, k, k == 0, PART ? k == cnt - 1 : k == PZ - 1, res, t + 2u);
            *reinterpret_cast<float4*>(sc + k * plane) = make_float4(res[0], res[1], res[2], res[3]);
        };
        // the inner planes while the neighbours' are on their way
        auto sweep = [&](auto parity) {
            using K1 = std::integral_constant<int, (PZ > 2 ? 1 : 0)>;
            using K2 = std::integral_constant<int, (PZ > 3 ? 2 : 0)>;
            if (PZ > 2 && !PART) update(K1{}, parity);
            if (PZ > 3 && !PART) update(K2{}, parity);
            receive();
            update(std::integral_constant<int, 0>{}, parity);
            if (PZ > 2 && PART) update(K1{}, parity);
            if (PZ > 3 && PART) update(K2{}, parity);
            if (PZ > 1) update(std::integral_constant<int, PZ - 1>{}, parity);
        };
        if (cnt > 0) {
            if (flags & 1u) sweep(std::integral_constant<int, 1>{});
            else sweep(std::integral_constant<int, 0>{});
        }
        if (!GRID) __syncthreads();  // GRID: the barrier of the next fetch
        ++t;
    };
    using No = std::false_type;
    using Yes = std::true_type;
    using C0 = std::integral_constant<int, 0>;
    using C1 = std::integral_constant<int, 1>;
    int checks = 0;
    // the largest value over all CTAs (every thread gets it); keys order as the
    // values; bit 63 of the result: some CTA saw `bad` or a wait that ran out
    auto max_of_all = [&](unsigned long long key) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
            key = key < other ? other : key;
        }
        if (bad) atomicOr(&s_bad, 1);
        if (dead) atomicOr(&s_dead, 1);
        if (lane == 0) s_warp[warp] = key;
        __syncthreads();
        auto block_result = [&]() {
            unsigned long long m = 0ull;
            for (int w = 0; w < (threads + 31) / 32; ++w) m = m < s_warp[w] ? s_warp[w] : m;
            if (s_bad || s_dead) m |= 1ull << 63;
            return m;
        };
        unsigned long long m = 0ull, flag = 0ull;
        if (!GRID) {
            if (tid < ctas) st_remote(map_to(smem_u32(&s_red[checks & 1][rank]), tid), block_result());
            cluster_barrier();
            for (int i = 0; i < ctas; ++i) {
                const unsigned long long v = s_red[checks & 1][i];
                flag |= v & (1ull << 63);
                const unsigned long long u = v & ~(1ull << 63);
                m = m < u ? u : m;
            }
        } else {
            // every CTA's result as two numbered words that all CTAs poll
            const int all = int(gridDim.x);
            const uint32_t epoch = uint32_t(checks) + 1u;
            unsigned char* const red = a.words + size_t(all) * a.region + size_t(checks & 1) * all * 16;
            if (tid == 0) {
                const unsigned long long v = block_result();
                const float e = __uint_as_float(epoch);
                asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};\n" ::"l"(red + size_t(blockIdx.x) * 16),
                             "l"(pack2(__uint_as_float(uint32_t(v)), e)), "l"(pack2(__uint_as_float(uint32_t(v >> 32)), e))
                             : "memory");
            }
            unsigned long long most = 0ull, any = 0ull;
            for (int r = tid; r < all; r += threads) {
                pair_t lo = 0, hi = 0;  // half of the result and the number each
                for (int i = 0; (uint32_t(lo >> 32) != epoch || uint32_t(hi >> 32) != epoch) && !dead; ++i) {
                    load_global(red + size_t(r) * 16, lo, hi);
                    if (i == kPollLimit) dead = true;
                }
                const unsigned long long v = (hi << 32) | uint32_t(lo);
                any |= dead ? 1ull << 63 : v & (1ull << 63);
                const unsigned long long u = v & ~(1ull << 63);
                most = most < u ? u : most;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, most, o);
                most = most < other ? other : most;
                any |= __shfl_xor_sync(0xffffffffu, any, o);
            }
            __syncthreads();  // s_warp has been read
            if (lane == 0) s_warp[warp] = most | any;
            __syncthreads();
            for (int w = 0; w < (threads + 31) / 32; ++w) {
                const unsigned long long v = s_warp[w];
                flag |= v & (1ull << 63);
                const unsigned long long u = v & ~(1ull << 63);
                m = m < u ? u : m;
            }
            __syncthreads();
        }
        ++checks;
        return m | flag;
    };

    const bool first_cta = rank == 0 && yb == 0;
    int iterations = start_iterations;
    if (MODE == kFixed) {
        for (int it = iterations; it < max_iterations; ++it) {
            half_sweep(C0{}, No{});
            half_sweep(C1{}, No{});
        }
        if (GRID) max_of_all(0ull);  // every CTA has read the control block
        if (first_cta && tid == 0) {  // the state k_check leaves (no residual is taken)
            ctrl->iterations = max_iterations;
            ctrl->r0 = 0.0;
            ctrl->since = 0;
            ctrl->result.linear_solve.iterations = max_iterations;
            ctrl->result.linear_solve.final_residual = 0.0;
            ctrl->result.linear_solve.converged = 0.0 <= ctrl->target;
            ctrl->done = 1;
            ctrl->continue_flag = 0;
        }
    } else if (MODE == kMixed) {
        const double target = ctrl->target, drop = double(kRecentreDrop) * ctrl->r0;
        const unsigned int nonfinite0 = ctrl->nonfinite & kSolveErrors;
        const int since0 = ctrl->since;
        bool stop = false;
        while (!stop) {
            const int todo = min(a.interval, max_iterations - iterations);
            rmax = 0.f;
            for (int j = 0; j < todo; ++j) {
                half_sweep(C0{}, No{});
                if (j + 1 == a.interval) half_sweep(C1{}, Yes{});
                else half_sweep(C1{}, No{});
            }
            if (!a.flag_nonfinite) bad = 0u;
            const unsigned long long m = max_of_all(__float_as_uint(rmax));
            iterations += todo;
            const float rho = __uint_as_float(uint32_t(m));
            stop = double(rho) <= target || double(rho) <= drop ||
                   since0 + iterations - start_iterations >= kRecentreSweeps || iterations >= max_iterations ||
                   nonfinite0 != 0u || (m >> 63) != 0ull;
        }
        if (first_cta && tid == 0) {  // the state k_error_decide leaves
            ctrl->iterations = iterations;
            ctrl->since = since0 + iterations - start_iterations;
            ctrl->res32_bits = 0u;
            ctrl->recentre = 1;
            ctrl->result.linear_solve.iterations = iterations;
            if (s_bad) atomicOr(&ctrl->nonfinite, 4u);
        }
        if (!first_cta && tid == 0 && s_bad) atomicOr(&ctrl->nonfinite, 4u);
    } else {
        const double target = ctrl->target;
        const unsigned int nonfinite0 = ctrl->nonfinite & kSolveErrors;
        double res = 0.0;
        bool stop = false;
        while (!stop) {
            const int todo = min(a.interval, max_iterations - iterations);
            for (int j = 0; j < todo; ++j) {
                half_sweep(C0{}, No{});
                half_sweep(C1{}, No{});
            }
            iterations += todo;
            // the neighbours' planes into the halo slots: colour 0 as the last
            // half sweep read it, colour 1 after it
            if (GRID) {
                fetch(0, t);
                fetch(1, t + 1u);
            } else if ((link_lo || link_hi) && !dead) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint32_t from = words + uint32_t(c) * 2u * half_bytes, epoch = t + uint32_t(c);
                    float* const halo = s_x + c * colour_stride + row0;
                    if (link_lo) dead = !receive4(from, half_bytes, halo - plane, epoch) || dead;
                    if (link_hi) dead = !receive4(from + 4u * half_bytes, half_bytes, halo + cnt * plane, epoch) || dead;
                }
            }
            // FP64 residual of both colours in the order of StencilLinearSystem.cpp:53-70
            double r = 0.0;
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int k = 0; k < PZ; ++k) {
                    if (k >= cnt) break;
                    // missing neighbours are zeros in shared memory: -1 * 0
                    // leaves the sum's bits unchanged
                    const float* so = s_x + (1 - c) * colour_stride + row0 + k * plane;
                    const int z = z0 + pl0 + k, s = (y + z + c) & 1;
                    float o[4], ym[4], yp[4], zm[4], zp[4];
                    ld4(so, o);
                    ld4(so - row, ym);
                    ld4(so + row, yp);
                    ld4(so - plane, zm);
                    ld4(so + plane, zp);
                    const float edge = s ? so[4] : so[-1];
                    const float e[5] = {s ? o[0] : edge, s ? o[1] : o[0], s ? o[2] : o[1], s ? o[3] : o[2], s ? edge : o[3]};
                    const int dyz2 = int(y > 0) + int(y + 1 < n) + int(z > 0) + int(z + 1 < n);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int x = 2 * (i0 + j) + s;
                        const float xc = X[c][k][j], bi = B[c][k][j];
                        double ax = double(float(int(x > 0) + int(x + 1 < n) + dyz2)) * double(xc);
                        ax += -1.0 * double(e[j]);
                        ax += -1.0 * double(e[j + 1]);
                        ax += -1.0 * double(ym[j]);
                        ax += -1.0 * double(yp[j]);
                        ax += -1.0 * double(zm[j]);
                        ax += -1.0 * double(zp[j]);
                        if (i0 + j < a.hw && x < n) {
                            if (!isfinite(xc) || !isfinite(bi)) bad = 1u;
                            const double d = fabs(double(bi) - ax);
                            r = r < d ? d : r;
                        }
                    }
                }
            const unsigned long long m = max_of_all((unsigned long long)__double_as_longlong(r));
            res = __longlong_as_double((long long)(m & ~(1ull << 63)));
            stop = res <= target || iterations >= max_iterations || nonfinite0 != 0u || (m >> 63) != 0ull;
        }
        if (first_cta && tid == 0) {  // the state k_check leaves
            const int converged = res <= target;
            ctrl->iterations = iterations;
            ctrl->res_bits = 0ull;
            ctrl->r0 = res;
            ctrl->since = 0;
            ctrl->result.linear_solve.iterations = iterations;
            ctrl->result.linear_solve.final_residual = res;
            ctrl->result.linear_solve.converged = converged;
            ctrl->done = 1;
            ctrl->continue_flag = 0;
        }
        if (tid == 0 && s_bad) atomicOr(&ctrl->nonfinite, 4u);
    }
    if (dead) atomicOr(&s_dead, 1);
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int k = 0; k < PZ; ++k) {
            if (k >= cnt) continue;
            float* g = a.xs + (c * rows + size_t(z0 + pl0 + k) * n + y) * a.hw + i0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i0 + j < a.hw) g[j] = X[c][k][j];
        }
    if (GRID) __syncthreads();
    else cluster_barrier();  // the neighbours' last stores have arrived; no CTA is written to after it exits
    if (tid == 0 && s_dead) atomicOr(&ctrl->nonfinite, 8u);
}

// Floats per shared-memory row: at least 4 zeros behind the slots (the x
// neighbours beyond the walls), and as few bank conflicts as 16-byte accesses
// leave: 8 lanes at a time, consecutive groups of consecutive rows of one
// parity.
inline int row_floats(int hwp) {
    const int G = hwp / 4;
    int best = hwp + 4, best_cost = 1 << 30;
    for (int row = hwp + 4; row <= hwp + 16; row += 4) {
        int cost = 0;
        for (int phase = 0; phase < G; ++phase) {
            int used[8] = {}, most = 0;
            for (int lane = 8 * phase; lane < 8 * phase + 8; ++lane)
                most = std::max(most, ++used[(lane / G * 2 * row / 4 + lane % G) % 8]);
            cost += most;
        }
        if (cost < best_cost) {
            best = row;
            best_cost = cost;
        }
    }
    return best;
}

// A launch: CTAs (of one cluster, or over the device), threads and bytes of
// shared memory of each.
struct Shape {
    int ctas, threads, smem;
};
// Launches the kernel of this mode, kind and guard, or with `query` says whether
// the device can hold the launch (sor_resident_launch.cuh).
template <int PZ, bool GRID>
bool launch_planes(Mode mode, int kind, int guard, const Shape& p, const Args& a, bool query, cudaStream_t s);

inline Args make_args(const ProjectionArgs& p, float* x, const float* b, ProjControl* ctrl) {
    Args a{};
    a.n = p.g.n;
    a.hw = (a.n + 1) / 2;
    a.groups = (a.hw + 3) / 4;
    a.omega = p.omega;
    a.two_product = 1;
    for (int d = 0; d < 7; ++d) {
        const float relax = std::max(float(d), p.diagonal_floor);
        a.w[d] = p.omega / relax;
        a.relax[d] = relax;
        if (d >= 3 && !(relax == 3.f || relax == 4.f || relax == 5.f || relax == 6.f)) a.two_product = 0;
        a.zh[d] = float(1.0 / double(relax));
        a.zl[d] = float((1.0 - double(relax) * double(a.zh[d])) / double(relax));
    }
    a.xs = x;
    a.bs = b;
    a.diag = p.diag;
    a.ctrl = ctrl;
    // the z-marching sweep of rows of 4-slot groups knows no diagonal below 3
    // in its table (solid corners): the same weights here
    if (p.diag && a.hw % 4 == 0)
        for (int d = 0; d < 3; ++d) a.w[d] = a.w[3];
    a.interval = p.options.residual_check_interval;
    a.wait_probe = p.wait_probe;
    return a;
}

}  // namespace resident
}  // namespace vb
