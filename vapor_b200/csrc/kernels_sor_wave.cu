// Two red+black iterations (four half sweeps) of the divide-free relaxation in
// one pass over a large grid: the mixed solver's sweeps and the FPCG
// preconditioner's smoothing on unmasked grids with n % 8 == 0.
//
// One launch per colour reads iterate and right-hand side anew for every colour:
// at 256^3, where they (134 MB) do not stay in L2, the two launches of an
// iteration move 224 MB, 13.4 bytes a cell, in 46 us. The latency of the
// neighbour rows' loads bounds them, at 59% of the DRAM throughput and 64% of the
// issue slots (cache hints and a serpentine order of the planes changed the time
// by less than 5%). This pass reads both once for two iterations: 199 MB, 6 bytes
// a cell and iteration.
//
// A CTA owns a tile of 64 cells in x by up to 56 rows in y and a chunk of planes,
// and marches up the chunk: at step tau plane tau arrives, half sweep t = 1 .. 4
// updates its colour in plane tau - t, and plane tau - 4 is written. A thread
// holds 4 slots of a row in both colours: a half sweep finds its own column (the
// cell, the planes above and below) in registers and the x and y neighbours in
// shared memory, where they were published one step before, so that one
// rendezvous of the warps per plane is enough. The planes arrive by TMA a step
// ahead (rows, slots and planes outside the grid as 0); the right-hand side stays
// in a ring of planes for the half sweeps that follow. The tile has a halo of a
// 4-slot group in x (what TMA can align; 4 cells are needed), 4 rows and 4 planes
// on each side: every half sweep invalidates one more ring of cells.
//
// All four half sweeps of a step meet a row with the same parity s, and a warp's
// rows have one parity (kept together in shared memory too), so a warp runs code
// in which the x neighbours, the wall slots and the ring positions are fixed:
// some 300 instructions a step for 16 cell updates. A warp arrives at the
// rendezvous once it has loaded what half sweep 4 needs and waits for it before
// it publishes half sweep 1 (the warps that fetch wait first), so half of a step
// runs while others are behind.
//
// Bound by shared memory (1760 wavefronts of 2690 cycles a step; the L1 pipe is
// 74% busy) and issue (65%), no longer by DRAM (39%): 62.8 us a pass at 256^3. Measured, staged mixed
// projection, per iteration in all, one-colour launches against this pass: 136^3
// 19.1 / 16.4 us, 160^3 23.0 / 18.6, 192^3 31.7 / 22.8, 224^3 47.2 / 31.1, 256^3
// 58.0 / 38.3 (of which the sweeps 46 / 31). Moving the planes with 8-byte
// cp.async instead of TMA took 128 us a pass, twice as long.
//
// The update of every cell is k_sor_rbz's: the same operations in the same order
// up to signs, so the results are the same bit for bit. It is out of place
// (neighbouring tiles read each other's cells as halo).
#include "engine.hpp"
#include "tc_conv.cuh"

#include <algorithm>
#include <cudaTypedefs.h>
#include <map>
#include <mutex>
#include <set>
#include <type_traits>

namespace vb {
namespace {

constexpr int kGroups = 10;                 // 4-slot groups per tile row: 8 owned, one of halo each side
constexpr int kRow = 4 * kGroups;           // floats per row in shared memory
constexpr int kRows = 32;                   // rows of one parity (at most)
constexpr int kHalo = 4;                    // rows and planes
constexpr int kPad = 64;                    // floats before a block: a row and a value beyond its ends stay in bounds
constexpr int kBlock = kPad + kRows * kRow; // floats: the rows of one parity of one plane
constexpr int kPlane = 2 * kBlock;          // one colour of one plane of the tile
// shared memory, in planes: second colour (ring of 4), first colour (2),
// published half sweeps 1 .. 3 (2 each), right-hand side of either colour (4)
constexpr int kXB = 0, kXA = 4, kPub = 6, kBA = 12, kBB = 16, kPlanes = 20;
constexpr int kSmem = (kPlanes * kPlane + kPad) * 4;
constexpr int kHalf = kRows * kGroups;      // threads per row parity: 10 warps
constexpr int kThreads = 2 * kHalf;
constexpr int kWaitLimit = 1 << 20;
constexpr int kDrainLimit = 1 << 14;

struct WaveArgs {
    int n, hw;
    int rows;                // of one parity in a tile, halo included
    int ytile, zchunk;       // rows and planes owned by a CTA
    int first;               // colour of the first half sweep
    float w[7];              // omega / max(d, floor)
    float* xout;
    const float* q;          // DOT: the vector of the second product
    double* partials;        // DOT: 2 per CTA, z.b and z.q
    ProjControl* ctrl;
    int guarded, sweep_index;
    int wait_probe;          // see ProjectionArgs
};

__device__ __forceinline__ void load_rows(uint32_t dst, const CUtensorMap* map, int x, int parity, int row, int z,
                                          int colour, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
        "%6}], [%7];\n" ::"r"(dst),
        "l"(map), "r"(x), "r"(parity), "r"(row), "r"(z), "r"(colour), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void ld4(const float* p, float (&o)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
}
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void copy4(float (&a)[4], const float (&b)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) a[j] = b[j];
}

struct Near {
    float ym[4], yp[4], b[4], edge;
};
// a += b, two lanes at a time (each rounded by itself)
__device__ __forceinline__ void add4(float (&a)[4], const float (&b)[4]) {
#pragma unroll
    for (int j = 0; j < 4; j += 2)
        asm("{\n .reg .b64 u, v;\n mov.b64 u, {%0, %1};\n mov.b64 v, {%2, %3};\n add.rn.f32x2 u, u, v;\n"
            " mov.b64 {%0, %1}, u;\n}\n"
            : "+f"(a[j]), "+f"(a[j + 1])
            : "f"(b[j]), "f"(b[j + 1]));
}

// FROM_ZERO: the iterate starts as 0 and is not read. RESID: the largest
// residual of the last half sweep's cells into ctrl->res32_bits. DOT: FP64
// partials of z.b and z.q over both colours of the result.
template <bool FROM_ZERO, bool RESID, bool DOT>
__global__ void __launch_bounds__(kThreads, 1) k_sor_wave(const __grid_constant__ CUtensorMap xmap,
                                                          const __grid_constant__ CUtensorMap bmap, WaveArgs a) {
    extern __shared__ __align__(128) float s_mem[];
    __shared__ float s_max[32];
    __shared__ double s_sum[32];
    __shared__ uint64_t s_full[2], s_go, s_probe;
    __shared__ int s_fetched[8];  // per fetching warp, the last step it fetched for
    const int n = a.n, hw = a.hw;
    int sweeps = 2;
    if (a.guarded) {
        const int left = a.ctrl->max_iterations - a.ctrl->iterations - a.sweep_index;
        sweeps = a.ctrl->done ? 0 : max(0, min(2, left));
    }
    const int tid = threadIdx.x, lane = tid & 31;
    const int odd = tid >= kHalf ? 1 : 0, task = tid - odd * kHalf;
    const int r = task / kGroups, g = task - r * kGroups;
    const int y0 = blockIdx.y * a.ytile, y = y0 - kHalo + 2 * r + odd;  // ytile is even
    const int x0 = blockIdx.x * 32 - 4, slot0 = x0 + 4 * g;
    const int z0 = blockIdx.z * a.zchunk, z1 = min(n, z0 + a.zchunk);
    const bool there = r < a.rows && y >= 0 && y < n && slot0 >= 0 && slot0 < hw;
    const bool own = there && r >= kHalo / 2 && r < a.rows - kHalo / 2 && g > 0 && g < kGroups - 1;
    const bool left_wall = slot0 == 0, right_wall = slot0 + 4 == hw;
    const int cA = a.first, cB = 1 - a.first;
    const int plane_floats = n * hw;
    const uint32_t smem = static_cast<uint32_t>(__cvta_generic_to_shared(s_mem));
    const uint32_t full = static_cast<uint32_t>(__cvta_generic_to_shared(s_full));
    const uint32_t go = static_cast<uint32_t>(__cvta_generic_to_shared(&s_go));
    const uint32_t probe = static_cast<uint32_t>(__cvta_generic_to_shared(&s_probe));
    const int mine = odd * kBlock + kPad + r * kRow + 4 * g;          // this thread's slots in a plane
    const int ym_at = (odd ? mine - kBlock : mine + kBlock - kRow);   // rows before and behind: the other parity's
    const int yp_at = (odd ? mine - kBlock + kRow : mine + kBlock);
    constexpr int kLoads = FROM_ZERO ? 4 : 8;
    if (tid == 0) {
        tc::mbar_init(full, kLoads);
        tc::mbar_init(full + 8, kLoads);
        tc::mbar_init(go, kThreads / 32);
        tc::mbar_init(probe, 1);
        tc::fence_mbarrier_init();
    }
    for (int i = tid; i < kPlanes * kPlane + kPad; i += kThreads) s_mem[i] = 0.f;
    tc::fence_proxy_async();
    __syncthreads();

    const int tau0 = z0 - kHalo;
    const int steps = z1 > z0 ? z1 - z0 + 2 * kHalo : 0;
    // Arrivals for step k (tau = tau0 + k): second colour in plane tau, first
    // colour and its right-hand side in tau - 1, the second's in tau - 2; the
    // first lane of a warp each fetches one row parity of one of them. Planes,
    // rows and slots outside the grid arrive as 0.
    const int job = tid >> 5, job_array = (FROM_ZERO ? 2 : 0) + (job >> 1), job_parity = job & 1;
    const bool fetcher_warp = job < kLoads, fetcher = fetcher_warp && lane == 0;
    auto fetch = [&](int k) {
        if (!fetcher) return;
        s_fetched[job] = k;
        const uint32_t bar = full + 8u * uint32_t(k & 1);
        const int lag = (job_array + 1) >> 1;  // 0, 1, 1, 2
        const int ring = job_array == 0 ? kXB + (k & 3) : (job_array == 1 ? kXA + (k & 1) : (job_array == 2 ? kBA : kBB) + (k & 3));
        tc::mbar_expect_tx(bar, uint32_t(a.rows) * kRow * 4);
        load_rows(smem + 4u * uint32_t(ring * kPlane + job_parity * kBlock + kPad), job_array < 2 ? &xmap : &bmap, x0, job_parity,
                  (y0 - kHalo) / 2, tau0 + k - lag, (job_array == 0 || job_array == 3) ? cB : cA, bar);
    };
    if (steps > 0) fetch(0);
    // registers, newest plane first (A: first colour, B: second): B0 B1 B2 the
    // iterate in planes tau .. tau - 2, B3 B4 after half sweep 2 in tau - 3,
    // tau - 4; A1 the iterate in tau - 1, A2 A3 after half sweep 1 in tau - 2,
    // tau - 3, A4 A5 after half sweep 3 in tau - 4, tau - 5
    float A1[4] = {}, A2[4] = {}, A3[4] = {}, A4[4] = {}, A5[4] = {};
    float B0[4] = {}, B1[4] = {}, B2[4] = {}, B3[4] = {}, B4[4] = {};
    const bool y_wall = y == 0 || y == n - 1;
    float rmax = 0.f;
    double dzr = 0.0, dzq = 0.0;
    int limit = kWaitLimit;  // 0 once a wait has run out
    if (a.wait_probe > 0 && !tc::mbar_wait(probe, 0u, a.wait_probe)) limit = 0;
    const long out = long(z0) * plane_floats + long(y) * hw + slot0;
    float* outA = a.xout + (there ? out + long(cA) * n * plane_floats : 0);
    float* outB = a.xout + (there ? out + long(cB) * n * plane_floats : 0);

    int first_plane[4], count[4];  // planes that a half sweep updates, by the halo planes it takes in
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        first_plane[h] = max(0, z0 - h);
        count[h] = min(n, z1 + h) - first_plane[h];
    }
    // One half sweep of this thread's 4 slots in a plane, in two parts: what
    // comes from shared memory (c: the other colour of the plane) ...
    auto load = [&](auto parity, const float* rhs, const float* c, Near& m) {
        constexpr int s = decltype(parity)::value;
        m.edge = s ? c[mine + 4] : c[mine - 1];
        ld4(c + ym_at, m.ym);
        ld4(c + yp_at, m.yp);
        ld4(rhs + mine, m.b);
    };
    // ... and v = x + (b - off - diag x) w; o: the other colour in this row, zm,
    // zp: in the planes below and above. The neighbours are added up with their
    // own sign, which only flips that of the sum (a zero's sign does not reach
    // v), two slots to an addition.
    auto relax = [&](auto parity, auto last, int z, float (&x)[4], const Near& m, const float (&o)[4],
                     const float (&zm)[4], const float (&zp)[4]) {
        constexpr int s = decltype(parity)::value;
        constexpr bool LAST = decltype(last)::value;
        const bool z_wall = z == 0 || z == n - 1;
        const float wi = z_wall ? a.w[5] : a.w[6], wy = z_wall ? a.w[4] : a.w[5], wx = z_wall ? a.w[3] : a.w[4];
        const float di = z_wall ? -5.f : -6.f;
        const float d0 = y_wall ? di + 1.f : di, w0 = y_wall ? wy : wi;
        const bool x_wall = s ? right_wall : left_wall;
        const float d1 = x_wall ? d0 + 1.f : d0, w1 = x_wall ? (y_wall ? wx : wy) : w0;
        constexpr int kAtWall = s ? 3 : 0;
        const float e[5] = {s ? o[0] : m.edge, s ? o[1] : o[0], s ? o[2] : o[1], s ? o[3] : o[2], s ? m.edge : o[3]};
        float sum[4], t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[j] = e[j] + e[j + 1];
        add4(sum, m.ym);
        add4(sum, m.yp);
        add4(sum, zm);
        add4(sum, zp);
        add4(sum, m.b);
#pragma unroll
        for (int j = 0; j < 4; ++j) t[j] = (j == kAtWall ? d1 : d0) * x[j];
        add4(t, sum);
#pragma unroll
        for (int j = 0; j < 4; ++j) t[j] *= j == kAtWall ? w1 : w0;
        add4(x, t);
        if (RESID && LAST && own)
#pragma unroll
            for (int j = 0; j < 4; ++j) rmax = fmaxf(rmax, fabsf(sum[j] + (j == kAtWall ? d1 : d0) * x[j]));
    };
    auto dot = [&](const float (&z)[4], const float (&b)[4], int colour, int plane) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(a.q + out + (long(colour) * n + plane - z0) * plane_floats));
        const float qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            dzr = fma(double(z[j]), double(b[j]), dzr);  // the product is exact
            dzq = fma(double(z[j]), double(qv[j]), dzq);
        }
    };
    using No = std::false_type;
    using Yes = std::true_type;
    auto step = [&](auto parity, auto phase, int k) {
        using P = decltype(parity);
        constexpr int K = decltype(phase)::value;  // k & 3
        const int tau = tau0 + k;
        auto plane = [&](int ring) { return s_mem + ring * kPlane; };
        float* const pub = plane(kPub + (K & 1));           // published now: half sweep t at + 2 (t - 1) planes
        float* const before = plane(kPub + 1 - (K & 1));    // one step ago
        auto in = [&](int z, int reach) { return unsigned(z - first_plane[reach]) < unsigned(count[reach]); };
        // all warps have read what they need of the step before and published
        auto gate = [&]() {
            if (!tc::mbar_wait(go, uint32_t(K + 1) & 1u, limit)) limit = 0;
        };
        if (fetcher_warp) {
            gate();
            if (k + 1 < steps && limit != 0) fetch(k + 1);
        }
        if (!tc::mbar_wait(full + 8 * (K & 1), uint32_t(k >> 1) & 1u, limit)) limit = 0;
        if (!FROM_ZERO) {
            ld4(plane(kXB + K) + mine, B0);
            ld4(plane(kXA + (K & 1)) + mine, A1);
        }
        if (DOT && own) {  // the next step's values of q
            const long at = out + long(tau - 2 - z0) * plane_floats;
            if (in(tau - 2, 0)) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.q + at + long(cA) * n * plane_floats));
            if (in(tau - 3, 0)) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.q + at + (long(cB) * n - 1) * plane_floats));
        }
        // 1: first colour in plane tau - 1, between B planes tau - 2 and tau
        const bool live1 = there && sweeps > 0 && in(tau - 1, 3);
        if (live1) {
            Near m;
            load(P{}, plane(kBA + K), plane(kXB + ((K + 3) & 3)), m);
            relax(P{}, No{}, tau - 1, A1, m, B1, B2, B0);
        }
        if (!fetcher_warp) gate();
        if (there) {
            if (live1) st4(pub + mine, A1);
            // 2: second colour in plane tau - 2, between A planes tau - 3 and tau - 1
            if (sweeps > 0 && in(tau - 2, 2)) {
                Near m;
                load(P{}, plane(kBB + K), before, m);
                relax(P{}, No{}, tau - 2, B2, m, A2, A3, A1);
                st4(pub + 2 * kPlane + mine, B2);
            }
            // 3: first colour in plane tau - 3, between B planes tau - 4 and tau - 2
            if (sweeps > 1 && in(tau - 3, 1)) {
                Near m;
                load(P{}, plane(kBA + ((K + 2) & 3)), before + 2 * kPlane, m);
                relax(P{}, No{}, tau - 3, A3, m, B3, B4, B2);
                st4(pub + 4 * kPlane + mine, A3);
                if (DOT && own && in(tau - 3, 0)) dot(A3, m.b, cA, tau - 3);
            }
        }
        // 4: second colour in plane tau - 4, between A planes tau - 5 and tau - 3
        Near m;
        load(P{}, plane(kBB + ((K + 2) & 3)), before + 4 * kPlane, m);
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(go);
        if (there && in(tau - 4, 0)) {
            if (sweeps > 1) relax(P{}, Yes{}, tau - 4, B4, m, A4, A5, A3);
            if (own) {
                st4(outA, A4);
                st4(outB, B4);
                if (DOT) dot(B4, m.b, cB, tau - 4);
            }
            outA += plane_floats;
            outB += plane_floats;
        }
        // the next step's names
        copy4(A5, A4);
        copy4(A4, A3);
        copy4(A3, A2);
        copy4(A2, A1);
        copy4(B4, B3);
        copy4(B3, B2);
        copy4(B2, B1);
        copy4(B1, B0);
        if (FROM_ZERO) {
#pragma unroll
            for (int j = 0; j < 4; ++j) A1[j] = 0.f;
        }
    };
    // All half sweeps of step tau meet the same s = (y + tau - 1 + cA) & 1.
    auto march = [&](auto parity) {
        using P0 = decltype(parity);
        using P1 = std::integral_constant<int, 1 - P0::value>;
        for (int k = 0; k < steps; k += 4) {
            step(P0{}, std::integral_constant<int, 0>{}, k);
            if (k + 1 == steps) break;
            step(P1{}, std::integral_constant<int, 1>{}, k + 1);
            if (k + 2 == steps) break;
            step(P0{}, std::integral_constant<int, 2>{}, k + 2);
            if (k + 3 == steps) break;
            step(P1{}, std::integral_constant<int, 3>{}, k + 3);
        }
    };
    if ((odd + tau0 + 1 + cA) & 1) march(std::integral_constant<int, 1>{});
    else march(std::integral_constant<int, 0>{});
    if (limit == 0) {
        atomicOr(&a.ctrl->nonfinite, 8u);
        // Before the CTA's shared memory goes: the fetches of the last two steps
        // may still be on their way. A fetcher begins one only after it has seen
        // the barrier's one before it complete, so these are the phases to wait
        // for (in vain, for the time of the limit, when another fetcher gave up).
        if (fetcher && steps > 0)
            for (int f = s_fetched[job]; f >= max(0, s_fetched[job] - 1); --f)
                tc::mbar_wait(full + 8u * uint32_t(f & 1), uint32_t(f >> 1) & 1u, kDrainLimit);
    }
    __syncthreads();
    if (RESID) {
        const float br = block_max(rmax, s_max);
        if (tid == 0 && br > 0.f) atomicMax(&a.ctrl->res32_bits, __float_as_uint(br));
    }
    if (DOT) {
        const double zr = block_sum(dzr, s_sum);
        const double zq = block_sum(dzq, s_sum);
        if (tid == 0) {
            const int blk = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
            a.partials[2 * blk] = zr;
            a.partials[2 * blk + 1] = zq;
        }
    }
}

struct Plan {
    int xtiles = 0, ytiles = 0, zchunks = 0, ytile = 0, zchunk = 0;
    int ctas() const { return xtiles * ytiles * zchunks; }
};

// Row tiles and plane chunks: the least time in all, counting waves of one CTA
// per SM; a step costs a fixed part and one that follows its rows.
Plan search_plan(int n, int sms) {
    Plan best;
    double least = 0.0;
    const int xtiles = (n / 2 + 31) / 32;
    for (int ytile = 8; ytile <= 2 * kRows - 2 * kHalo; ytile += 2)
        for (int zchunk = 4; zchunk <= n; ++zchunk) {
            Plan p;
            p.xtiles = xtiles;
            p.ytile = ytile;
            p.zchunk = zchunk;
            p.ytiles = (n + ytile - 1) / ytile;
            p.zchunks = (n + zchunk - 1) / zchunk;
            const int waves = (p.ctas() + sms - 1) / sms;
            const double cost = double(waves) * (zchunk + 2 * kHalo + 2) * (0.3 + 0.7 * (ytile + 2 * kHalo) / (2 * kRows));
            if (best.xtiles == 0 || cost < least) {
                best = p;
                least = cost;
            }
        }
    return best;
}
Plan plan_for(int n) {
    static std::mutex mutex;
    static std::map<std::pair<int, int>, Plan> known;
    int device = 0, sms = 0;
    VB_CUDA(cudaGetDevice(&device));
    VB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    std::lock_guard<std::mutex> lock(mutex);
    const auto key = std::make_pair(n, sms);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    return known[key] = search_plan(n, sms);
}

// cuTensorMapEncodeTiled from the driver (no link-time dependency on libcuda).
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q);
        return (e == cudaSuccess && q == cudaDriverEntryPointSuccess)
                   ? reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f)
                   : nullptr;
    }();
    if (!fn) fail(VAPOR_RUNTIME_ERROR, "cuTensorMapEncodeTiled is not available from the CUDA driver");
    return fn;
}

// A red-black split field as (slot, row parity, row pair, plane, colour); the
// box: a tile's rows of one parity in one plane.
CUtensorMap field_map(const float* field, int n, int rows) {
    CUtensorMap map;
    const cuuint64_t hw = cuuint64_t(n) / 2, row = hw * 4;
    const cuuint64_t dims[5] = {hw, 2, cuuint64_t(n) / 2, cuuint64_t(n), 2};
    const cuuint64_t strides[4] = {row, 2 * row, row * cuuint64_t(n), row * cuuint64_t(n) * cuuint64_t(n)};
    const cuuint32_t box[5] = {cuuint32_t(kRow), 1, cuuint32_t(rows), 1, 1};
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    const CUresult r = tensor_map_encoder()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<float*>(field), dims,
                                            strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) fail(VAPOR_RUNTIME_ERROR, "cuTensorMapEncodeTiled failed for a pressure field");
    return map;
}

template <bool FROM_ZERO, bool RESID, bool DOT>
void launch(const Plan& p, const WaveArgs& a, const float* xin, const float* b, cudaStream_t s) {
    static OncePerDevice once;
    once([] {
        VB_CUDA(cudaFuncSetAttribute(k_sor_wave<FROM_ZERO, RESID, DOT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kSmem));
    });
    const CUtensorMap bmap = field_map(b, a.n, a.rows);
    const CUtensorMap xmap = FROM_ZERO ? bmap : field_map(xin, a.n, a.rows);
    count_launch();
    k_sor_wave<FROM_ZERO, RESID, DOT><<<dim3(p.xtiles, p.ytiles, p.zchunks), kThreads, kSmem, s>>>(xmap, bmap, a);
}

WaveArgs make_args(const ProjectionArgs& p, const Plan& plan, int first, float* xout, ProjControl* ctrl) {
    WaveArgs a{};
    a.n = p.g.n;
    a.hw = a.n / 2;
    a.rows = (plan.ytile + 2 * kHalo) / 2;
    a.ytile = plan.ytile;
    a.zchunk = plan.zchunk;
    a.first = first;
    for (int d = 0; d < 7; ++d) a.w[d] = p.omega / std::max(float(d), p.diagonal_floor);
    a.xout = xout;
    a.ctrl = ctrl;
    a.wait_probe = p.wait_probe;
    return a;
}

}  // namespace

// Whole 4-slot groups (n % 8 == 0, which also aligns the rows for TMA), 32-bit
// offsets; up to 128^3 the resident sweeps are faster.
bool sor_wave_applies(int n, bool masked) { return !masked && n % 8 == 0 && n > 128 && rb_count(n) < (size_t(1) << 31); }
// The preconditioner sweeps four times from zero and four times back; below 192^3
// its colour launches run from L2. A learned plume step, colour launches against
// passes: 17.0 / 17.2 ms at 160^3, 22.6 / 22.4 at 192^3, 31.7 / 30.2 at 224^3,
// 42.8 / 39.8 at 256^3.
bool smooth_wave_applies(int n, bool masked) { return n >= 192 && sor_wave_applies(n, masked); }

void launch_sor_wave(const ProjectionArgs& p, const float* xin, float* xout, const float* b, ProjControl* ctrl,
                     int sweep_index, bool measure, cudaStream_t s) {
    const Plan plan = plan_for(p.g.n);
    WaveArgs a = make_args(p, plan, 0, xout, ctrl);
    a.guarded = 1;
    a.sweep_index = sweep_index;
    if (measure) launch<false, true, false>(plan, a, xin, b, s);
    else launch<false, false, false>(plan, a, xin, b, s);
}

void launch_smooth_wave_from_zero(const ProjectionArgs& p, float* z, const float* r, ProjControl* ctrl, cudaStream_t s) {
    const Plan plan = plan_for(p.g.n);
    launch<true, false, false>(plan, make_args(p, plan, 0, z, ctrl), nullptr, r, s);
}

int launch_smooth_wave_back(const ProjectionArgs& p, const float* zin, float* zout, const float* r, const float* q,
                            double* partials, int partial_capacity, ProjControl* ctrl, cudaStream_t s) {
    const Plan plan = plan_for(p.g.n);
    WaveArgs a = make_args(p, plan, 1, zout, ctrl);
    if (!q || 2 * plan.ctas() > partial_capacity) {
        launch<false, false, false>(plan, a, zin, r, s);
        return 0;
    }
    a.q = q;
    a.partials = partials;
    launch<false, false, true>(plan, a, zin, r, s);
    return plan.ctas();
}

}  // namespace vb
