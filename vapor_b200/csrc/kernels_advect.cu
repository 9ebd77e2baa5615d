// Staggered-grid semi-Lagrangian and MacCormack advection
// (reference: src/solvers/mac3d/CpuAdvectionKernels.cpp:18-269, GLSL
// semi_lagrangian.comp:100-110 and maccormack.comp:151-204).
//
// A thread takes one point of the plane of sample points through up to 8
// planes. The forward pass writes fwd; the MacCormack pass re-traces forward
// through fwd, applies the 8-donor clamping limiter on the immutable source and
// falls back to fwd when either trace leaves [0, box] or |v| dt / h exceeds the
// CFL limit.
//
// Bound by instruction issue and the latency of the gathers (issue slots 60%
// busy, DRAM 16%). At a node the velocity's brackets depend on the node's index
// alone, so those along x and y serve all planes of a thread, those along z the
// whole block, and a plane's corner values serve the node below and above it;
// the MacCormack pass reads the traced velocities back; a division by a cell
// size that is no power of two takes four operations (div_h). At 160^3, h =
// 1/160, a face field: forward pass 83 -> 67 us (504 -> 335 instructions a
// point), MacCormack pass 110 -> 65 us (680 -> 335).
//
// A launch covers a set of fields: the smoke (cell centres) alone, or the
// three velocity components together (grid rows are the planes of u, then v,
// then w, in chunks), so a velocity advection is one forward launch and one MacCormack
// launch. When the cell size is a power of two the divisions by h run as
// multiplications by the exact 1/h (same bits, see div_h).
#include "kernels.hpp"

#include <algorithm>
#include <cmath>

namespace vb {
namespace {

constexpr int kThreads = 256;

constexpr int kMaxPlanes = 8;

// Traced velocity of every sample point, written by the forward pass and read
// back by the MacCormack pass instead of sampling the flow again (null: the
// MacCormack pass samples it itself). One array per component.
struct VelCache {
    float* p[3];
};

struct FieldSet {
    const float* src[3];
    float* fwd[3];
    float* out[3];
    VelCache vel[3];
};

// Sample point of location LOC: staggered axis at i*h, the others at (i+.5)h
// (`Vec3 face{ x * dx, (y + .5f) * dx, (z + .5f) * dx }`).
template <int LOC>
__device__ __forceinline__ void position(int x, int y, int z, float h, float& px, float& py, float& pz) {
    px = LOC == FACE_X ? float(x) * h : (float(x) + 0.5f) * h;
    py = LOC == FACE_Y ? float(y) * h : (float(y) + 0.5f) * h;
    pz = LOC == FACE_Z ? float(z) * h : (float(z) + 0.5f) * h;
}

// Base donor index of the limiter: int(pos/h) on the staggered axis, else
// int(pos/h - .5), clamped to the location's index range.
template <bool STAGGERED, bool POW2>
__device__ __forceinline__ int donor(float coord, const CellSize& c, int n) {
    return STAGGERED ? clampi_ref(int(div_h<POW2>(coord, c)), 0, n)
                     : clampi_ref(int(div_h<POW2>(coord, c) - 0.5f), 0, n - 1);
}

template <int LOC, bool POW2>
__device__ __forceinline__ float maccormack_point(const Grid& g, const CellSize& c, float dt, float cfl_limit, int x,
                                                  int y, int z, int i, const Vel& vel, const float* __restrict__ src,
                                                  const float* __restrict__ fwd) {
    const int n = g.n;
    const float h = g.h, box = g.box;
    float px, py, pz;
    position<LOC>(x, y, z, h, px, py, pz);
    const float fx = px - vel.x * dt, fy = py - vel.y * dt, fz = pz - vel.z * dt;
    const float bx = px + vel.x * dt, by = py + vel.y * dt, bz = pz + vel.z * dt;
    const float cfl = div_h<POW2>(sqrtf(vel.x * vel.x + vel.y * vel.y + vel.z * vel.z) * dt, c);
    const float f0 = fwd[i];
    const bool leaves = fx < 0.f || fx > box || fy < 0.f || fy > box || fz < 0.f || fz > box || bx < 0.f ||
                        bx > box || by < 0.f || by > box || bz < 0.f || bz > box;
    if (leaves || cfl > cfl_limit) return f0;
    const float back = sample<LOC, POW2>(fwd, n, c, bx, by, bz);
    const float corrected = f0 + 0.5f * (__ldg(src + i) - back);
    const int ex = n + (LOC == FACE_X), ey = n + (LOC == FACE_Y), ez = n + (LOC == FACE_Z);
    const int gx = donor<LOC == FACE_X, POW2>(fx, c, n);
    const int gy = donor<LOC == FACE_Y, POW2>(fy, c, n);
    const int gz = donor<LOC == FACE_Z, POW2>(fz, c, n);
    const int x1 = min(gx + 1, ex - 1), y1 = min(gy + 1, ey - 1), z1 = min(gz + 1, ez - 1);
    // row offsets of the donor cube (32-bit: fields hold < 2^31 values)
    const int r00 = ex * (gy + ey * gz), r10 = ex * (y1 + ey * gz);
    const int r01 = ex * (gy + ey * z1), r11 = ex * (y1 + ey * z1);
    const float s000 = __ldg(src + (r00 + gx));
    float lo = s000, hi = s000;
    const float s[7] = {__ldg(src + (r00 + x1)), __ldg(src + (r10 + gx)), __ldg(src + (r10 + x1)),
                        __ldg(src + (r01 + gx)), __ldg(src + (r01 + x1)), __ldg(src + (r11 + gx)),
                        __ldg(src + (r11 + x1))};
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        lo = minf_ref(lo, s[k]);
        hi = maxf_ref(hi, s[k]);
    }
    return clampf_ref(corrected, lo, hi);
}

// The block's share of one field: 256 points of the (x, y) plane in `planes`
// consecutive planes. A point's brackets along x and y serve all its planes;
// those along z, one pair per plane, are formed once per block.
enum Pass { kForward, kCorrect, kCorrectTraced };  // the last reads the forward pass's velocities
// Resident blocks of each pass. At 160^3: the traced correction 64.6 us with 6
// and 66.4 with 5, the forward pass 67.4 us with 4 and 70.8 with 5 (spills).
constexpr int kBlocks[3] = {4, 3, 6};
template <int LOC, Pass PASS, bool POW2>
__device__ __forceinline__ void advect_block(const Grid& g, float dt, float cfl_limit, int chunk, int planes,
                                             const float* __restrict__ src, const float* __restrict__ fwd,
                                             const float* __restrict__ u, const float* __restrict__ v,
                                             const float* __restrict__ w, float* __restrict__ out, float post_scale,
                                             const VelCache& cache, NodeAxis* s_z) {
    const int n = g.n;
    const CellSize c = cell_size<POW2>(g.h);
    const int ex = n + (LOC == FACE_X), ey = n + (LOC == FACE_Y), ez = n + (LOC == FACE_Z);
    const int z0 = chunk * planes, z1 = min(ez, z0 + planes);
    constexpr bool MC = PASS != kForward, traced = PASS == kCorrectTraced;
    if (!traced) {
        if (int(threadIdx.x) < z1 - z0) s_z[threadIdx.x] = node_axis<LOC == FACE_Z, POW2>(z0 + threadIdx.x, c, n);
        __syncthreads();
    }
    const int xy = int(blockIdx.x) * kThreads + threadIdx.x;
    if (xy >= ex * ey) return;
    const int y = xy / ex, x = xy - y * ex;
    ColumnSample<FACE_X> at_u;
    ColumnSample<FACE_Y> at_v;
    ColumnSample<FACE_Z> at_w;
    if constexpr (!traced) {
        const NodeAxis ax = node_axis<LOC == FACE_X, POW2>(x, c, n), ay = node_axis<LOC == FACE_Y, POW2>(y, c, n);
        at_u.start(n, ax.s, ay.c);
        at_v.start(n, ax.c, ay.s);
        at_w.start(n, ax.c, ay.c);
    }
    int i = xy + ex * ey * z0;
    for (int z = z0; z < z1; ++z, i += ex * ey) {
        Vel vel;
        if constexpr (traced) {
            vel.x = __ldg(cache.p[0] + i);
            vel.y = __ldg(cache.p[1] + i);
            vel.z = __ldg(cache.p[2] + i);
        } else {
            const NodeAxis& az = s_z[z - z0];
            vel.x = at_u.next(u, n, az.c);
            vel.y = at_v.next(v, n, az.c);
            vel.z = at_w.next(w, n, az.s);
        }
        if constexpr (MC) {
            out[i] = maccormack_point<LOC, POW2>(g, c, dt, cfl_limit, x, y, z, i, vel, src, fwd) * post_scale;
        } else {
            if (cache.p[0]) {
                cache.p[0][i] = vel.x;
                cache.p[1][i] = vel.y;
                cache.p[2][i] = vel.z;
            }
            float px, py, pz;
            position<LOC>(x, y, z, g.h, px, py, pz);
            const float qx = px - vel.x * dt, qy = py - vel.y * dt, qz = pz - vel.z * dt;
            out[i] = sample<LOC, POW2>(src, n, c, qx, qy, qz) * post_scale;
        }
    }
}

// blockIdx.y -> (field of the set, chunk of planes). FACES: the set is u, v, w
// (planes n, n and n + 1); otherwise the smoke (n planes).
template <bool FACES, Pass PASS, bool POW2>
__global__ void __launch_bounds__(kThreads, kBlocks[PASS]) k_advect_set(Grid g, float dt, float cfl_limit, FieldSet f, int planes,
                                                         const float* __restrict__ u, const float* __restrict__ v,
                                                         const float* __restrict__ w, float post_scale) {
    __shared__ NodeAxis s_z[kMaxPlanes];
    int field = 0, chunk = int(blockIdx.y);
    if (FACES) {
        const int chunks = (g.n + planes - 1) / planes;
        field = min(chunk / chunks, 2);
        chunk -= field * chunks;
    }
#define VB_FIELD(LOC, K, SCALE)                                                                               \
    advect_block<LOC, PASS, POW2>(g, dt, cfl_limit, chunk, planes, f.src[K], f.fwd[K], u, v, w,                 \
                                PASS != kForward ? f.out[K] : f.fwd[K], SCALE, f.vel[K], s_z)
    if (!FACES) VB_FIELD(CELL, 0, post_scale);
    else if (field == 0) VB_FIELD(FACE_X, 0, 1.f);
    else if (field == 1) VB_FIELD(FACE_Y, 1, 1.f);
    else VB_FIELD(FACE_Z, 2, 1.f);
#undef VB_FIELD
}

// One location at a time (staged calls): the same device code, one field.
template <int LOC, Pass PASS, bool POW2>
__global__ void __launch_bounds__(kThreads, kBlocks[PASS]) k_advect_one(Grid g, float dt, float cfl_limit, int planes,
                                                         const float* __restrict__ src,
                                                         const float* __restrict__ fwd,
                                                         const float* __restrict__ u, const float* __restrict__ v,
                                                         const float* __restrict__ w, float* __restrict__ out,
                                                         float post_scale, VelCache cache) {
    __shared__ NodeAxis s_z[kMaxPlanes];
    advect_block<LOC, PASS, POW2>(g, dt, cfl_limit, int(blockIdx.y), planes, src, fwd, u, v, w, out, post_scale, cache,
                                s_z);
}

// Planes per thread: as many as leave 8 blocks for each of 148 SMs. Four staged
// MacCormack fields at 160^3: 582 us with at most 8 planes, 590-635 with 4, 619-641
// with 16; with 4 blocks for each SM and 16 planes 632 (128^3: 308 against 347).
int planes_for(size_t blocks_per_plane, int planes) {
    return int(std::max<size_t>(1, std::min<size_t>(kMaxPlanes, blocks_per_plane * planes / (148 * 8))));
}

bool power_of_two(float h) {
    int e = 0;
    return std::isfinite(h) && h > 0.f && std::frexp(h, &e) == 0.5f;
}

template <bool FACES, bool POW2>
void advect_set(const Grid& g, float dt, float cfl_limit, bool maccormack, const FieldSet& f, const float* u,
                const float* v, const float* w, float post_scale, cudaStream_t s) {
    const int n = g.n;
    const int plane = FACES ? (n + 1) * n : n * n;
    const int blocks = (plane + kThreads - 1) / kThreads;
    const int planes = planes_for(blocks, FACES ? 3 * n + 1 : n);
    const int chunks = (n + planes - 1) / planes;
    const dim3 grid(blocks, FACES ? 2 * chunks + (n + planes) / planes : chunks);
    count_launch();
    k_advect_set<FACES, kForward, POW2><<<grid, kThreads, 0, s>>>(g, dt, cfl_limit, f, planes, u, v, w,
                                                               maccormack ? 1.f : post_scale);
    if (!maccormack) return;
    count_launch();
    if (f.vel[0].p[0]) k_advect_set<FACES, kCorrectTraced, POW2><<<grid, kThreads, 0, s>>>(g, dt, cfl_limit, f, planes, u, v, w, post_scale);
    else k_advect_set<FACES, kCorrect, POW2><<<grid, kThreads, 0, s>>>(g, dt, cfl_limit, f, planes, u, v, w, post_scale);
}

template <int LOC, bool POW2>
void advect_loc(const Grid& g, float dt, float cfl_limit, bool maccormack, const float* src, const float* u,
                const float* v, const float* w, float* fwd, float* out, float post_scale, float* const* vel_cache, cudaStream_t s) {
    const int ex = extent(g.n, LOC, 0), ey = extent(g.n, LOC, 1), ez = extent(g.n, LOC, 2);
    const int blocks = (ex * ey + kThreads - 1) / kThreads, planes = planes_for(blocks, ez);
    const dim3 grid(blocks, (ez + planes - 1) / planes);
    VelCache cache{};
    if (maccormack && vel_cache) cache = {{vel_cache[0], vel_cache[1], vel_cache[2]}};
    count_launch();
    k_advect_one<LOC, kForward, POW2><<<grid, kThreads, 0, s>>>(g, dt, cfl_limit, planes, src, nullptr, u, v, w,
                                                             maccormack ? fwd : out, maccormack ? 1.f : post_scale, cache);
    if (!maccormack) return;
    count_launch();
    if (cache.p[0])
        k_advect_one<LOC, kCorrectTraced, POW2><<<grid, kThreads, 0, s>>>(g, dt, cfl_limit, planes, src, fwd, u, v, w, out, post_scale, cache);
    else
        k_advect_one<LOC, kCorrect, POW2><<<grid, kThreads, 0, s>>>(g, dt, cfl_limit, planes, src, fwd, u, v, w, out, post_scale, cache);
}

template <bool POW2>
void advect_any(const Grid& g, int loc, float dt, float cfl_limit, bool maccormack, const float* src,
                const float* u, const float* v, const float* w, float* fwd, float* out, float post_scale,
                float* const* vel_cache, cudaStream_t s) {
    switch (loc) {
        case CELL: advect_loc<CELL, POW2>(g, dt, cfl_limit, maccormack, src, u, v, w, fwd, out, post_scale, vel_cache, s); break;
        case FACE_X: advect_loc<FACE_X, POW2>(g, dt, cfl_limit, maccormack, src, u, v, w, fwd, out, post_scale, vel_cache, s); break;
        case FACE_Y: advect_loc<FACE_Y, POW2>(g, dt, cfl_limit, maccormack, src, u, v, w, fwd, out, post_scale, vel_cache, s); break;
        default: advect_loc<FACE_Z, POW2>(g, dt, cfl_limit, maccormack, src, u, v, w, fwd, out, post_scale, vel_cache, s); break;
    }
}

}  // namespace

void launch_advect(const Grid& g, int loc, float dt, float cfl_limit, bool maccormack, const float* src,
                   const float* u, const float* v, const float* w, float* fwd, float* out, float post_scale,
                   float* const* vel_cache, cudaStream_t s) {
    if (power_of_two(g.h)) advect_any<true>(g, loc, dt, cfl_limit, maccormack, src, u, v, w, fwd, out, post_scale, vel_cache, s);
    else advect_any<false>(g, loc, dt, cfl_limit, maccormack, src, u, v, w, fwd, out, post_scale, vel_cache, s);
}

void launch_advect_velocity(const Grid& g, float dt, float cfl_limit, bool maccormack, const float* const src[3],
                            const float* u, const float* v, const float* w, float* const fwd[3],
                            float* const out[3], float* vel_cache, cudaStream_t s) {
    FieldSet f{};
    const size_t faces = size_t(g.n) * g.n * (g.n + 1);
    for (int c = 0; c < 3; ++c) {
        f.src[c] = src[c];
        // without MacCormack the forward pass is the result
        f.fwd[c] = maccormack ? fwd[c] : out[c];
        f.out[c] = out[c];
        if (maccormack && vel_cache)
            for (int k = 0; k < 3; ++k) f.vel[c].p[k] = vel_cache + (3 * c + k) * faces;
    }
    if (power_of_two(g.h)) advect_set<true, true>(g, dt, cfl_limit, maccormack, f, u, v, w, 1.f, s);
    else advect_set<true, false>(g, dt, cfl_limit, maccormack, f, u, v, w, 1.f, s);
}

void launch_advect_smoke(const Grid& g, float dt, float cfl_limit, bool maccormack, const float* src,
                         const float* u, const float* v, const float* w, float* fwd, float* out, float post_scale,
                         float* vel_cache, cudaStream_t s) {
    FieldSet f{};
    const size_t cells = size_t(g.n) * g.n * g.n;
    f.src[0] = src;
    f.fwd[0] = maccormack ? fwd : out;
    f.out[0] = out;
    if (maccormack && vel_cache)
        for (int k = 0; k < 3; ++k) f.vel[0].p[k] = vel_cache + k * cells;
    if (power_of_two(g.h)) advect_set<false, true>(g, dt, cfl_limit, maccormack, f, u, v, w, post_scale, s);
    else advect_set<false, false>(g, dt, cfl_limit, maccormack, f, u, v, w, post_scale, s);
}

}  // namespace vb
