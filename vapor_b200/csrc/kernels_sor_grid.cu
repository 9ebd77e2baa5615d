// Red-black SOR of medium grids (beyond one cluster, up to about 128^3) with the
// iterate resident on the chip: every SM holds a block of rows and a slab of
// planes in registers and shared memory for a whole stretch of sweeps, and only
// the blocks' surfaces travel. See kernels_sor_cluster.cu for the update and
// the numbered words; here the words go through global memory (L2), one
// exchange per half sweep with the up to four neighbours, and the residual
// maxima of the checks are exchanged the same way, so no grid barrier is
// needed. The launch is cooperative: its CTAs run at the same time.
//
// One launch per colour took 5.1 us a half sweep at 128^3 and 3.8 at 96^3 (in a
// recorded step), this 2.3 and 1.5: 0.5 of arithmetic at 128^3, the rest the
// exchange (a store to L2, a poll, two block barriers). A Reflection step to
// 1e-6 went from 24.5 to 12.2 ms at 128^3 and from 13.4 to 6.9 at 96^3. The
// split takes the least work per SM; for scenes that share the device
// (`compact`) the fewest SMs, because cooperative launches wait for theirs:
// eight scenes of 32^3 to 128^3 take 27.4 ms a step with the former and 22.9
// with the latter.
#include "sor_resident.cuh"

namespace vb {
namespace {

using namespace resident;

struct Plan {
    int yblocks = 0, zblocks = 0, pz = 0, threads = 0, smem = 0, row = 0, planes = 0, plane = 0, half = 0, region = 0;
    bool full = false;  // every thread owns pz planes
    int ctas() const { return yblocks * zblocks; }
    size_t bytes() const { return size_t(ctas()) * region + size_t(ctas()) * 32; }
};

int device_sms() {
    static std::mutex mutex;
    static std::map<int, int> known;
    int device = 0;
    VB_CUDA(cudaGetDevice(&device));
    std::lock_guard<std::mutex> lock(mutex);
    auto it = known.find(device);
    if (it != known.end()) return it->second;
    int sms = 0, cooperative = 0;
    VB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    VB_CUDA(cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device));
    return known[device] = cooperative ? sms : 0;
}

// The split with the least work per SM (planes per thread times threads, and a
// part of the halo it fetches), fewer planes per thread on ties: one CTA per
// SM, within its registers and shared memory. `compact`: with the fewest SMs
// instead, for scenes that share the device.
Plan search_plan(int n, int sms, bool compact) {
    Plan best;
    if (n < 16) return best;
    const int hwp = ((n + 1) / 2 + 3) / 4 * 4, G = hwp / 4, row = row_floats(hwp);
    double least = 0.0;
    for (int yblocks = 1; yblocks <= n / 4; ++yblocks)
        for (int zblocks = 2; zblocks <= n && yblocks * zblocks <= sms; ++zblocks)
            for (int pz : {1, 2, 3, 4}) {
                Plan p;
                p.yblocks = yblocks;
                p.zblocks = zblocks;
                p.pz = pz;
                const int rows = (n + yblocks - 1) / yblocks, slab = (n + zblocks - 1) / zblocks;
                const int blocks = (slab + pz - 1) / pz;
                p.half = ((rows + 1) / 2 * G + 31) / 32 * 32;
                p.threads = 2 * p.half * blocks;
                p.row = row;
                p.planes = slab + 2;
                p.plane = (rows + 2) * p.row;
                p.smem = 2 * p.planes * p.plane * 4 + kTable * 4 * p.threads;
                p.full = n % zblocks == 0 && slab % pz == 0;
                p.region = 8 * 2 * p.half * 16 + 8 * slab * G * 16;
                if (p.threads > max_threads(pz) || p.smem > kSmemLimit - 2048) continue;
                const int items = 4 * p.half + 2 * slab * G;
                if (items > kItems * p.threads) continue;
                const double work = double(pz) * p.threads * (p.full ? 1.0 : 1.2) + 0.25 * items +
                                    (compact ? 1e6 * p.ctas() : 0.0);
                if (best.pz == 0 || work < least) {
                    best = p;
                    least = work;
                }
            }
    return best;
}
// The search takes about a millisecond, so its results are kept: a few dozen
// bytes for each grid size that a program uses.
Plan plan_for(int n, bool compact) {
    static std::mutex mutex;
    static std::map<std::tuple<int, int, bool>, Plan> known;
    const std::tuple<int, int, bool> key(n, device_sms(), compact);
    std::lock_guard<std::mutex> lock(mutex);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    return known[key] = search_plan(n, std::get<1>(key), compact);
}

bool launch(Mode mode, Args& a, unsigned char* words, bool compact, bool query, cudaStream_t s) {
    const Plan p = plan_for(a.n, compact);
    a.row = p.row;
    a.planes = p.planes;
    a.half = p.half;
    a.yblocks = p.yblocks;
    a.zblocks = p.zblocks;
    a.region = p.region;
    a.plane = p.plane;
    a.colour_stride = p.planes * p.plane;
    a.half_bytes = 2 * p.half * 16;
    a.y_half = (p.planes - 2) * a.groups * 16;
    a.words = words;
    if (!query) VB_CUDA(cudaMemsetAsync(words, 0, p.bytes(), s));  // the numbers start anew
    // one weight and divisor when the floor is at or above the largest diagonal
    const bool uniform = a.relax[3] == a.relax[6] && (mode == kMixed || a.two_product);
    const bool plain = a.hw % 4 == 0 && a.n % 2 == 0;
    const int kind = mode == kMixed && a.diag ? kMasked : (uniform ? kUniform : kGeneral);
    const int guard = p.full && plain ? 0 : 2;
    const Shape shape{p.ctas(), p.threads, p.smem};
    switch (p.pz) {
        case 1: return launch_planes<1, true>(mode, kind, guard, shape, a, query, s);
        case 2: return launch_planes<2, true>(mode, kind, guard, shape, a, query, s);
        case 3: return launch_planes<3, true>(mode, kind, guard, shape, a, query, s);
        default: return launch_planes<4, true>(mode, kind, guard, shape, a, query, s);
    }
}

}  // namespace

size_t sor_grid_words(int n) {
    size_t bytes = 0;
    for (bool compact : {false, true}) {
        const Plan p = plan_for(n, compact);
        if (p.pz > 0) bytes = std::max(bytes, p.bytes());
    }
    return bytes;
}

bool sor_grid_runs(const ProjectionArgs& p, SweepMode mode, bool compact) {
    if (plan_for(p.g.n, compact).pz == 0) return false;
    Args a = make_args(p, nullptr, nullptr, nullptr);
    return launch(Mode(mode), a, nullptr, compact, true, nullptr);
}

void launch_sor_grid_fixed(const ProjectionArgs& p, float* x, const float* b, ProjControl* ctrl, unsigned char* words,
                           bool compact, cudaStream_t s) {
    Args a = make_args(p, x, b, ctrl);
    a.subtract_mean = 1;
    launch(kFixed, a, words, compact, false, s);
}

void launch_sor_grid_tolerance(const ProjectionArgs& p, float* x, const float* b, ProjControl* ctrl,
                               unsigned char* words, bool compact, cudaStream_t s) {
    Args a = make_args(p, x, b, ctrl);
    a.subtract_mean = 1;
    launch(kTolerance, a, words, compact, false, s);
}

void launch_sor_grid_mixed(const ProjectionArgs& p, float* e, const float* r32, ProjControl* ctrl,
                           unsigned char* words, bool compact, cudaStream_t s) {
    Args a = make_args(p, e, r32, ctrl);
    a.flag_nonfinite = a.hw % 4 != 0;  // as the separate residual pass of those sizes does
    launch(kMixed, a, words, compact, false, s);
}

}  // namespace vb
