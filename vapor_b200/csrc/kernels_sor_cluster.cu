// Red-black SOR of small grids in one thread-block cluster.
//
// A sweep of a grid of up to 64^3 cells is shorter than the launch that starts
// it: with one launch per colour a half sweep took 2.7 us at 32^3 (4.1 without
// a graph) for 0.05 us of arithmetic. Here one launch runs every sweep up to
// the next decision of the solve: the whole fixed budget, the whole
// tolerance-driven solve with its FP64 residual checks, or the mixed solver's
// sweeps up to the next FP64 re-centring.
//
// The grid is cut into slabs of z-planes, one per CTA of the cluster. A thread
// owns 4 consecutive slots of one row in both colours for PZ planes and keeps
// their iterate and right-hand side in registers for the whole launch; the
// iterate is also published in shared memory for the neighbours in y and x and
// across threads in z. Between CTAs a boundary thread writes its updated slots
// straight to the one thread above or below that reads them: 8-byte words of a
// value and the half sweep's number in that CTA's shared memory, which the
// reader polls. So a half sweep costs one block barrier and one store to a
// neighbour SM, with no fence and no barrier over the cluster (st.async with
// complete_tx bytes, or stores with an arrival per warp on a remote mbarrier,
// took 0.4 us more a half sweep). Measured per half sweep of a fixed
// budget: 0.40 us at 16^3, 0.46 at 32^3 and 0.83 at 48^3, bound by that chain of
// shared-memory loads, seven dependent additions, barrier and neighbour store;
// 1.55 at 64^3 (mixed 1.51), bound by the issue slots of 16 SMs. Hence the shape of the update: what a slot's
// place selects is constant per warp (rows of one parity share a warp) or per
// launch (GUARD, KIND), and parameters are not indexed by the diagonal (an
// indexed parameter read replays per diagonal met in the warp).
//
// Every cell's update is the colour sweep's (k_sor_rbz): the same operations in
// the same order, missing neighbours read as zero, so iterates, residuals and
// iteration counts are the same bit for bit. The division by max(diagonal,
// floor) uses the two-product form of Brisebarre, Muller and Raina (2004,
// "Accelerating correctly rounded floating-point division when the divisor is
// known in advance") when the divisor is 3, 4, 5 or 6, for which it was checked
// against the division on every significand; below 2^-96, above 2^127 and for
// other divisors the division itself runs.
#include "sor_resident.cuh"

namespace vb {
namespace {

using namespace resident;

struct Plan {
    int ctas = 0, pz = 0, threads = 0, smem = 0, row = 0, planes = 0, half = 0;
    bool full = false;  // every thread owns pz planes
};

// Planes per thread as few as the threads allow, since they are updated one
// after the other (3 are never the fewest: 2 reach 48^3, from there 4 are
// needed); then CTAs that divide n, so that no thread owns fewer; then
// as many CTAs as the cluster allows.
Plan plan_for(int n) {
    Plan best;
    if (n < 2) return best;
    const int hwp = ((n + 1) / 2 + 3) / 4 * 4, G = hwp / 4, row = row_floats(hwp);
    for (int pz : {1, 2, 4})
        for (bool divides : {true, false})
            for (int ctas = std::min(n, kMaxCtas); ctas >= 2; --ctas) {
                const int slab = (n + ctas - 1) / ctas, blocks = (slab + pz - 1) / pz;
                const bool full = n % ctas == 0 && slab % pz == 0;
                if (full != divides) continue;
                Plan p;
                p.ctas = ctas;
                p.pz = pz;
                p.half = ((n + 1) / 2 * G + 31) / 32 * 32;
                p.threads = 2 * p.half * blocks;
                p.row = row;
                p.planes = slab + 2;
                p.smem = 2 * p.planes * (n + 2) * p.row * 4 + 8 * 2 * p.half * 16;
                p.full = full;
                if (p.threads <= max_threads(pz) && p.smem <= kSmemLimit - 2048) return p;
            }
    return best;
}

bool launch(Mode mode, Args& a, bool query, cudaStream_t s) {
    const Plan p = plan_for(a.n);
    a.row = p.row;
    a.planes = p.planes;
    a.half = p.half;
    a.plane = (a.n + 2) * p.row;
    a.colour_stride = p.planes * a.plane;
    a.half_bytes = 2 * p.half * 16;
    // one weight and divisor when the floor is at or above the largest diagonal
    const bool uniform = a.relax[3] == a.relax[6] && (mode == kMixed || a.two_product);
    const bool plain = a.hw % 4 == 0 && a.n % 2 == 0;
    const int kind = mode == kMixed && a.diag ? kMasked : (uniform ? kUniform : kGeneral);
    const int guard = !p.full ? 2 : (plain ? 0 : 1);
    const Shape shape{p.ctas, p.threads, p.smem};
    switch (p.pz) {
        case 1: return launch_planes<1, false>(mode, kind, guard, shape, a, query, s);
        case 2: return launch_planes<2, false>(mode, kind, guard, shape, a, query, s);
        default: return launch_planes<4, false>(mode, kind, guard, shape, a, query, s);
    }
}

}  // namespace

bool sor_cluster_applies(int n) { return plan_for(n).ctas > 0; }

bool sor_cluster_runs(const ProjectionArgs& p, SweepMode mode) {
    if (!sor_cluster_applies(p.g.n)) return false;
    Args a = make_args(p, nullptr, nullptr, nullptr);
    return launch(Mode(mode), a, true, nullptr);
}

void launch_sor_cluster_fixed(const ProjectionArgs& p, float* x, const float* b, ProjControl* ctrl, cudaStream_t s) {
    Args a = make_args(p, x, b, ctrl);
    a.subtract_mean = 1;
    launch(kFixed, a, false, s);
}

void launch_sor_cluster_tolerance(const ProjectionArgs& p, float* x, const float* b, ProjControl* ctrl,
                                  cudaStream_t s) {
    Args a = make_args(p, x, b, ctrl);
    a.subtract_mean = 1;
    launch(kTolerance, a, false, s);
}

void launch_sor_cluster_mixed(const ProjectionArgs& p, float* e, const float* r32, ProjControl* ctrl, cudaStream_t s) {
    Args a = make_args(p, e, r32, ctrl);
    a.flag_nonfinite = a.hw % 4 != 0;  // as the separate residual pass of those sizes does
    launch(kMixed, a, false, s);
}

}  // namespace vb
