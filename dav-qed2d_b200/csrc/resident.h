// resident.h -- host interface of the on-chip CG (resident.cu, resident_f64.cu).
#pragma once

#include <cuda_runtime.h>

#include <utility>
#include <vector>

#include "internal.h"

namespace qed2d {

// One system of a launch: lattice, place in the field arrays, mass, and how the
// lattice is split over the blocks of a team (see resident.cu).
struct ResRep {
    int L1, L2;
    long long off;      // first site of the lattice in the batch (0: single lattice)
    double m2;          // 2 + m0
    int ntx, nty;       // warp tiles along i1 (<= 32 sites wide) and i2 (<= K sites high)
    int bx, by;         // blocks of the team along i1 and i2
    int wx, wy;         // most warp tiles of a block along i1 and i2
    int id, pad;        // index of the system in the caller's order
};

// outcome of one system
struct ResOut {
    int it, conv, nupd, pad;
    double rr, bb;
};

// Shape of a launch: blocks of a team, worker warps of a block, halo slots of a block's buffer.
struct ResGeom {
    int K, cl, f64, nb, nw, nslots;
    int missing = 0;      // self-test: blocks left out of the launch,
    unsigned polls = 0;   // polls after which a wait gives up (0: the default)
};
ResGeom res_geom(const ResPlan& p);
// one that runs both (of the same K, cl and f64): teams and blocks of the larger, parts of
// which idle in the smaller's systems
inline ResGeom res_join(ResGeom a, const ResGeom& b) {
    a.nb = a.nb > b.nb ? a.nb : b.nb;
    a.nw = a.nw > b.nw ? a.nw : b.nw;
    a.nslots = a.nslots > b.nslots ? a.nslots : b.nslots;
    return a;
}

// K = 0 where the state does not fit on chip
ResPlan res_plan_single(int L1, int L2, int nb, bool f64);
ResPlan res_plan_pair(int L1, int L2, bool f64);   // a grid of two blocks
std::vector<ResPlan> res_plan_batch(const std::vector<std::pair<int, int>>& sizes, const std::vector<int>& n, int num_sms);
int res_clusters(const ResGeom& g);
ResRep res_rep(const ResPlan& p, int L1, int L2, long long off, double m2, int id);

struct ResArgs {
    const ResRep* reps = nullptr;   // device; null: rep0 alone
    ResRep rep0{};
    const double* m2 = nullptr;     // device, by system index: masses in the place of the ResReps'
    int nrep = 1;
    const double2* U = nullptr;
    const double2* b = nullptr;
    double2* x = nullptr;
    double2* t64 = nullptr;         // g5Dw x
    double2* r64 = nullptr;         // workspace
    double mu2 = 0.0, eps = 0.0;
    int maxiter = 0, guess = 0;
    int want_g5 = 0;                // FP64: t64 = g5Dw x is wanted (the mixed solver always leaves it)
    ResOut* out = nullptr;          // [nrep]
    void* slots = nullptr;          // res_slot_bytes(geom, nteams)
    DevCtl* ctl = nullptr;
    bool reset = true;              // clear the control block's error flag first
    int single = 0;                 // write the context's record of the solve
};
// the multishift solve: every shift's solution (the base system's is a.x)
struct ResShifts {
    int n, base;
    double d[QED2D_MAXPOLES];       // mu_i^2 - mu_base^2
    double2* x[QED2D_MAXPOLES];
};
int res_plan_ms(int L1, int L2, int nb, int n, int device, ResPlan* best);   // K = 0 where it does not fit
int res_launch_ms(const ResArgs& a, const ResPlan& plan, const ResShifts& s, cudaStream_t stream);
// Pure-gauge molecular dynamics on chip (resident_gauge.cu): kick first; ns times
// { m times: links by u[k], then kick c[k]; kick first again, if each and not the last
// step }, the very last kick `last`.
struct ResMd {
    double first, u[5], c[5], last;
    int m, ns, each;
};
bool res_gauge_fits(Ctx& c);
int res_gauge_md(Ctx& c, double* mom, double2* U, const ResMd& s, const ResPlan& p, int missing = 0, unsigned polls = 0);
size_t res_slot_bytes(const ResGeom& g, int nteams);
// one launch: nteams teams of geom.nb blocks solve the nrep systems
int res_launch(const ResArgs& a, const ResGeom& geom, int nteams, cudaStream_t stream);

}  // namespace qed2d
