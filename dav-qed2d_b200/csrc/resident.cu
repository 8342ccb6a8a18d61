// resident.cu -- the on-chip mixed CG (resident.cuh), and for both number types how a
// lattice is split over the blocks and the launch.
#include "resident.cuh"

#include <algorithm>

namespace qed2d {

// resident_f64.cu
int res_f64_clusters(const ResGeom& g);
int res_f64_launch(const ResP& P, const ResGeom& g, cudaStream_t stream);
int res_ms_limit(int device, size_t* limit);
bool res_ms_fits(const ResPlan& p, int n, size_t limit);
int res_ms_launch(const ResP& P, const ResPlan& plan, const ResMs& m, cudaStream_t stream);

static int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Modelled time of an iteration, us: waiting for exchanges, the depth of a thread's
// column, a scheduler's warps and the rows they walk (`share` blocks on an SM), the blocks
// whose sums arrive, and in a cluster columns of faces between blocks (bx > 1).  Fitted to
// cycles measured on a B200 at 1.92 GHz; within 8% of 60 splits of lattices from 16^2 to 512^2.
static double res_cost(int K, int warps, int bx, int by, bool cl, int share, bool f64) {
    const int wps = ceil_div(warps * share, 4), rows = wps * K, n = bx * by;
    if (f64) return ((n == 1 ? 3000 : cl ? 3390 : 5600) + 340 * K * K + 400 * rows) / 1920.0;
    if (cl || n == 1) return (3060 + (bx > 1 ? 40 : 20) * K * K + 100 * wps + 170 * rows + 14 * n) / 1920.0;
    return (5700 + 110 * rows + 3 * n) / 1920.0;
}

static std::vector<ResPlan> res_plans(int L1, int L2, int nb, int max_cluster, bool f64) {
    std::vector<ResPlan> best(nb + 1);
    for (ResPlan& p : best) p.K = 0;
    for (int K : {1, 2, 4}) {
        const int ntx = ceil_div(L1, 32), nty = ceil_div(L2, K);
        if (f64 && K > 2) continue;       // twice the registers a site
        if (L2 / nty < K - 1) continue;   // tiles have K or K - 1 rows
        for (int bx = 1; bx <= std::min(ntx, nb); bx++)
            for (int by = 1; by <= std::min(nty, nb / bx); by++) {
                const int wx = ceil_div(ntx, bx), wy = ceil_div(nty, by), n = bx * by;
                if (wx * wy > kResWarps) continue;
                const bool cl = n <= max_cluster;
                const double cost = res_cost(K, wx * wy, bx, by, cl, 1, f64);
                if (!best[n].K || cost < best[n].cost)
                    best[n] = ResPlan{K, cl ? 1 : 0, f64 ? 1 : 0, bx, by, wx, wy, ntx, nty, cost};
            }
    }
    std::vector<ResPlan> out;
    for (const ResPlan& p : best)
        if (p.K) out.push_back(p);
    return out;
}

ResRep res_rep(const ResPlan& p, int L1, int L2, long long off, double m2, int id) {
    return ResRep{L1, L2, off, m2, p.ntx, p.nty, p.bx, p.by, p.wx, p.wy, id, 0};
}

ResGeom res_geom(const ResPlan& p) {
    return ResGeom{p.K, p.cl, p.f64, p.blocks(), p.wx * p.wy, res_slots(p, p.f64 ? 2 : 1)};
}

// clusters of this shape that the device runs at a time
int res_clusters(const ResGeom& g) {
    if (g.f64) return res_f64_clusters(g);
    return g.K == 1 ? res_clusters_k<float, 1>(g) : g.K == 2 ? res_clusters_k<float, 2>(g) : res_clusters_k<float, 4>(g);
}

// A single lattice: the split with the least time.  Clusters of up to 16 blocks
// exchange over distributed shared memory, which takes a third of the time through
// L2, so a small lattice stays in one; beyond, the lattice spreads over as many SMs
// as there are.  Clusters of more than 8 blocks only where the device takes them.
ResPlan res_plan_single(int L1, int L2, int nb, bool f64) {
    for (int mc : {kResCluster, 8, 0}) {
        ResPlan best;
        best.K = 0;
        for (const ResPlan& p : res_plans(L1, L2, nb, mc, f64))
            if (!best.K || p.cost < best.cost) best = p;
        if (best.K == 0 || !best.cl || res_clusters(res_geom(best)) > 0) return best;
    }
    return ResPlan{};
}

ResPlan res_plan_pair(int L1, int L2, bool f64) {
    for (const ResPlan& p : res_plans(L1, L2, 2, 0, f64))
        if (p.blocks() == 2) return p;
    ResPlan none;
    none.K = 0;
    return none;
}

// A multishift solve with n shifts: the split with the least time, where the shifts'
// vectors fit and their updates hide behind the iteration or bound it.  Cycles an iteration
// measured on a B200 over 90 splits of lattices from 8^2 to 64^2, 2 to 12 shifts, and 128^2
// with 24: the base system as in res_cost, but 1400 more in a single block, whose sums no
// longer are cheap when the shift warps join them; shifts, K = 1: 3650 and 355 for each item
// (row and shift) of a shift warp, and no less than 106 for each of the block's (12^2 in one
// block, 3 shift warps: 4 shifts 7850, 6 shifts 10700; 128^2 over 128: 24 shifts 9800); K = 2:
// 1650 for each item of a warp (7 items: 11200 to 14500).  With 36 cycles an item and no
// penalty 16^2 with 4 shifts ran in one block in 5.8 us an iteration; spread over four
// 2.95, the grid kernel 5.0.
int res_plan_ms(int L1, int L2, int nb, int n, int device, ResPlan* best) {
    size_t limit = 0;
    QTRY(res_ms_limit(device, &limit));
    best->K = 0;
    for (int K : {1, 2}) {
        const int ntx = ceil_div(L1, 32), nty = ceil_div(L2, K);
        for (int bx = 1; bx <= std::min(ntx, nb); bx++)
            for (int by = 1; by <= std::min(nty, nb / bx); by++) {
                ResPlan p{K, 0, 1, bx, by, ceil_div(ntx, bx), ceil_div(nty, by), ntx, nty, 0.0};
                if (p.wx * p.wy > kResWarps || !res_ms_fits(p, n, limit)) continue;
                const int nw = p.wx * p.wy, items = nw * K * (n - 1), per = ceil_div(items, std::min(items, kResWarps - nw));
                const double shifts = K == 1 ? std::max(3650 + 355 * per, 106 * items) : 1650 * per;
                p.cost = std::max(res_cost(K, nw, bx, by, false, 1, true) + (bx * by == 1 ? 1400 : 0) / 1920.0, shifts / 1920);
                if (!best->K || p.cost < best->cost) *best = p;
            }
    }
    return QED2D_OK;
}

// Modelled time per iteration of n equal lattices under plan p: rounds of as many
// teams as run at a time.
static double res_time(const ResPlan& p, int n, int num_sms) {
    const int at = p.cl ? res_clusters(res_geom(p)) : num_sms / p.blocks();
    if (at < 1) return 1e30;
    const int m = std::min(n, at), share = ceil_div(m * p.blocks(), num_sms);
    return ceil_div(n, at) * res_cost(p.K, p.wx * p.wy, p.bx, p.by, p.cl, share, p.f64);
}

// A batch of lattices: sizes (L1, L2), counts n.  One size: the split with the least
// time for all of them.  Several: the one that occupies the least SM time per
// lattice, unless a single lattice then takes longer than the whole batch needs with
// every SM busy; such a size gets the least SM time among the splits that do not, or
// the fastest split.  Empty where a size does not fit.
std::vector<ResPlan> res_plan_batch(const std::vector<std::pair<int, int>>& sizes, const std::vector<int>& n, int num_sms) {
    std::vector<ResPlan> out;
    std::vector<std::vector<ResPlan>> cand;
    for (const auto& sz : sizes) {
        cand.push_back({});
        for (const ResPlan& p : res_plans(sz.first, sz.second, num_sms, kResCluster, false))
            if (!p.cl || res_clusters(res_geom(p)) > 0) cand.back().push_back(p);
        if (cand.back().empty()) return {};
    }
    if (sizes.size() == 1) {
        double tb = 1e30;
        out.resize(1);
        for (const ResPlan& p : cand[0]) {
            const double t = res_time(p, n[0], num_sms);
            if (t < tb) tb = t, out[0] = p;
        }
        return out;
    }
    double total = 0;
    for (size_t i = 0; i < sizes.size(); i++) {
        double sm = 1e30;
        for (const ResPlan& p : cand[i]) sm = std::min(sm, p.cost * p.blocks());
        total += n[i] * sm / num_sms;
    }
    for (size_t i = 0; i < sizes.size(); i++) {
        ResPlan best, fast;
        best.K = fast.K = 0;
        for (const ResPlan& p : cand[i]) {
            if (!fast.K || p.cost < fast.cost) fast = p;
            if (p.cost <= total && (!best.K || p.cost * p.blocks() < best.cost * best.blocks())) best = p;
        }
        out.push_back(best.K ? best : fast);
    }
    return out;
}

size_t res_slot_bytes(const ResGeom& g, int nteams) {
    if (g.cl) return 16;
    return sizeof(ulonglong2) * nteams * ((size_t)g.nb * (2 * g.nslots + 4) + kResAcc / 2) + 16;
}

// the kernel's parameters; clears the slots
static int res_fill(const ResArgs& a, const ResGeom& g, int nteams, cudaStream_t stream, ResP& P) {
    P.reps = a.reps;
    P.rep0 = a.rep0;
    P.nrep = a.nrep;
    P.nteams = nteams;
    P.nb = g.nb;
    P.U = a.U;
    P.b = a.b;
    P.x = a.x;
    P.t64 = a.t64;
    P.r64 = a.r64;
    P.mu2 = a.mu2;
    P.eps = a.eps;
    P.delta2 = kReliableDelta * kReliableDelta;
    P.maxiter = a.maxiter;
    P.guess = a.guess;
    P.want_g5 = a.want_g5;
    P.nslots = g.nslots;
    P.psum = (ulonglong2*)a.slots;
    P.slots = P.psum + (size_t)nteams * 4 * P.nb;
    P.acc = (u64*)(P.slots + (size_t)nteams * P.nb * 2 * P.nslots);
    P.queue = (int*)(P.acc + (size_t)nteams * kResAcc);
    P.m2 = a.m2;
    P.out = a.out;
    P.ctl = a.ctl;
    P.single = a.single;
    P.polls = g.polls ? g.polls : g.cl ? kWaitPolls<true> : kWaitPolls<false>;
    if (a.reset) QCHECK(cudaMemsetAsync(&a.ctl->bar, 0, 2 * sizeof(unsigned long long) + sizeof(int), stream));
    if (!g.cl) QCHECK(cudaMemsetAsync(a.slots, 0, res_slot_bytes(g, nteams), stream));
    return QED2D_OK;
}

int res_launch(const ResArgs& a, const ResGeom& g, int nteams, cudaStream_t stream) {
    ResP P{};
    QTRY(res_fill(a, g, nteams, stream, P));
    if (g.f64) return res_f64_launch(P, g, stream);
    switch (g.K * 2 + g.cl) {
        case 2: return res_launch_k<float, 1, false>(P, g, stream);
        case 3: return res_launch_k<float, 1, true>(P, g, stream);
        case 4: return res_launch_k<float, 2, false>(P, g, stream);
        case 5: return res_launch_k<float, 2, true>(P, g, stream);
        case 8: return res_launch_k<float, 4, false>(P, g, stream);
        default: return res_launch_k<float, 4, true>(P, g, stream);
    }
}

int res_launch_ms(const ResArgs& a, const ResPlan& plan, const ResShifts& s, cudaStream_t stream) {
    ResP P{};
    QTRY(res_fill(a, res_geom(plan), 1, stream, P));
    ResMs M{};
    M.n = s.n;
    M.base = s.base;
    for (int i = 0; i < s.n; i++) {
        M.d[i] = s.d[i];
        M.x[i] = s.x[i];
    }
    return res_ms_launch(P, plan, M, stream);
}

}  // namespace qed2d
