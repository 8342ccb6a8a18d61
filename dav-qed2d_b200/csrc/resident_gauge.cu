// resident_gauge.cu -- pure-gauge molecular dynamics with the links and momenta on
// chip for the whole integration (one launch).
//
// Tiles, faces and slots as in resident.cuh: a thread holds a column of K sites (links
// and momenta in registers).  A plaquette needs U1 of the row above the tile and U2 of the
// column to its right as well; these are carried along (their momenta get the force that
// their owners compute), so a kick needs one exchange with the neighbouring tiles: the
// plaquettes' v of the first and last column and of the lowest and highest row.  Nothing
// is summed, so a tile waits for its four neighbours only.  A slot is sent to again two
// kicks later; its sender has by then the receiver's v of the kick between, sent after the
// slot was read.
//
// What bounds it: the exchange of a kick (about 1000 cycles through L2) and the chain of a
// link update (sincos, plaquette); from about 400^2 on FP64 arithmetic, half of it the
// sincos of link updates.  OMF4 step (5 link updates, 6 kicks) on a B200 against one
// kernel per update and kick (launch and L2 round trips, 5.8 us a pass): 32^2 37.6 -> 6.6
// us, 128^2 35.0 -> 9.3, 256^2 35.1 -> 11.6, 512^2 49.5 -> 22.5.  With two exchanges a kick
// (the links to the right and above sent first, then v) 128^2 took 10.8, 256^2 15.2, 512^2 25.3.
#include <algorithm>

#include "resident.cuh"

namespace qed2d {

struct ResGaugeP {
    ResRep rep;
    int nb, nslots;
    double2* U;
    double* mom;
    double beta;
    // kick first; ns times { m times: links by u[k], kick c[k]; kick first again (every
    // step but the last, if each) }; the very last kick is `last`
    double first, u[5], c[5], last;
    int m, ns, each;
    ulonglong2* slots;
    unsigned polls;
    DevCtl* ctl;
};

// a plaquette's v takes one slot, a link two
template <bool CL>
__device__ __forceinline__ void send1(u64 p, double v, unsigned seq) {
    const u64 a = (u64)__double_as_longlong(v);
    st_slot<CL>(p, tag((unsigned)a, seq), tag((unsigned)(a >> 32), seq));
}

template <int K, bool CL>
__global__ void __launch_bounds__(32 * (kResWarps + 1), 1) k_res_gauge(const __grid_constant__ ResGaugeP P) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ ResBlock B;
    constexpr int BOX = 2 * K + 64, E = 32;   // bytes of a face entry
    constexpr int TOP = K > 1 ? K - 2 : 0;    // the highest row is K - 1 or this
    const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* const boxes = reinterpret_cast<double*>(dyn);   // two copies of the inboxes, in turn
    if (threadIdx.x == 0) {
        B.rep = P.rep;
        B.C.nb = P.nb;
        B.C.rank = blockIdx.x;
        B.C.nslots = P.nslots;
        B.C.polls = P.polls;
        B.C.err = &P.ctl->err;
        B.C.slots = CL ? smem_u32(dyn + (size_t)nw * BOX * sizeof(double2)) : (u64)P.slots;
    }
    if constexpr (CL) {
        ulonglong2* sl = reinterpret_cast<ulonglong2*>(dyn + (size_t)nw * BOX * sizeof(double2));
        for (int i = threadIdx.x; i < 2 * P.nslots; i += blockDim.x) sl[i] = make_ulonglong2(0, 0);
    }
    __syncthreads();
    if (lane == 0) res_place<double, K, CL>(B, warp);
    if constexpr (CL) cooperative_groups::this_cluster().sync();
    else __syncthreads();
    const int4 t4 = B.tile[warp];
    const WarpFace& W = B.face[warp];
    const int w = t4.z, h = t4.w, L1 = P.rep.L1;
    const bool on = h > 0, full = h == K, el = on && lane == 0, er = on && lane == w - 1;
    const int srcR = min(lane + 1, 31), srcL = max(lane - 1, 0);
    const long long V = (long long)L1 * P.rep.L2, g0 = t4.x + lane + (long long)L1 * t4.y;
    const bool v_ok = lane < w;
    double2 u1[K], u2[K];
    double m1[K], m2[K], F1[K], F2[K];
#pragma unroll
    for (int j = 0; j < K; j++) {
        u1[j] = u2[j] = make_double2(0, 0);
        m1[j] = m2[j] = F1[j] = F2[j] = 0.0;
        if (v_ok && j < h) {
            const long long g = g0 + (long long)j * L1;
            u1[j] = P.U[g];
            u2[j] = P.U[g + V];
            m1[j] = P.mom[g];
            m2[j] = P.mom[g + V];
        }
    }
    // the links beyond the tile that its plaquettes need, carried along with their momenta:
    // U1 of the row above (a lane a column) and U2 of the column to the right (lane j row j)
    double2 ua = make_double2(0, 0), ur = ua;
    double ma = 0.0, mr = 0.0, Fa = 0.0, Fr = 0.0;
    if (on && v_ok) {
        const long long g = t4.x + lane + (long long)L1 * (t4.y + h == P.rep.L2 ? 0 : t4.y + h);
        ua = P.U[g];
        ma = P.mom[g];
    }
    if (on && lane < h) {
        const long long g = V + (t4.x + w == L1 ? 0 : t4.x + w) + (long long)L1 * (t4.y + lane);
        ur = P.U[g];
        mr = P.mom[g];
    }
    unsigned seq = 0;
    bool ok = true;
    // F of the present links; false when a wait gave up (in all threads of the block)
    auto force = [&]() -> bool {
        double v[K];
#pragma unroll
        for (int j = 0; j < K; j++) {
            double2 r = make_double2(__shfl_sync(0xffffffffu, u2[j].x, srcR), __shfl_sync(0xffffffffu, u2[j].y, srcR));
            const double2 e = make_double2(__shfl_sync(0xffffffffu, ur.x, j), __shfl_sync(0xffffffffu, ur.y, j));
            if (er) r = e;
            double2 a = j + 1 < K ? u1[j + 1 < K ? j + 1 : j] : ua;
            if (j == TOP && K > 1) a = make_double2(full ? a.x : ua.x, full ? a.y : ua.y);
            v[j] = P.beta * plaquette_of(u1[j], r, a, u2[j]).y;
        }
        const double top = full ? v[K - 1] : v[TOP];
        ++seq;
        double* const box = boxes + (seq & 1u) * nw * BOX;
        double* const mine = box + warp * BOX;
        const u64 from = B.C.slots + (u64)(seq & 1u) * P.nslots * 16;
        const u64 to = CL ? (u64)(seq & 1u) * P.nslots * 16 : from;   // W.to holds addresses in a cluster
        if (on) {
            if (W.warp[2] >= 0) box[W.warp[2] * BOX + 2 * K + 32 + lane] = v[0];
            else send1<CL>(to + W.to[2] + E * lane, v[0], seq);
            if (W.warp[3] >= 0) box[W.warp[3] * BOX + 2 * K + lane] = top;
            else send1<CL>(to + W.to[3] + E * lane, top, seq);
            if (el) {
#pragma unroll
                for (int j = 0; j < K; j++) {
                    if (W.warp[0] >= 0) box[W.warp[0] * BOX + K + j] = v[j];
                    else send1<CL>(to + W.to[0] + E * j, v[j], seq);
                }
            }
            if (er) {
#pragma unroll
                for (int j = 0; j < K; j++) {
                    if (W.warp[1] >= 0) box[W.warp[1] * BOX + j] = v[j];
                    else send1<CL>(to + W.to[1] + E * j, v[j], seq);
                }
            }
        }
        if (__syncthreads_or(!ok)) return false;
        double down = 0.0, up = 0.0;
        if (on) {
            const int side = lane >= K ? 1 : 0;   // the first 2K lanes read a row each of the left and right columns
            const bool rx = lane < 2 * K && W.warp[side] < 0 && lane - side * K < h;
            const bool rd = W.warp[2] < 0, ru = W.warp[3] < 0;
            const u64 px = from + W.from[side] + E * (lane - side * K);
            ulonglong2 qx, qd, qu;
            Patience pt;
            for (;;) {
                if (rd) qd = ld_slot<CL>(from + W.from[2] + E * lane);
                if (ru) qu = ld_slot<CL>(from + W.from[3] + E * lane);
                if (rx) qx = ld_slot<CL>(px);
                const bool ready = (!rd || tagged(qd, seq)) && (!ru || tagged(qu, seq)) && (!rx || tagged(qx, seq));
                if (__all_sync(0xffffffffu, ready)) break;
                if (!pt.more(B.C)) {
                    ok = false;
                    break;
                }
            }
            if (rx) mine[lane] = slot_double(qx);
            __syncwarp();
            down = rd ? slot_double(qd) : mine[2 * K + lane];
            up = ru ? slot_double(qu) : mine[2 * K + 32 + lane];
        }
        double vr = 0.0;   // lane j: v of the tile's last column, row j
#pragma unroll
        for (int j = 0; j < K; j++) {
            double l = __shfl_sync(0xffffffffu, v[j], srcL);
            if (el && (j < K - 1 || full)) l = mine[j];
            F1[j] = -v[j] + (j > 0 ? v[j > 0 ? j - 1 : 0] : down);
            F2[j] = v[j] - l;
            const double e = __shfl_sync(0xffffffffu, v[j], max(w - 1, 0));
            if (lane == j) vr = e;
        }
        Fa = -up + top;
        if (on && lane < h) Fr = mine[K + lane] - vr;
        return true;
    };
    // explicit fma: the carried links' momenta get the bits that their owners' get (and the
    // compiler contracts the rest alike in every row: a test moves the field by some sites
    // and wants the same bits moved)
    auto kick = [&](double e) {
#pragma unroll
        for (int j = 0; j < K; j++) {
            m1[j] = fma(e, F1[j], m1[j]);
            m2[j] = fma(e, F2[j], m2[j]);
        }
        ma = fma(e, Fa, ma);
        mr = fma(e, Fr, mr);
    };
    auto move = [&](double2 u, double em) {
        double s, c;
        sincos(em, &s, &c);
        return cmul(make_double2(c, s), u);
    };
    bool alive = force();
    if (alive) kick(P.first);
    for (int i = 0; i < P.ns && alive; i++) {
        for (int k = 0; k < P.m && alive; k++) {
            const double e = P.u[k];
#pragma unroll
            for (int j = 0; j < K; j++) {
                u1[j] = move(u1[j], e * m1[j]);
                u2[j] = move(u2[j], e * m2[j]);
            }
            ua = move(ua, e * ma);
            ur = move(ur, e * mr);
            alive = force();
            if (alive) kick(i == P.ns - 1 && k == P.m - 1 ? P.last : P.c[k]);
        }
        if (P.each && i < P.ns - 1) kick(P.first);   // the next step's first kick: the same links
    }
    alive = !__syncthreads_or(!ok || !alive);   // a block that gave up leaves its fields as they were
#pragma unroll
    for (int j = 0; j < K; j++)
        if (alive && v_ok && j < h) {
            const long long g = g0 + (long long)j * L1;
            P.U[g] = u1[j];
            P.U[g + V] = u2[j];
            P.mom[g] = m1[j];
            P.mom[g + V] = m2[j];
        }
    if (!ok && lane == 0) atomicCAS(&P.ctl->status, 0, QED2D_ERR_TIMEOUT);
    if constexpr (CL) cooperative_groups::this_cluster().sync();   // others may still write here
}

// ---------------------------------------------------------------------------
// host side
static size_t gauge_smem(const ResPlan& p) {
    return (size_t)p.wx * p.wy * (2 * p.K + 64) * sizeof(double2) + (p.cl ? sizeof(ulonglong2) * 2 * res_slots(p, 2) : 0);
}

template <int K, bool CL>
static int gauge_launch(const ResGaugeP& P, const ResPlan& p, cudaStream_t stream, bool query, int* clusters, int missing) {
    const void* kern = (const void*)k_res_gauge<K, CL>;
    const size_t sm = gauge_smem(p);
    QTRY(res_allow_smem(kern));
    if (CL) QCHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.blocks() - missing);
    cfg.blockDim = dim3(32 * p.wx * p.wy);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    if (CL) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = p.blocks();
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (query) {
        if (!CL) *clusters = 1;
        else QCHECK(cudaOccupancyMaxActiveClusters(clusters, kern, &cfg));
        return QED2D_OK;
    }
    QCHECK(cudaLaunchKernelEx(&cfg, k_res_gauge<K, CL>, P));
    count_launch();
    return QED2D_OK;
}

static int gauge_dispatch(const ResGaugeP& P, const ResPlan& p, cudaStream_t s, bool query, int* n, int missing = 0) {
    switch (p.K * 2 + p.cl) {
        case 2: return gauge_launch<1, false>(P, p, s, query, n, missing);
        case 3: return gauge_launch<1, true>(P, p, s, query, n, missing);
        case 4: return gauge_launch<2, false>(P, p, s, query, n, missing);
        case 5: return gauge_launch<2, true>(P, p, s, query, n, missing);
        case 8: return gauge_launch<4, false>(P, p, s, query, n, missing);
        default: return gauge_launch<4, true>(P, p, s, query, n, missing);
    }
}

// The split with the least modelled cycles per link update and kick: the exchange, the
// chain of a thread's column, and what the block's warps issue.  Fitted to 16 splits of
// lattices from 64^2 to 256^2 (2945 to 6050 cycles, within 7%).  K = 0: the fields do not fit.
static int gauge_plan(int L1, int L2, int num_sms, ResPlan* best) {
    for (int mc : {kResCluster, 8, 0}) {
        best->K = 0;
        for (int K : {1, 2, 4}) {
            const int ntx = (L1 + 31) / 32, nty = (L2 + K - 1) / K;
            if (L2 / nty < K - 1) continue;
            for (int bx = 1; bx <= std::min(ntx, num_sms); bx++)
                for (int by = 1; by <= std::min(nty, num_sms / bx); by++) {
                    ResPlan p{K, bx * by <= mc ? 1 : 0, 1, bx, by, (ntx + bx - 1) / bx, (nty + by - 1) / by, ntx, nty, 0.0};
                    if (p.wx * p.wy > kResWarps) continue;
                    p.cost = 300.0 * K + 60 * K * K + 30 * p.wx * p.wy * (K + 1) + (bx * by == 1 ? 1700 : p.cl ? 2100 : 3160);
                    if (!best->K || p.cost < best->cost) *best = p;
                }
        }
        if (best->K == 0 || !best->cl) return QED2D_OK;
        int n = 0;
        if (gauge_dispatch(ResGaugeP{}, *best, nullptr, true, &n) == QED2D_OK && n > 0) return QED2D_OK;
        cudaGetLastError();
    }
    return QED2D_OK;
}

bool res_gauge_fits(Ctx& c) {
    if (c.res_gauge.K < 0 && gauge_plan(c.g.L1, c.g.L2, c.num_sms, &c.res_gauge) != QED2D_OK) c.res_gauge.K = 0;
    return c.res_gauge.K > 0;
}

int res_gauge_md(Ctx& c, double* mom, double2* U, const ResMd& s, const ResPlan& p, int missing, unsigned polls) {
    ResGaugeP P{};
    P.rep = res_rep(p, c.g.L1, c.g.L2, 0, 0.0, 0);
    P.nb = p.blocks();
    P.nslots = res_slots(p, 2);
    P.U = U;
    P.mom = mom;
    P.beta = c.beta;
    P.first = s.first;
    P.last = s.last;
    P.m = s.m;
    P.ns = s.ns;
    P.each = s.each;
    for (int k = 0; k < s.m; k++) {
        P.u[k] = s.u[k];
        P.c[k] = s.c[k];
    }
    P.polls = polls ? polls : p.cl ? kWaitPolls<true> : kWaitPolls<false>;
    P.ctl = c.ctl;
    QCHECK(cudaMemsetAsync(&c.ctl->bar, 0, 2 * sizeof(unsigned long long) + sizeof(int), c.stream));
    if (!p.cl) {
        const size_t bytes = sizeof(ulonglong2) * 2 * P.nslots * (size_t)P.nb;
        P.slots = (ulonglong2*)c.buf("res_slots_gauge", bytes);
        if (!P.slots) return QED2D_ERR_NO_MEMORY;
        QCHECK(cudaMemsetAsync(P.slots, 0, bytes, c.stream));
    }
    return gauge_dispatch(P, p, c.stream, false, nullptr, missing);
}

}  // namespace qed2d
