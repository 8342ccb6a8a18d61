// resident_gauge.cu -- pure-gauge molecular dynamics with the links and momenta on
// chip for the whole integration (one launch).
//
// Tiles, faces and slots as in resident.cuh: a thread holds a column of K sites (links
// and momenta in registers), so a kick needs two exchanges with the neighbouring tiles
// and nothing else:
//   U2 of the first column goes left, U1 of the lowest row down: every site's plaquette;
//   v of the last column goes right, of the highest row up:       every site's force.
// Nothing is summed, so a tile waits for its four neighbours only.  A slot is reused
// two kicks later; its sender has by then the receiver's answer to it (the plaquettes
// travel against the links), so it has been read.
//
// What bounds it: the two exchanges of a kick (about 1000 cycles each through L2), and
// from about 256^2 on FP64 arithmetic, half of it the two sincos of a link update.
// OMF4 step (5 link updates, 6 kicks) on a B200 against one kernel per update and kick
// (launch and L2 round trips, 5.8 us a pass): 32^2 37.6 -> 7.5 us, 128^2 35.0 -> 10.8,
// 256^2 35.1 -> 15.2, 512^2 49.5 -> 25.3.
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
    double2* box = reinterpret_cast<double2*>(dyn);
    if (threadIdx.x == 0) {
        B.rep = P.rep;
        B.C.nb = P.nb;
        B.C.rank = blockIdx.x;
        B.C.nslots = P.nslots;
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
    unsigned seq = 0;
    bool ok = true;
    // waits for the slots of one exchange: the first K lanes a row of the column from
    // side sx (into this warp's inbox), every lane its row entry from side sy
    auto receive = [&](int sx, int sy, bool link, double2& row) {
        const u64 slots = B.C.slots + (u64)(seq & 1u) * P.nslots * 16;
        double2* mine = box + warp * BOX;
        const bool rx = on && W.warp[sx] < 0 && lane < h, ry = on && W.warp[sy] < 0;
        const u64 px = slots + W.from[sx] + E * lane, py = slots + W.from[sy] + E * lane;
        if (W.warp[sx] < 0 || W.warp[sy] < 0) {
            Patience pt;
            for (;;) {
                ulonglong2 x0, x1, y0, y1;
                bool ready = true;
                if (rx) {
                    x0 = ld_slot<CL>(px);
                    if (link) x1 = ld_slot<CL>(px + 16);
                }
                if (ry) {
                    y0 = ld_slot<CL>(py);
                    if (link) y1 = ld_slot<CL>(py + 16);
                }
                if (rx) ready = tagged(x0, seq) && (!link || tagged(x1, seq));
                if (ry) ready = ready && tagged(y0, seq) && (!link || tagged(y1, seq));
                if (__all_sync(0xffffffffu, ready)) {
                    if (rx) mine[(sx == 1 ? K : 0) + lane] = make_double2(slot_double(x0), link ? slot_double(x1) : 0.0);
                    if (ry) row = make_double2(slot_double(y0), link ? slot_double(y1) : 0.0);
                    break;
                }
                if (!pt.more(B.C.err)) {
                    ok = false;
                    break;
                }
            }
            __syncwarp();
        }
        if (on && W.warp[sy] >= 0) row = mine[2 * K + (sy == 3 ? 32 : 0) + lane];
    };
    // F of the present links; false when a wait gave up (in all threads of the block)
    auto force = [&]() -> bool {
        ++seq;
        const u64 slots = (CL ? 0 : B.C.slots) + (u64)(seq & 1u) * P.nslots * 16;   // W.to holds addresses in a cluster
        if (on) {
            if (W.warp[2] >= 0) box[W.warp[2] * BOX + 2 * K + 32 + lane] = u1[0];
            else send2<CL>(slots + W.to[2] + E * lane, u1[0], seq);
            if (el) {
#pragma unroll
                for (int j = 0; j < K; j++) {
                    if (W.warp[0] >= 0) box[W.warp[0] * BOX + K + j] = u2[j];
                    else send2<CL>(slots + W.to[0] + E * j, u2[j], seq);
                }
            }
        }
        if (__syncthreads_or(!ok)) return false;
        double2 up = make_double2(0, 0);
        receive(1, 3, true, up);
        double v[K];
        const double2* mine = box + warp * BOX;
#pragma unroll
        for (int j = 0; j < K; j++) {
            double2 r = make_double2(__shfl_sync(0xffffffffu, u2[j].x, srcR), __shfl_sync(0xffffffffu, u2[j].y, srcR));
            if (er && (j < K - 1 || full)) r = mine[K + j];
            double2 a = j + 1 < K ? u1[j + 1 < K ? j + 1 : j] : up;
            if (j == TOP && K > 1) a = make_double2(full ? a.x : up.x, full ? a.y : up.y);
            v[j] = P.beta * plaquette_of(u1[j], r, a, u2[j]).y;
        }
        if (on) {
            const double top = full ? v[K - 1] : v[TOP];
            if (W.warp[3] >= 0) box[W.warp[3] * BOX + 2 * K + lane].x = top;
            else send1<CL>(slots + W.to[3] + E * lane, top, seq);
            if (er) {
#pragma unroll
                for (int j = 0; j < K; j++) {
                    if (W.warp[1] >= 0) box[W.warp[1] * BOX + j].x = v[j];
                    else send1<CL>(slots + W.to[1] + E * j, v[j], seq);
                }
            }
        }
        if (__syncthreads_or(!ok)) return false;
        double2 down = make_double2(0, 0);
        receive(0, 2, false, down);
#pragma unroll
        for (int j = 0; j < K; j++) {
            double l = __shfl_sync(0xffffffffu, v[j], srcL);
            if (el && (j < K - 1 || full)) l = mine[j].x;
            const double d = j > 0 ? v[j > 0 ? j - 1 : 0] : down.x;
            F1[j] = -v[j] + d;
            F2[j] = v[j] - l;
        }
        return true;
    };
    auto kick = [&](double e) {
#pragma unroll
        for (int j = 0; j < K; j++) {
            m1[j] = m1[j] + e * F1[j];
            m2[j] = m2[j] + e * F2[j];
        }
    };
    bool alive = force();
    if (alive) kick(P.first);
    for (int i = 0; i < P.ns && alive; i++) {
        for (int k = 0; k < P.m && alive; k++) {
            const double e = P.u[k];
#pragma unroll
            for (int j = 0; j < K; j++) {
                double s1, c1, s2, c2;
                sincos(e * m1[j], &s1, &c1);
                sincos(e * m2[j], &s2, &c2);
                u1[j] = cmul(make_double2(c1, s1), u1[j]);
                u2[j] = cmul(make_double2(c2, s2), u2[j]);
            }
            alive = force();
            if (alive) kick(i == P.ns - 1 && k == P.m - 1 ? P.last : P.c[k]);
        }
        if (P.each && i < P.ns - 1) kick(P.first);   // the next step's first kick: the same links
    }
#pragma unroll
    for (int j = 0; j < K; j++)
        if (v_ok && j < h) {
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
static int gauge_launch(const ResGaugeP& P, const ResPlan& p, cudaStream_t stream, bool query, int* clusters) {
    const void* kern = (const void*)k_res_gauge<K, CL>;
    const size_t sm = gauge_smem(p);
    QCHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    if (CL) QCHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.blocks());
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

static int gauge_dispatch(const ResGaugeP& P, const ResPlan& p, cudaStream_t s, bool query, int* n) {
    switch (p.K * 2 + p.cl) {
        case 2: return gauge_launch<1, false>(P, p, s, query, n);
        case 3: return gauge_launch<1, true>(P, p, s, query, n);
        case 4: return gauge_launch<2, false>(P, p, s, query, n);
        case 5: return gauge_launch<2, true>(P, p, s, query, n);
        case 8: return gauge_launch<4, false>(P, p, s, query, n);
        default: return gauge_launch<4, true>(P, p, s, query, n);
    }
}

// The split with the least modelled cycles per kick: FP64 arithmetic of the busiest
// SM (about 125 a row of 32 sites) and two exchanges.  K = 0: the fields do not fit.
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
                    p.cost = 125.0 * p.wx * p.wy * K + 500 + (bx * by == 1 ? 0 : p.cl ? 900 : 2000);
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

int res_gauge_md(Ctx& c, double* mom, double2* U, const ResMd& s) {
    const ResPlan& p = c.res_gauge;
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
    P.ctl = c.ctl;
    QCHECK(cudaMemsetAsync(&c.ctl->bar, 0, 2 * sizeof(unsigned long long) + sizeof(int), c.stream));
    if (!p.cl) {
        const size_t bytes = sizeof(ulonglong2) * 2 * P.nslots * (size_t)P.nb;
        P.slots = (ulonglong2*)c.buf("res_slots_gauge", bytes);
        if (!P.slots) return QED2D_ERR_NO_MEMORY;
        QCHECK(cudaMemsetAsync(P.slots, 0, bytes, c.stream));
    }
    return gauge_dispatch(P, p, c.stream, false, nullptr);
}

}  // namespace qed2d
