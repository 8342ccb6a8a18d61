// resident_f64.cu -- the on-chip CG in FP64 (resident.cuh): QED2D_PREC_F64, and the
// multishift solver on top of it.
#include "resident.cuh"

namespace qed2d {

int res_f64_clusters(const ResGeom& g) {
    return g.K == 1 ? res_clusters_k<double, 1>(g) : res_clusters_k<double, 2>(g);
}

int res_f64_launch(const ResP& P, const ResGeom& g, cudaStream_t stream) {
    switch (g.K * 2 + g.cl) {
        case 2: return res_launch_k<double, 1, false>(P, g, stream);
        case 3: return res_launch_k<double, 1, true>(P, g, stream);
        case 4: return res_launch_k<double, 2, false>(P, g, stream);
        default: return res_launch_k<double, 2, true>(P, g, stream);
    }
}

// ---------------------------------------------------------------------------
// Multishift CG (k_cg_multishift's recurrences): the base system runs as in the plain
// solve; the other shifts' x_i and p_i (64 bytes a site and shift) lie in shared memory,
// and the block's remaining warps update them,
//   x_i += a_i p_i,  p_i = z_i r + b_i p_i,
// one iteration behind the residual they read.  Nothing in the base system waits for
// them except at the next sum: they join that barrier, which keeps the two copies of r
// apart.  Shared memory holds about 3000 site-shifts a block, so a lattice is spread
// over at least that many blocks: 128^2 with 12 shifts over 128 of them.
template <int K>
struct ResMsSm {
    static size_t base(int nw) { return ResSm<double, K>::bytes(nw); }
    static size_t bytes(int nw, int n) {   // r twice, then x and p of n - 1 shifts
        return base(nw) + (size_t)nw * K * 32 * sizeof(double4x) * (2 + 2 * (n - 1));
    }
};

// The shift warps.  Items are (row of a worker warp, shift), a contiguous range per warp.
template <int K>
__device__ __forceinline__ void res_shifts(const ResP& P, const ResMs& M, ResBlock& B, const ResMsBlock& S,
                                           const double4x* rbuf, double4x* sx) {
    const int nw = M.nw, nwk = 32 * nw, ns = M.n - 1, lane = threadIdx.x & 31;
    const int sw = (int)(threadIdx.x >> 5) - 1 - nw, nsw = (int)(blockDim.x >> 5) - 1 - nw;
    const int items = nw * K * ns, i0 = sw * items / nsw, i1 = (sw + 1) * items / nsw;
    double4x* sp = sx + (size_t)ns * K * nwk;
    const double4x zero = mk4<double>(0, 0, 0, 0);
    auto shift_of = [&](int it) { return it % ns < M.base ? it % ns : it % ns + 1; };
    // a round: the base system's barrier, then how it ended and the shifts' scalars
    int round = 0;
    auto next_round = [&]() -> int {
        bar_sync_n(5, blockDim.x);
        bar_sync_n(4, blockDim.x - nwk);
        return *(const volatile int*)&S.flag[round++ & 1];
    };
    int flag = next_round();   // |b|^2; the worker warps' tiles are placed
    if (flag == RF_ABORT) return;
    const int L1 = B.rep.L1;
    const long long V = (long long)L1 * B.rep.L2;
    // this lane's site in row `row` (row j of worker warp row / K), -1: none
    auto site_of = [&](int row) -> long long {
        const int4 t = B.tile[row / K];
        const int j = row % K;
        return lane < t.z && j < t.w ? t.x + lane + (long long)L1 * (t.y + j) : -1;
    };
    for (int it = i0; it < i1; it++) {   // x_i = 0, p_i = b
        const int row = it / ns;
        const long long g = site_of(row);
        double4x b = zero;
        if (g >= 0) {
            const double2 a = __ldg(P.b + g), c = __ldg(P.b + V + g);
            b = mk4<double>(a.x, a.y, c.x, c.y);
        }
        sx[it * 32 + lane] = zero;
        sp[it * 32 + lane] = b;
    }
    for (int m = 0; flag == RF_GO; m++) {
        flag = next_round();   // |r|^2
        if (flag == RF_ABORT) return;
        if (m == 0) continue;   // before the first iteration
        int at = -1;
        double4x r = zero;
#pragma unroll 1
        for (int it = i0; it < i1; it++) {
            const int i = shift_of(it), row = it / ns, state = S.state[i];
            if (state == 0) continue;
            double4x p = sp[it * 32 + lane];
            sx[it * 32 + lane] = axpy4<double>(S.a[i], p, sx[it * 32 + lane]);
            if (state == 1) continue;
            if (row != at) {   // row j of worker warp w
                at = row;
                r = rbuf[((m & 1) * K + row % K) * nwk + 32 * (row / K) + lane];
            }
            const double z = S.z[i], b = S.b[i];
            p.x = z * r.x + b * p.x;
            p.y = z * r.y + b * p.y;
            p.z = z * r.z + b * p.z;
            p.w = z * r.w + b * p.w;
            sp[it * 32 + lane] = p;
        }
    }
    for (int it = i0; it < i1; it++) {
        const long long g = site_of(it / ns);
        const double4x v = sx[it * 32 + lane];
        if (g >= 0) st_d(M.x[shift_of(it)], V, g, Pair<double>{make_double2(v.x, v.y), make_double2(v.z, v.w)});
    }
}

template <int K>
__global__ void __launch_bounds__(32 * (kResWarps + 1), 1)
    k_res_ms(const __grid_constant__ ResP P, const __grid_constant__ ResMs M) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ ResBlock B;
    __shared__ ResMsBlock S;
    if (threadIdx.x == 0) {
        B.abort = 0;
        B.nwk = 32 * M.nw;
        B.C.nb = P.nb;
        B.C.rank = blockIdx.x;
        B.C.nslots = P.nslots;
        B.C.polls = P.polls;
        B.C.err = &P.ctl->err;
        B.C.slots = (u64)P.slots;
        B.C.psum = (u64)P.psum;
        B.C.acc = P.acc;
        B.rep = P.rep0;
    }
    __syncthreads();
    double4x* rbuf = reinterpret_cast<double4x*>(dyn + ResSm<double, K>::bytes(M.nw));
    double4x* sx = rbuf + 2 * K * 32 * M.nw;
    u64 base0 = 0, base1 = 0;
    if (threadIdx.x < 32) res_scalar<false, false, true>(P, B, 0, base0, base1, &M, &S);
    else if ((int)threadIdx.x < 32 * (M.nw + 1)) res_worker<double, K, false, true>(P, B, dyn, 0, rbuf);
    else res_shifts<K>(P, M, B, S, rbuf, sx);
    if (blockIdx.x == 0 && threadIdx.x == 0 && ld_volatile_int(&P.ctl->err) != 0)
        atomicCAS(&P.ctl->status, 0, QED2D_ERR_TIMEOUT);
}

static size_t res_ms_smem(const ResPlan& p, int n) {
    const int nw = p.wx * p.wy;
    return p.K == 1 ? ResMsSm<1>::bytes(nw, n) : ResMsSm<2>::bytes(nw, n);
}

constexpr size_t kMsStatic = (sizeof(ResBlock) + 15) / 16 * 16 + sizeof(ResMsBlock);   // static shared memory of k_res_ms

int res_ms_limit(int device, size_t* limit) {
    int optin = 0;
    QCHECK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    *limit = (size_t)optin - (kMsStatic + 15) / 16 * 16;
    return QED2D_OK;
}

bool res_ms_fits(const ResPlan& p, int n, size_t limit) {
    const int nw = p.wx * p.wy;
    return n > 1 && nw <= kResWarps - 2 && res_ms_smem(p, n) <= limit;
}

int res_ms_launch(const ResP& P0, const ResPlan& plan, const ResMs& m, cudaStream_t stream) {
    ResP P = P0;
    ResMs M = m;
    const int nw = plan.wx * plan.wy;
    M.nw = nw;
    const size_t sm = res_ms_smem(plan, M.n);
    const void* kern = plan.K == 1 ? (const void*)k_res_ms<1> : (const void*)k_res_ms<2>;
    QTRY(res_allow_smem(kern, kMsStatic));
    const int items = nw * plan.K * (M.n - 1), shift_warps = items < kResWarps - nw ? items : kResWarps - nw;
    void* args[] = {(void*)&P, (void*)&M};
    QCHECK(cudaLaunchCooperativeKernel(kern, dim3(P.nb), dim3(32 * (1 + nw + shift_warps)), args, sm, stream));
    count_launch();
    return QED2D_OK;
}

}  // namespace qed2d
