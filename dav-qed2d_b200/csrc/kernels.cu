// kernels.cu -- standalone (one tile per block) kernels of libqed2d and their
// launchers: the reference's device kernels (gamm5Dw, gamm5, tr_dQwdU,
// plaquette!, qtop!, krnl_force!, updt_fld!, unfold, plwv), the fused momentum
// kick, random fields, BLAS-1 and deterministic single-launch reductions.
#include <atomic>

#include "stencil.cuh"

namespace qed2d {

static std::atomic<int64_t> g_launches{0};
void count_launch(int n) { g_launches += n; }
int64_t launches() { return g_launches.load(); }

static inline unsigned tiles_grid(const Lat& g) { return (unsigned)num_tiles(g); }

// Tile kernels run on a 2D grid of tiles (x along i1, y along i2), so a thread
// finds its site without an index division; lattices taller than 65535 tiles
// fall back to a 1D grid.
static inline dim3 tiles_grid2(const Lat& g) {
    const unsigned nt1 = (unsigned)((g.L1 + TX - 1) / TX), nt2 = (unsigned)((g.L2 + TY - 1) / TY);
    return nt2 <= 65535 ? dim3(nt1, nt2) : dim3(tiles_grid(g));
}
__device__ __forceinline__ Site tile_site(const Lat& g) {
    return gridDim.y > 1 || g.L2 <= TY ? site_at(g, blockIdx.x, blockIdx.y, threadIdx.x)
                                       : site_of_tile(g, blockIdx.x, threadIdx.x);
}

// ---------------------------------------------------------------------------
// gamm5Dw (src/QED2dDirac.jl:2-33); optionally  so += addc * addv  with complex
// addc (the mu^2 si term of gamm5Dw_sqr_musq, :92, and the +-i mu terms of
// generate_pseudofermion!, src/QED2dRHMC.jl:308,317) and optionally so2 *= -1
// (Dw = g5 (g5 Dw), :157-169)
__global__ void __launch_bounds__(TILE) k_g5dw(double2* __restrict__ so, const double2* __restrict__ U,
                                               const double2* __restrict__ si, double m2, Lat g,
                                               const double2* __restrict__ addv, double2 addc, int g5_out) {
    const Site q = tile_site(g);
    if (!q.ok) return;
    Pair<double> o = g5dw_at<double>(SpDro{si, g.V}, LkD{U, g.V}, q, m2);
    if (addv) {
        o.a = o.a + cmul(addc, __ldg(addv + q.x));
        o.b = o.b + cmul(addc, __ldg(addv + q.x + g.V));
    }
    if (g5_out) o.b = -o.b;
    st_d(so, g.V, q.x, o);
}

// gamm5Dw on complex64 fields in the reference layout: the FP32 arithmetic of
// the mixed solver's inner iterations on complex64 spinors and links
__global__ void __launch_bounds__(TILE) k_g5dw_c64(float2* __restrict__ so, const float2* __restrict__ U,
                                                   const float2* __restrict__ si, float m2, Lat g) {
    const Site q = tile_site(g);
    if (!q.ok) return;
    const Pair<float> o = g5dw_at<float>(SpF2{si, g.V}, LkF2{U, g.V}, q, m2);
    so[q.x] = o.a;
    so[q.x + g.V] = o.b;
}

// gamm5 (src/QED2dDirac.jl:130-146)
__global__ void k_g5(double2* __restrict__ so, const double2* __restrict__ si, long long V) {
    const long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (x >= V) return;
    so[x] = si[x];
    so[x + V] = -si[x + V];
}

// tr_dQwdU (src/QED2dDirac.jl:172-199); frc = [accumulate ? frc : 0] + rho * force
__global__ void __launch_bounds__(TILE) k_force(double* __restrict__ frc, const double2* __restrict__ U,
                                                const double2* __restrict__ X, const double2* __restrict__ G,
                                                Lat g, double rho, int accumulate) {
    const Site q = tile_site(g);
    if (!q.ok) return;
    double f1, f2;
    fermion_force_at(U, X, G, g.V, q, f1, f2);
    if (accumulate) {
        frc[q.x] += rho * f1;
        frc[q.x + g.V] += rho * f2;
    } else {
        frc[q.x] = rho * f1;
        frc[q.x + g.V] = rho * f2;
    }
}

// The RHMC force of all poles of a flavour in two launches instead of two per
// pole (src/QED2dHMC.jl:528-545): k_g5dw_poles applies gamm5Dw to every pole's
// solution (blockIdx.z = pole), k_force_poles sums rho_i tr_dQwdU(X_i, g5Dw X_i)
// over the poles in pole order, each term as k_force computes it (the same bits
// as one k_force launch per pole).
struct Poles {
    const double2* X[QED2D_MAXPOLES];
    double2* G[QED2D_MAXPOLES];
    double rho[QED2D_MAXPOLES];
    int n;
};
__global__ void __launch_bounds__(TILE) k_g5dw_poles(const double2* __restrict__ U, const Poles P, double m2, Lat g) {
    const Site q = tile_site(g);
    if (!q.ok) return;
    const int i = blockIdx.z;
    st_d(P.G[i], g.V, q.x, g5dw_at<double>(SpDro{P.X[i], g.V}, LkD{U, g.V}, q, m2));
}
__global__ void __launch_bounds__(TILE) k_force_poles(double* __restrict__ frc, const double2* __restrict__ U,
                                                      const Poles P, Lat g, int accumulate) {
    const Site q = tile_site(g);
    if (!q.ok) return;
    double a1 = 0.0, a2 = 0.0;
    for (int i = 0; i < P.n; i++) {
        double f1, f2;
        fermion_force_at(U, P.X[i], P.G[i], g.V, q, f1, f2);
        if (i == 0 && !accumulate) {
            a1 = P.rho[0] * f1;
            a2 = P.rho[0] * f2;
        } else {
            if (i == 0) {
                a1 = frc[q.x];
                a2 = frc[q.x + g.V];
            }
            a1 += P.rho[i] * f1;
            a2 += P.rho[i] * f2;
        }
    }
    frc[q.x] = a1;
    frc[q.x + g.V] = a2;
}

// plaquette! (mode 0, Re P) and qtop! (mode 1, arg P) -- src/QED2dAction.jl:2-32
__global__ void __launch_bounds__(TILE) k_plaq_field(double* __restrict__ plx, const double2* __restrict__ U, Lat g,
                                                     int mode) {
    const Site q = tile_site(g);
    if (!q.ok) return;
    const double2 p = plaquette_of(__ldg(U + q.x), __ldg(U + g.V + q.xp1), __ldg(U + q.xp2), __ldg(U + g.V + q.x));
    plx[q.x] = mode == 0 ? p.x : atan2(p.y, p.x);
}

// krnl_force! -- src/QED2dAction.jl:34-53: every element of frc1 and frc2 written once
__global__ void __launch_bounds__(TILE) k_krnl_force(double* __restrict__ frc1, double* __restrict__ frc2,
                                                     const double2* __restrict__ U, Lat g, double beta) {
    const Site q = tile_site(g);
    if (!q.ok) return;
    const double2 p = plaquette_of(__ldg(U + q.x), __ldg(U + g.V + q.xp1), __ldg(U + q.xp2), __ldg(U + g.V + q.x));
    const double v = beta * p.y;
    frc1[q.x] = -v;
    frc1[q.x + g.V] = v;
    frc2[q.xp1 + g.V] = -v;
    frc2[q.xp2] = v;
}

// updt_fld! -- src/QED2dAction.jl:55-65; also refreshes the packed FP32 copy
__global__ void k_updt_fld(double2* __restrict__ U, const double* __restrict__ mom, double eps, long long V,
                           float4* __restrict__ U32) {
    const long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (x >= V) return;
    double s1, c1, s2, c2;
    sincos(eps * mom[x], &s1, &c1);
    sincos(eps * mom[x + V], &s2, &c2);
    const double2 u1 = cmul(make_double2(c1, s1), U[x]);
    const double2 u2 = cmul(make_double2(c2, s2), U[x + V]);
    U[x] = u1;
    U[x + V] = u2;
    if (U32) st_links32(U32, V, x, u1, u2);
}

__global__ void k_pack_links(float4* __restrict__ U32, const double2* __restrict__ U, long long V) {
    const long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (x >= V) return;
    const double2 u1 = U[x], u2 = U[x + V];
    st_links32(U32, V, x, u1, u2);
}

// krnl_unfold! / krnl_reflect! -- src/QED2dFields.jl:12-25,37-50
__global__ void k_unfold(double2* __restrict__ Uout, const double2* __restrict__ Uin, Lat g, int reflect) {
    const long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (x >= 2 * g.V) return;
    const int mu = x >= g.V;
    const long long s = x - mu * g.V;
    const int i2 = (int)(s / g.L1), i1 = (int)(s - (long long)i2 * g.L1);
    const long long L1n = 2LL * g.L1, Vout = 4 * g.V;
    const double2 u = Uin[x];
    const double2 uc = reflect ? conj(u) : u;
    double2* o = Uout + mu * Vout;
    o[i1 + L1n * i2] = u;
    o[i1 + g.L1 + L1n * i2] = uc;
    o[i1 + L1n * (i2 + g.L2)] = uc;
    o[i1 + g.L1 + L1n * (i2 + g.L2)] = u;
}

// plwv -- src/QED2dUtils.jl:2-11; pref = i sqrt(-sin^2 k1 - sin^2 k2) / (sin k1 + i sin k2)
__global__ void k_plwv(double2* __restrict__ so, Lat g, double k1, double k2, double2 pref) {
    const long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (x >= g.V) return;
    const int i2 = (int)(x / g.L1), i1 = (int)(x - (long long)i2 * g.L1);
    double s, c;
    sincos(k1 * i1 + k2 * i2, &s, &c);
    const double2 e = make_double2(c, s);
    so[x] = cmul(pref, e);
    so[x + g.V] = e;
}

// n N(0,1) numbers of (seed, stream, counter), times scale
__global__ void k_random_normal(double* __restrict__ out, long long n, uint64_t seed, uint32_t stream,
                                uint32_t counter, double scale) {
    const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (2 * j >= n) return;
    double z0, z1;
    normal_pair(seed, stream, counter, (uint64_t)j, z0, z1);
    out[2 * j] = scale * z0;
    if (2 * j + 1 < n) out[2 * j + 1] = scale * z1;
}

// mom += eps * (frc1 + frc2 [+ fermion force]) -- the kick of OMF4!/update_momenta!
// (src/QED2dHMC.jl:256,478,554) with krnl_force!'s two scattered buffers gathered
// per link, so no force arrays are stored.  The total gauge force on the links
// of site x is F1 = -v(x) + v(x - 2), F2 = v(x) - v(x - 1) with v = beta Im P
// (gauge_force_at).  Each thread computes the plaquette of its own site once
// into shared memory; the last warp also computes the row below the tile and
// the second-last warp's first TY lanes the column left of it (the tile's halo;
// two warps with two plaquettes each, the others one); every thread reads its
// neighbours' values from there: 4 link loads per site instead of 10, the same
// plaquette arithmetic, so the same bits.  FERM: add the fermion force of
// (X, G = g5Dw X); FRC: add frc.  The kicks without the fermion force fit in 40
// registers (6 blocks per SM on this streaming kernel), the fermion ones in 64.
template <bool FERM, bool FRC>
__global__ void __launch_bounds__(TILE, FERM ? 4 : 6) k_mom_kick(double* __restrict__ mom, const double2* __restrict__ U, Lat g,
                                                   double beta, double eps, const double2* __restrict__ X,
                                                   const double2* __restrict__ G, const double* __restrict__ frc) {
    __shared__ double sv[TY + 1][TX + 1];   // [1 + row][1 + column]; row 0 / column 0: the halo
    int t1, t2;
    if (gridDim.y > 1 || g.L2 <= TY) {
        t1 = blockIdx.x;
        t2 = blockIdx.y;
    } else {
        const int nt1 = (g.L1 + TX - 1) / TX;
        t2 = blockIdx.x / nt1;
        t1 = blockIdx.x - t2 * nt1;
    }
    const Site q = site_at(g, t1, t2, threadIdx.x);
    const int lx = threadIdx.x & (TX - 1), ly = threadIdx.x >> 5;
    const long long V = g.V;
    double mo1 = 0.0, mo2 = 0.0;
    if (q.ok) {
        mo1 = mom[q.x];   // issued with the link loads
        mo2 = mom[q.x + V];
        const double2 u1x = __ldg(U + q.x), u2x = __ldg(U + V + q.x);
        const double2 u2xp1 = __ldg(U + V + q.xp1), u1xp2 = __ldg(U + q.xp2);
        sv[ly + 1][lx + 1] = beta * plaquette_of(u1x, u2xp1, u1xp2, u2x).y;
    }
    if (ly == TY - 1) {   // v(y - 2) for y in the tile's first row: links of y - 2, y - 2 + 1 and y
        const Site y = site_at(g, t1, t2, lx);
        if (y.ok) {
            const long long xp1m2 = y.xm2 + (y.xp1 - y.x);
            sv[0][lx + 1] = beta * plaquette_of(__ldg(U + y.xm2), __ldg(U + V + xp1m2), __ldg(U + y.x),
                                                __ldg(U + V + y.xm2)).y;
        }
    } else if (ly == TY - 2 && lx < TY) {   // v(y - 1) for y in the tile's first column: links of y - 1, y, y - 1 + 2
        const Site y = site_at(g, t1, t2, TX * lx);
        if (y.ok) {
            const long long xm1p2 = y.xp2 + (y.xm1 - y.x);
            sv[lx + 1][0] = beta * plaquette_of(__ldg(U + y.xm1), __ldg(U + V + y.x), __ldg(U + xm1p2),
                                                __ldg(U + V + y.xm1)).y;
        }
    }
    __syncthreads();
    if (!q.ok) return;
    const double v = sv[ly + 1][lx + 1];
    double F1 = -v + sv[ly][lx + 1];
    double F2 = v - sv[ly + 1][lx];
    if constexpr (FERM) {
        double f1, f2;
        fermion_force_at(U, X, G, V, q, f1, f2);
        F1 = F1 + f1;
        F2 = F2 + f2;
    }
    if constexpr (FRC) {
        F1 = F1 + frc[q.x];
        F2 = F2 + frc[q.x + V];
    }
    mom[q.x] = mo1 + eps * F1;
    mom[q.x + V] = mo2 + eps * F2;
}

// updt_fld! followed by the pure-gauge kick, in one pass (OMF4! and leapfrog
// pure gauge alternate the two, src/QED2dHMC.jl:248-305): Uout = e^{i eu mom_in} Uin,
// mom_out = mom_in + ek F(Uout), each with the operations of updt_fld! and k_mom_kick.
// Reads Uin and mom_in, writes Uout and mom_out (distinct buffers: neighbours read the
// old momenta).  Lattices of whole tiles only.  Per site: links in 32 + out 32, momenta
// in 16 + out 16 (96 B) instead of 80 + 64 B for the two kernels.
//
// A tile is 32 x 8K sites, a thread a column of K: its links and momenta stay in registers
// from the update to the kick.  What the tile's plaquettes need beyond it (U1 of the rows
// above and below, U2 of the row below, U2 of the column to the right, both links of the
// column to the left) is updated again by the warps that `halo` names, a lane a link;
// neighbouring columns come by shuffle, neighbouring warps' rows through shared memory.
//
// Bound by memory: with 16 rows a tile (K = 2) 1/8 more links are updated than the lattice
// has.  With tiles of 8 rows staged in shared memory by a loop over their links (index
// divisions, wrapping and 64-bit addresses for each) it was bound by issue: 505 warp
// instructions for 32 sites, 86 of them FP64, at 68% of the issue slots and 48% of the
// DRAM rate.  Two OMF4 steps (10 passes and two kicks) on a B200: 768^2 185 -> 125 us, 1024^2
// 231 -> 200, 2048^2 1043 -> 731, 4096^2 3924 -> 2732 (18.3 GB at 6.7 TB/s); K = 1 at 4096^2
// 2948, K = 4 (spills, idle halo warps) 3195.  Passes alternate between upward and
// downward (`back`), so that the next one starts with what the last left in L2: 1024^2
// 211 -> 200, 2048^2 755 -> 731, 4096^2 2770 -> 2732.
template <int K>
__global__ void __launch_bounds__(TILE, K == 1 ? 6 : 4)
    k_updt_kick(double2* __restrict__ Uout, const double2* __restrict__ Uin, double* __restrict__ mom_out,
                const double* __restrict__ mom_in, Lat g, double beta, double eu, double ek, int back) {
    constexpr int W = TILE / 32, H = W * K;   // warps, rows of a tile
    __shared__ double2 s_low[W + 1][TX];      // U1 of every warp's lowest row, and of the row above the tile
    __shared__ double2 s_b2[TX + 1];          // U2 of the row below, columns 0..32
    __shared__ double2 s_r2[H], s_l1[H + 1], s_l2[H];   // U2 of column 32; U1, U2 of column -1
    __shared__ double s_top[W + 1][TX];       // v of the row below the tile and of every warp's highest row
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nt1 = g.L1 / TX;
    int t1 = blockIdx.x, t2 = blockIdx.y;
    if (gridDim.y == 1 && g.L2 > H) {   // more rows of tiles than a grid's second dimension holds
        t2 = t1 / nt1;
        t1 -= t2 * nt1;
    }
    if (back) t2 = g.L2 / H - 1 - t2;
    const int L1 = g.L1, V = L1 * g.L2;   // V <= 2^30 is checked at context creation: 2V - 1 fits
    const int x0 = t1 * TX, y0 = t2 * H;
    const int xl = x0 == 0 ? L1 - 1 : x0 - 1, xr = x0 + TX == L1 ? 0 : x0 + TX;
    const int yb = y0 == 0 ? g.L2 - 1 : y0 - 1, ya = y0 + H == g.L2 ? 0 : y0 + H;
    auto updated = [&](double2 u, double m) {
        double s, c;
        sincos(eu * m, &s, &c);
        return cmul(make_double2(c, s), u);
    };
    // own links
    const int x = x0 + lane + L1 * (y0 + w * K);
    double2 u1[K], u2[K];
    double m1[K], m2[K];
#pragma unroll
    for (int j = 0; j < K; j++) {
        const int i = x + j * L1;
        u1[j] = Uin[i];
        u2[j] = Uin[i + V];
        m1[j] = mom_in[i];
        m2[j] = mom_in[i + V];
    }
    // halo: rows 0 U1 above, 1 U1 below, 2 U2 below; from 3 on the columns' links, a lane each
    int hx = -1;
    double2* to = nullptr;
    if (w < 3) {
        hx = x0 + lane + L1 * (w == 0 ? ya : yb) + (w == 2 ? V : 0);
        to = w == 0 ? &s_low[W][lane] : w == 2 ? &s_b2[lane] : nullptr;
    } else {
        const int i = threadIdx.x - 96;
        if (i < H) hx = xl + L1 * (y0 + i), to = s_l1 + i;
        else if (i < 2 * H) hx = xl + L1 * (y0 + i - H) + V, to = s_l2 + i - H;
        else if (i < 3 * H) hx = xr + L1 * (y0 + i - 2 * H) + V, to = s_r2 + i - 2 * H;
        else if (i == 3 * H) hx = xl + L1 * ya, to = s_l1 + H;
        else if (i == 3 * H + 1) hx = xr + L1 * yb + V, to = s_b2 + TX;
    }
    double2 hu = make_double2(0, 0);
    if (hx >= 0) {
        hu = updated(Uin[hx], mom_in[hx]);
        if (to) *to = hu;
    }
#pragma unroll
    for (int j = 0; j < K; j++) {
        const int i = x + j * L1;
        u1[j] = updated(u1[j], m1[j]);
        u2[j] = updated(u2[j], m2[j]);
        Uout[i] = u1[j];
        Uout[i + V] = u2[j];
    }
    s_low[w][lane] = u1[0];
    __syncthreads();
    // v(y) = beta Im P(y) from U1(y), U2(y + 1), U1(y + 2), U2(y)
    double v[K];
#pragma unroll
    for (int j = 0; j < K; j++) {
        double2 r = make_double2(__shfl_down_sync(0xffffffffu, u2[j].x, 1), __shfl_down_sync(0xffffffffu, u2[j].y, 1));
        if (lane == 31) r = s_r2[w * K + j];
        v[j] = beta * plaquette_of(u1[j], r, j + 1 < K ? u1[j + 1 < K ? j + 1 : j] : s_low[w + 1][lane], u2[j]).y;
    }
    s_top[w + 1][lane] = v[K - 1];
    if (w == 1) {   // the row below
        s_top[0][lane] = beta * plaquette_of(hu, s_b2[lane + 1], s_low[0][lane], s_b2[lane]).y;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < K; j++) {
        const int i = x + j * L1;
        double l = __shfl_up_sync(0xffffffffu, v[j], 1);
        if (lane == 0)
            l = beta * plaquette_of(s_l1[w * K + j], u2[j], s_l1[w * K + j + 1], s_l2[w * K + j]).y;
        mom_out[i] = m1[j] + ek * (-v[j] + (j > 0 ? v[j > 0 ? j - 1 : 0] : s_top[w][lane]));
        mom_out[i + V] = m2[j] + ek * (v[j] - l);
    }
}

// y = a x + b z (complex scalars; z may alias y)
__global__ void k_zaxpby(double2* y, double2 a, const double2* x, double2 b, const double2* z,
                         long long n) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double2 v = cmul(a, x[i]);
    if (z) v = v + cmul(b, z[i]);
    y[i] = v;
}

// ---------------------------------------------------------------------------
// single-launch deterministic reductions: per-block compensated sums to part[]
// (hi, lo pairs), the last block to finish merges part[] in a fixed order into
// ctl->scal[slot..] (hi + lo)
constexpr int RB = 256;

template <int NV>
__device__ __forceinline__ void finish_reduce(DSum (&v)[NV], double* part, DevCtl* ctl, int slot) {
    static_assert(2 * NV <= kMaxPartVals, "partials hold (hi, lo) pairs");
    __shared__ double smem[64 * NV];
    __shared__ bool last;
    block_dsum<NV>(v, smem);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            part[(size_t)(2 * k) * kMaxPartBlocks + blockIdx.x] = v[k].hi;
            part[(size_t)(2 * k + 1) * kMaxPartBlocks + blockIdx.x] = v[k].lo;
        }
        __threadfence();
        last = atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < 32) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            DSum s{0.0, 0.0};
            for (int i = threadIdx.x; i < (int)gridDim.x; i += 32)
                dsum_merge(s, DSum{__ldcg(part + (size_t)(2 * k) * kMaxPartBlocks + i),
                                   __ldcg(part + (size_t)(2 * k + 1) * kMaxPartBlocks + i)});
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const DSum t{__shfl_xor_sync(0xffffffffu, s.hi, o), __shfl_xor_sync(0xffffffffu, s.lo, o)};
                dsum_merge(s, t);
            }
            if (threadIdx.x == 0) ctl->scal[slot + k] = s.hi + s.lo;
        }
        if (threadIdx.x == 0) ctl->ticket = 0;
    }
}

// |x|^2 (kind 0) or <x, y> (kind 1), compensated
__global__ void __launch_bounds__(RB) k_reduce_vec(int kind, const double2* __restrict__ x,
                                                   const double2* __restrict__ y, long long n, double* part,
                                                   DevCtl* ctl, int slot) {
    DSum v[2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (long long i = blockIdx.x * (long long)RB + threadIdx.x; i < n; i += (long long)gridDim.x * RB) {
        const double2 a = x[i];
        if (kind == 0) {
            dsum_add(v[0], norm2(a));
        } else {
            const double2 d = cjmul(a, y[i]);
            dsum_add(v[0], d.x);
            dsum_add(v[1], d.y);
        }
    }
    finish_reduce<2>(v, part, ctl, slot);
}

// (sum Re P, sum arg P, sum mom^2), compensated -- Action/Plaquette/Qtop/Hamiltonian
// (src/QED2dHMC.jl:198-237)
__global__ void __launch_bounds__(RB) k_reduce_gauge(const double2* __restrict__ U, const double* __restrict__ mom,
                                                     Lat g, double* part, DevCtl* ctl, int slot) {
    DSum v[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    for (long long x = blockIdx.x * (long long)RB + threadIdx.x; x < g.V; x += (long long)gridDim.x * RB) {
        const int i2 = (int)(x / g.L1), i1 = (int)(x - (long long)i2 * g.L1);
        const long long xp1 = (i1 + 1 == g.L1) ? x - (g.L1 - 1) : x + 1;
        const long long xp2 = (i2 + 1 == g.L2) ? (long long)i1 : x + g.L1;
        const double2 p = plaquette_of(__ldg(U + x), __ldg(U + g.V + xp1), __ldg(U + xp2), __ldg(U + g.V + x));
        dsum_add(v[0], p.x);
        dsum_add(v[1], atan2(p.y, p.x));
        if (mom) dsum_add(v[2], mom[x] * mom[x] + mom[x + g.V] * mom[x + g.V]);
    }
    finish_reduce<3>(v, part, ctl, slot);
}

__global__ void k_copy_scalar(DevCtl* ctl, int dst, int src) { ctl->scal[dst] = ctl->scal[src]; }

// y = x / ctl->scal[slot] (the power method's normalisation, kept on the device)
__global__ void k_scale_inv(double2* y, const double2* x, long long n, const DevCtl* __restrict__ ctl, int slot) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double d = ctl->scal[slot];
    y[i] = make_double2(x[i].x / d, x[i].y / d);
}

// ---------------------------------------------------------------------------
// launchers
static int post_launch(const char* name) {
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_status(e, name);
    return QED2D_OK;
}

static unsigned blocks_for(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

static unsigned reduce_grid(long long n) {
    long long b = (n + RB - 1) / RB;
    if (b > 4 * 148) b = 4 * 148;
    if (b < 1) b = 1;
    return (unsigned)b;
}

int launch_g5dw_c64(Ctx& c, float2* so, const float2* U, const float2* si, double am0) {
    k_g5dw_c64<<<tiles_grid2(c.g), TILE, 0, c.stream>>>(so, U, si, (float)(2.0 + am0), c.g);
    return post_launch("k_g5dw_c64");
}

int launch_g5dw(Ctx& c, double2* so, const double2* U, const double2* si, double am0, const double2* addv,
                double2 addc, bool g5_out) {
    k_g5dw<<<tiles_grid2(c.g), TILE, 0, c.stream>>>(so, U, si, 2.0 + am0, c.g, addv, addc, g5_out ? 1 : 0);
    return post_launch("k_g5dw");
}

int launch_g5(Ctx& c, double2* so, const double2* si) {
    k_g5<<<blocks_for(c.g.V, 256), 256, 0, c.stream>>>(so, si, c.g.V);
    return post_launch("k_g5");
}

int launch_tr_dqwdu(Ctx& c, double* frc, const double2* U, const double2* X, const double2* G) {
    k_force<<<tiles_grid2(c.g), TILE, 0, c.stream>>>(frc, U, X, G, c.g, 1.0, 0);
    return post_launch("k_force");
}

int launch_force_accum(Ctx& c, double* frc, const double2* U, const double2* X, const double2* G, double rho,
                       bool accumulate) {
    k_force<<<tiles_grid2(c.g), TILE, 0, c.stream>>>(frc, U, X, G, c.g, rho, accumulate ? 1 : 0);
    return post_launch("k_force");
}

int launch_force_poles(Ctx& c, double* frc, const double2* U, const double2* const* X, double2* const* G,
                       const double* rho, int n, double am0, bool accumulate) {
    if (n < 1 || n > QED2D_MAXPOLES) return QED2D_ERR_BAD_ARG;
    Poles P{};
    for (int i = 0; i < n; i++) {
        P.X[i] = X[i];
        P.G[i] = G[i];
        P.rho[i] = rho[i];
    }
    P.n = n;
    dim3 grid = tiles_grid2(c.g);
    grid.z = (unsigned)n;
    k_g5dw_poles<<<grid, TILE, 0, c.stream>>>(U, P, 2.0 + am0, c.g);
    QTRY(post_launch("k_g5dw_poles"));
    k_force_poles<<<tiles_grid2(c.g), TILE, 0, c.stream>>>(frc, U, P, c.g, accumulate ? 1 : 0);
    return post_launch("k_force_poles");
}

int launch_plaq_field(Ctx& c, double* plx, const double2* U, int mode) {
    k_plaq_field<<<tiles_grid2(c.g), TILE, 0, c.stream>>>(plx, U, c.g, mode);
    return post_launch("k_plaq_field");
}

int launch_krnl_force(Ctx& c, double* frc1, double* frc2, const double2* U) {
    k_krnl_force<<<tiles_grid2(c.g), TILE, 0, c.stream>>>(frc1, frc2, U, c.g, c.beta);
    return post_launch("k_krnl_force");
}

int launch_updt_fld(Ctx& c, double2* U, const double* mom, double eps, float4* U32) {
    k_updt_fld<<<blocks_for(c.g.V, 256), 256, 0, c.stream>>>(U, mom, eps, c.g.V, U32);
    return post_launch("k_updt_fld");
}

int launch_pack_links(Ctx& c, float4* U32, const double2* U) {
    k_pack_links<<<blocks_for(c.g.V, 256), 256, 0, c.stream>>>(U32, U, c.g.V);
    return post_launch("k_pack_links");
}

int launch_unfold(Ctx& c, double2* Uout, const double2* Uin, int reflect) {
    k_unfold<<<blocks_for(2 * c.g.V, 256), 256, 0, c.stream>>>(Uout, Uin, c.g, reflect);
    return post_launch("k_unfold");
}

int launch_plwv(Ctx& c, double2* so, double k1, double k2) {
    // pref = i * sqrt(complex(-s1^2 - s2^2)) / (s1 + i s2); sqrt of a non-positive
    // real is i*sqrt(|.|), so pref = -sqrt(s1^2 + s2^2) / (s1 + i s2)
    const double s1 = sin(k1), s2 = sin(k2);
    const double r = sqrt(s1 * s1 + s2 * s2);
    double2 pref;
    // -r / (s1 + i s2) by Smith's scaled division
    if (fabs(s1) >= fabs(s2)) {
        const double t = s2 / s1, den = s1 + s2 * t;
        pref = make_double2(-r / den, (r * t) / den);
    } else {
        const double t = s1 / s2, den = s2 + s1 * t;
        pref = make_double2((-r * t) / den, r / den);
    }
    k_plwv<<<blocks_for(c.g.V, 256), 256, 0, c.stream>>>(so, c.g, k1, k2, pref);
    return post_launch("k_plwv");
}

int launch_random_normal(Ctx& c, double* out, int64_t n, uint64_t seed, uint32_t stream, uint32_t counter,
                         double scale) {
    if (n <= 0) return QED2D_OK;
    k_random_normal<<<blocks_for((n + 1) / 2, 256), 256, 0, c.stream>>>(out, n, seed, stream, counter, scale);
    return post_launch("k_random_normal");
}

bool updt_kick_fits(const Ctx& c) { return c.g.L1 % TX == 0 && c.g.L2 % TY == 0; }

int launch_updt_kick(Ctx& c, double2* Uout, const double2* Uin, double* mom_out, const double* mom_in, double eu,
                     double ek, bool back) {
    if (!updt_kick_fits(c)) return QED2D_ERR_UNSUPPORTED;
    const int K = c.g.L2 % (2 * TY) == 0 ? 2 : 1;
    const unsigned nt1 = c.g.L1 / TX, nt2 = c.g.L2 / (TY * K);
    const dim3 grid = nt2 <= 65535 ? dim3(nt1, nt2) : dim3(nt1 * nt2);
    if (K == 2) k_updt_kick<2><<<grid, TILE, 0, c.stream>>>(Uout, Uin, mom_out, mom_in, c.g, c.beta, eu, ek, back);
    else k_updt_kick<1><<<grid, TILE, 0, c.stream>>>(Uout, Uin, mom_out, mom_in, c.g, c.beta, eu, ek, back);
    return post_launch("k_updt_kick");
}

int launch_mom_kick(Ctx& c, double* mom, const double2* U, double eps, const double2* X, const double2* G,
                    const double* frc) {
    const dim3 grid = tiles_grid2(c.g);
    if (X && frc) k_mom_kick<true, true><<<grid, TILE, 0, c.stream>>>(mom, U, c.g, c.beta, eps, X, G, frc);
    else if (X) k_mom_kick<true, false><<<grid, TILE, 0, c.stream>>>(mom, U, c.g, c.beta, eps, X, G, frc);
    else if (frc) k_mom_kick<false, true><<<grid, TILE, 0, c.stream>>>(mom, U, c.g, c.beta, eps, X, G, frc);
    else k_mom_kick<false, false><<<grid, TILE, 0, c.stream>>>(mom, U, c.g, c.beta, eps, X, G, frc);
    return post_launch("k_mom_kick");
}

int launch_zaxpby(Ctx& c, double2* y, double2 a, const double2* x, double2 b, const double2* z, long long n) {
    k_zaxpby<<<blocks_for(n, 256), 256, 0, c.stream>>>(y, a, x, b, z, n);
    return post_launch("k_zaxpby");
}

int launch_copy(Ctx& c, void* dst, const void* src, size_t bytes) {
    if (dst == src || bytes == 0) return QED2D_OK;
    QCHECK(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, c.stream));
    return QED2D_OK;
}

int launch_zero(Ctx& c, void* dst, size_t bytes) {
    QCHECK(cudaMemsetAsync(dst, 0, bytes, c.stream));
    return QED2D_OK;
}

int launch_reduce_vec(Ctx& c, int kind, const double2* x, const double2* y, long long n, int slot) {
    k_reduce_vec<<<reduce_grid(n), RB, 0, c.stream>>>(kind, x, y, n, c.part, c.ctl, slot);
    return post_launch("k_reduce_vec");
}

int launch_reduce_gauge(Ctx& c, const double2* U, const double* mom, int slot) {
    k_reduce_gauge<<<reduce_grid(c.g.V), RB, 0, c.stream>>>(U, mom, c.g, c.part, c.ctl, slot);
    return post_launch("k_reduce_gauge");
}

int launch_scale_inv(Ctx& c, double2* y, const double2* x, long long n, int slot) {
    k_scale_inv<<<blocks_for(n, 256), 256, 0, c.stream>>>(y, x, n, c.ctl, slot);
    return post_launch("k_scale_inv");
}

int launch_copy_scalar(Ctx& c, int dst_slot, int src_slot) {
    k_copy_scalar<<<1, 1, 0, c.stream>>>(c.ctl, dst_slot, src_slot);
    return post_launch("k_copy_scalar");
}

}  // namespace qed2d
