// resident.cuh -- the on-chip CG: the whole state of a solve (links, r, p, q, x; in
// FP32 for the mixed solver, resident.cu, in FP64 for the other, resident_f64.cu) lives
// in registers and shared memory for the length of the solve, and only halos and
// partial sums leave an SM.
//
// A *team* of blocks solves one system.  The lattice is cut into warp tiles of at
// most 32 x K sites: lane = i1, a thread holds a column of K sites, so neighbours
// along i2 are in its own registers and neighbours along i1 one shuffle away.  A
// block holds wx x wy tiles; tile and block boundaries are a tensor-product grid
// (balanced splits, any lattice extents), so every face of a tile meets exactly
// one face of another.
//
// What crosses a face is the projected half spinor that the stencil needs there
// (8 bytes a site instead of 16, the backward ones already multiplied by the
// sender's link):
//   h1 = s1 - s2 (to the left),   h2 = conj(U1) (s1 + s2) (to the right),
//   h3 = s1 + i s2 (down),        h4 = conj(U2) (s1 - i s2) (up).
// Inside a block faces go through shared memory; between blocks through slots of
// 16 bytes, (value, sequence number) twice, each half a single 64-bit store: the
// receiver polls the slot itself, so there is no fence, no flag and no barrier on
// the way.  A team that is one thread-block cluster has its slots in the receivers'
// shared memory, a larger one in global memory.  There are two buffers of them, for
// the two stencils of an iteration.  The first's slots are sent to again after the sum
// that followed, to which a block adds when its warps have read them; the second's after
// the first exchange of the next iteration, whose face from the same neighbouring warp
// says that that warp has read them.
//
// Mixed: the iteration of the solver's other forms, with a sum behind each stencil,
//   w = g5Dw r          halo of r, |r|^2 summed meanwhile; x += alpha p while faces arrive
//   beta;  t = w + beta t (= g5Dw p)
//   w = g5Dw t          halo of t, <p, A p> = |t|^2 + mu^2 |p|^2 meanwhile; p = r + beta p
//   alpha; r -= alpha (w + mu^2 p)
// FP64: Chronopoulos and Gear's recurrences (J. Comput. Appl. Math. 25 (1989) 153),
// which need |r|^2 and <r, A r> = |g5Dw r|^2 + mu^2 |r|^2 only, so one sum:
//   t = g5Dw r          halo of r
//   w = g5Dw t + mu^2 r halo of t; the sum of both meanwhile, and p, x of the last iteration
//   beta = |r|^2 / |r_old|^2,  alpha = |r|^2 / (<r, A r> - beta |r|^2 / alpha_old)
//   q = w + beta q (= A p),  r -= alpha q;  later p = r_old + beta p, x += alpha p
// 128^2 takes 3.0 us an iteration instead of 4.4.  The difference in alpha's denominator
// (= <p, A p>) multiplies the relative error of the last one by
// beta alpha / alpha_old = (what is subtracted) / (what is left).  Where that exceeds one,
// errors would grow from iteration to iteration, and the iteration is made directly:
//   p = r + beta p,  t = g5Dw p,  sum <p, A p> = |t|^2 + mu^2 |p|^2,  q = g5Dw t + mu^2 p.
// Counts and residuals then are those of the two-sum form in ill-conditioned systems too
// (free links 64^2, m0 = 0.001: 267 iterations to 1e-12 and a true residual of 4e-11 in
// both, 355 and 6.5e-11 without; Gaussian links of width 0.45 on 40^2, m0 = -0.157: 800 in
// both, 1020 without), where a sixth to a third of the iterations are direct; at masses
// from -0.1 up on such links (128^2) none is.  The mixed solver does not use them, although 256^2 would take 2.9 us instead of
// 3.5: FP32 rounding and the jumps of r at reliable updates break the identity behind
// alpha near the critical mass, where solves that converge otherwise did not.  One extra
// warp per block does the block's sum, the team's sum and the scalar recurrences.
//
// What bounds it (B200): exchanges, until about 8 rows a scheduler's warps walk, then
// issue.  A sum over a grid takes 1.15 us from the last block's contribution until it is
// seen, plus 0.25 us of skew between the blocks, 0.2 us for the block's own sum and 0.25
// us for the recurrences, whatever the split; in a cluster about half of that, which the
// stencil's own chain (0.8 us) hides.  us an iteration, mixed: 64^2 1.95, 128^2 2.8, 256^2
// 3.5, 512^2 4.3; FP64: 64^2 2.2, 128^2 3.0, 256^2 4.0, 350x370 6.8.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "resident.h"
#include "stencil.cuh"

namespace qed2d {

constexpr int kResWarps = 15;      // most worker warps of a block (with the scalar warp: 128 registers a thread)
constexpr int kResCluster = 16;    // most blocks of a cluster
constexpr int kResAcc = 32;        // words of a team's fixed-point sums: two sets of four, 128 bytes apart

typedef unsigned long long u64;

// a spinor of the solver's number type, and how many slots of 16 bytes half of one takes
struct alignas(16) double4x { double x, y, z, w; };
template <class R> struct Num;
template <> struct Num<float> {
    using V4 = float4;
    static constexpr int SLOTS = 1;
};
template <> struct Num<double> {
    using V4 = double4x;
    static constexpr int SLOTS = 2;
};
template <class R> using V4 = typename Num<R>::V4;
template <class R> using V2 = typename cplx_of<R>::type;

struct ResP {
    const ResRep* reps;
    ResRep rep0;              // the system when there is only one
    const double* m2;         // 2 + m0 by system index (null: in the ResRep)
    int nrep, nteams, nb;     // systems, teams, blocks per team
    const double2* U;
    const double2* b;
    double2* x;
    double2* t64;             // g5Dw x of the solution (also the workspace of the updates)
    double2* r64;
    double mu2, eps, delta2;
    int maxiter, guess, want_g5;
    int* queue;               // next system (more systems than teams)
    ulonglong2* slots;        // halo slots: [team][block][2][slots]
    ulonglong2* psum;         // partial slots: [team][2][nb]
    u64* acc;                 // fixed-point sums: [team][kResAcc] words
    int nslots;               // slots of one buffer of a block
    ResOut* out;
    DevCtl* ctl;
    int single;               // write the context's solve record
    unsigned polls;           // after which a wait gives up
};

enum { RF_GO, RF_DIR, RF_UPD, RF_FIN, RF_STOP, RF_ZERO, RF_ABORT };   // the last three end the solve

// what the scalar warp hands to the workers after an exchange
struct ResSc {
    double alpha, beta;   // FP64 solver
    int flag;             // FP64 solver
    float2 cf;            // mixed solver: alpha or beta, and the flag's bits
    double s;             // scale of the FP32 vectors
};

// named barriers: 1 the workers' partials are in (scalar warp waits), 2 the faces
// inside the block are in (workers), 3 the exchange is over (all)
__device__ __forceinline__ void bar_sync_n(int id, int n) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive_n(int id, int n) {
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Slots: 16 bytes, two 64-bit words that carry a tag each.  Between blocks of a
// cluster (CL) they lie in the receiver's shared memory, else in global memory.
template <bool CL>
__device__ __forceinline__ void st_slot(u64 p, u64 a, u64 b) {
    if constexpr (CL)
        asm volatile("st.relaxed.cluster.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"((unsigned)p), "l"(a), "l"(b) : "memory");
    else
        asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
template <bool CL>
__device__ __forceinline__ ulonglong2 ld_slot(u64 p) {
    ulonglong2 v;
    if constexpr (CL)
        asm volatile("ld.relaxed.cluster.shared::cta.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"((unsigned)p) : "memory");
    else
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_rank(unsigned a, int rank) {   // address a of this block in block `rank` of the cluster
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ u64 tag(unsigned lo, unsigned seq) { return (u64)lo | ((u64)seq << 32); }
__device__ __forceinline__ double slot_double(const ulonglong2& q) {
    return __longlong_as_double((long long)((q.x & 0xffffffffull) | (q.y << 32)));
}
__device__ __forceinline__ bool tagged(const ulonglong2& v, unsigned seq) {
    return (unsigned)(v.x >> 32) == seq && (unsigned)(v.y >> 32) == seq;
}
template <bool CL>
__device__ __forceinline__ void send2(u64 p, float2 v, unsigned seq) {
    st_slot<CL>(p, tag(__float_as_uint(v.x), seq), tag(__float_as_uint(v.y), seq));
}
template <bool CL>
__device__ __forceinline__ void send2(u64 p, double2 v, unsigned seq) {
    const u64 a = (u64)__double_as_longlong(v.x), b = (u64)__double_as_longlong(v.y);
    st_slot<CL>(p, tag((unsigned)a, seq), tag((unsigned)(a >> 32), seq));
    st_slot<CL>(p + 16, tag((unsigned)b, seq), tag((unsigned)(b >> 32), seq));
}
// half a spinor on its way: its slots as last read
template <class R>
struct Arrival {
    ulonglong2 q[Num<R>::SLOTS];
    template <bool CL>
    __device__ __forceinline__ void ask(u64 p) {
#pragma unroll
        for (int i = 0; i < Num<R>::SLOTS; i++) q[i] = ld_slot<CL>(p + 16 * i);
    }
    __device__ __forceinline__ bool here(unsigned seq) const {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < Num<R>::SLOTS; i++) ok = ok && tagged(q[i], seq);
        return ok;
    }
    __device__ __forceinline__ V2<R> val() const {
        if constexpr (std::is_same<R, float>::value)
            return make_float2(__uint_as_float((unsigned)q[0].x), __uint_as_float((unsigned)q[0].y));
        else
            return make_double2(slot_double(q[0]), slot_double(q[1]));
    }
};
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// FP64 planes read at L2: other blocks wrote them in this launch
struct SpDcg {
    const double2* p;
    long long V;
    __device__ __forceinline__ Pair<double> ld(long long x) const { return {__ldcg(p + x), __ldcg(p + x + V)}; }
};

// dynamic shared memory of a block: per worker warp x, p and q of its sites and two
// inboxes (one per exchange of an iteration) of faces from other warps of the block
template <class R, int K>
struct ResSm {
    static constexpr int BOX = 2 * K + 64;   // left, right columns [K], lower, upper rows [32]
    static __host__ __device__ size_t bytes(int nw) {
        return (size_t)nw * (3 * K * 32 * sizeof(V4<R>) + 2 * BOX * sizeof(V2<R>));
    }
};

// a block's place in its team
struct TeamComm {
    u64 slots;           // global halo slots of the team, or this block's in shared memory (CL)
    u64 psum;            // the team's partials, [2][value][block], or this block's rows of them (CL)
    u64* acc;            // the team's fixed-point sums: two sets of words (not CL)
    int nb, rank, nslots;
    unsigned polls;      // after which a wait gives up
    int* err;
};

// Bounded wait of a warp: false when *err is set or the polls run out.  An exchange takes a
// few polls, another block's FP64 update some hundreds; a wait that lasts longer (another
// stream's work holds SMs that the rest of the grid needs, say) gives up after some 40 s,
// as the grid barriers do: 2^26 polls of L2 or 2^30 of shared memory.
template <bool CL> constexpr unsigned kWaitPolls = CL ? 1u << 30 : 1u << 26;
struct Patience {
    unsigned n = 0;
    __device__ __forceinline__ bool more(const TeamComm& C) {
        if ((++n & 255u) != 0) return true;
        const int e = ld_volatile_int(C.err);
        if (__any_sync(0xffffffffu, e != 0)) return false;
        if (n <= C.polls) return true;
        if ((threadIdx.x & 31) == 0) atomicExch(C.err, 2 /* QED2D_ERR_TIMEOUT */);
        return false;
    }
};

// The sums of an exchange: g, and in the FP64 solver (NV = 2) d.
struct Sums {
    double g, d;
};

// warp-wide: publishes this block's partials of sum `seq` in its slots of rows that
// the whole team polls, and returns the team's sums (same additions in the same order
// in every block).  For the few sums whose size is not known beforehand.
template <int NV>
__device__ __forceinline__ bool team_sum_slots(const TeamComm& C, unsigned seq, Sums v, Sums& tot) {
    const int nb = C.nb, lane = threadIdx.x & 31;
    bool ok = true;
    Patience pt;
    const u64 rows = C.psum + (u64)(seq & 1u) * 2 * nb * 16;
    if (lane < NV) {
        const u64 w = (u64)__double_as_longlong(lane ? v.d : v.g);
        st_slot<false>(rows + ((u64)lane * nb + C.rank) * 16, tag((unsigned)w, seq), tag((unsigned)(w >> 32), seq));
    }
    double s[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < NV; k++)
#pragma unroll 1
        for (int i = 0; i < nb && ok; i += 32) {
            ulonglong2 q;
            for (;;) {
                q = ld_slot<false>(rows + ((u64)k * nb + min(i + lane, nb - 1)) * 16);
                if (__all_sync(0xffffffffu, tagged(q, seq))) break;
                if (!(ok = pt.more(C))) break;
            }
            if (i + lane < nb) s[k] += slot_double(q);
        }
    tot.g = warp_sum(s[0]);
    if (NV > 1) tot.d = warp_sum(s[1]);
    return ok;
}

// The same in a cluster: every block's partials go to slots in every block's shared
// memory, lanes 0-15 for the first, 16-31 for the second.  (Every warp's partial to
// every block, without the block's own sum first, measured slower: 64^2 over 16 blocks
// 1970 cycles from partial to sum against 1400.)
template <int NV>
__device__ __forceinline__ bool cluster_sum_slots(const TeamComm& C, unsigned seq, Sums v, Sums& tot) {
    const int nb = C.nb, lane = threadIdx.x & 31;
    const int n2 = NV > 1 || nb > 8 ? kResCluster : nb > 4 ? 8 : nb > 2 ? 4 : 2;   // nb up to a power of two
    const int from = lane & (n2 - 1), k = NV > 1 ? lane / kResCluster : 0;
    const unsigned row = (unsigned)C.psum + 16 * ((seq & 1u) * 2 + k) * kResCluster;
    const u64 w = (u64)__double_as_longlong(k ? v.d : v.g);
    if ((NV > 1 ? from : lane) < nb)
        st_slot<true>(map_rank(row + 16 * C.rank, from), tag((unsigned)w, seq), tag((unsigned)(w >> 32), seq));
    ulonglong2 q;
    Patience pt;
    bool ok = true;
    for (;;) {
        q = ld_slot<true>(row + 16 * min(from, nb - 1));
        if (__all_sync(0xffffffffu, tagged(q, seq))) break;
        if (!(ok = pt.more(C))) break;
    }
    // every group of n2 lanes adds the same values in the same tree
    double s = from < nb ? slot_double(q) : 0.0;
#pragma unroll
    for (int o = kResCluster / 2; o > 0; o >>= 1)
        if (o < n2) s += __shfl_xor_sync(0xffffffffu, s, o);
    tot.g = NV > 1 ? __shfl_sync(0xffffffffu, s, 0) : s;
    if (NV > 1) tot.d = __shfl_sync(0xffffffffu, s, kResCluster);
    return ok;
}

// the exponent that scales this lane's words in team_sum_fixed, from an earlier sum
__device__ __forceinline__ int fixed_exponent(Sums est) {
    const double e = (threadIdx.x & 2) ? est.d : est.g;
    return min(max((int)((u64)__double_as_longlong(e) >> 52 & 0x7ff) - 1023, -900), 900);
}
// The same through atomic words (teams over global memory): a partial in 80-bit fixed
// point, 40 bits a word, scaled by a power of two (2^-ex) that every block derives from
// an earlier sum, with a count of the blocks in the top byte of each word.  Integer
// additions commute, so the sum does not depend on the order; each block's
// part is exact to 2^-76 of that earlier sum, the sum of 148 to 2^-68 (and repeated through
// the slots when it is below 2^-16 of the earlier one, which would leave less than 52 bits).
// The words only grow (modulo 2^64), two sets in turn, so nothing is cleared; `base` is the
// set's value before the exchange.  A partial out of range (or NaN) is counted in the next
// byte instead, and then every block falls back to team_sum_slots.  A lane per word, side by
// side, so that a block's atomics are one request and its poll another: with a line for each
// word 128^2 and 256^2 in FP64 took 2% more, with two polls in flight 13%.  Measured with 144
// blocks: 1610 cycles an exchange, against 2970 with a row of slots per block (whose
// polls grow with the square of the team), 4660 with one row, 2440 with an arrival
// counter and partials behind it, and 2740 through 7 clusters of 16 blocks (distributed
// shared memory, then L2 between the clusters' first blocks).
template <int NV>
__device__ __forceinline__ bool team_sum_fixed(const TeamComm& C, unsigned seq, Sums v, int ex, u64& base, Sums& tot,
                                               bool need_d, bool& exact) {
    const int lane = threadIdx.x & 31;
    u64* acc = C.acc + 16 * (seq & 1u) + (lane & 3);
    const double x = (lane & 2) ? v.d : v.g;
    if (lane < 2 * NV) {
        const double y = x * __longlong_as_double((long long)(1023 + 36 - ex) << 52);   // exact
        const bool fits = y < 1099511627776.0;   // 2^40; false for NaN
        const double hi = floor(y);
        const u64 part = fits ? (u64)((lane & 1) ? (y - hi) * 1099511627776.0 : hi) : (lane & 1) ? 0ull : 1ull << 48;
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(acc), "l"(part + (1ull << 56)) : "memory");
    }
    u64 d = 0;
    bool ok = true;
    Patience pt;
    for (;;) {
        u64 q = base;
        if (lane < 2 * NV) asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(q) : "l"(acc) : "memory");
        d = q - base;
        if (__all_sync(0xffffffffu, lane >= 2 * NV || (int)(d >> 56) == C.nb)) {
            base = q;
            break;
        }
        if (!(ok = pt.more(C))) break;
    }
    const double w = (double)(long long)(d & ((lane & 1) ? (1ull << 56) - 1 : (1ull << 48) - 1));
    const double s = (w + __shfl_xor_sync(0xffffffffu, w, 1) * 0x1p-40) * __longlong_as_double((long long)(1023 - 36 + ex) << 52);
    tot.g = __shfl_sync(0xffffffffu, s, 0);
    if (NV > 1) tot.d = __shfl_sync(0xffffffffu, s, 2);
    // no block out of range, and the sum of up to 255 blocks' truncated parts holds 52 bits
    const bool good = ((d >> 48) & 0xff) == 0 && s >= __longlong_as_double((long long)(1023 - 16 + ex) << 52);
    exact = __all_sync(0xffffffffu, good || !(lane == 0 || (NV > 1 && lane == 2 && need_d)));
    return ok;
}

// ---------------------------------------------------------------------------
// one warp tile
// Where a warp's faces go, kept in shared memory (left, right, down, up): the
// neighbouring warp of the block, or -1 and the slots in the team's array (of
// buffer 0) that its face is sent to and that the neighbour's face arrives in.
struct WarpFace {
    int warp[4];
    unsigned to[4], from[4];
};
struct Tile {
    int w, h;            // the warp's sites: w lanes, h rows (0: no tile)
    int srcL, srcR;      // lanes of the neighbours along i1
    bool el, er;         // this lane is the tile's first / last column
    // where this thread's faces go in the block's inboxes (column: el, er lanes; lower and
    // upper row), -1: to another block
    int xto, dto, uto;
    bool rx, rd, ru;     // this thread reads slots of a column, the lower, the upper row
    const WarpFace* W;
    unsigned sx, sd, su, fx, fd, fu;   // its slots to send to and to read
};
// The slots' addresses are worked out once where registers are left for them (512^2 mixed
// 4.35 -> 4.29 us an iteration, 128^2 in FP64 3.17 -> 2.98), not for FP64 columns of two
// sites, which spill (350x370 6.5 -> 8.4).
template <class R, int K, bool CL>
struct Slots {
    static constexpr bool REGS = K * sizeof(R) < 16 || std::is_same<R, float>::value;
    static constexpr bool PRE = REGS && !CL;   // read the block's own inbox before the slots have arrived (a cluster's do at once)
    static constexpr int E = 16 * Num<R>::SLOTS;   // bytes of a face entry
    static __device__ __forceinline__ int lane() { return threadIdx.x & 31; }
    static __device__ __forceinline__ int side() { return lane() >= K ? 1 : 0; }   // the first 2K lanes read a row each of the left and right columns
    static __device__ __forceinline__ void init(Tile& T) {
        if (!REGS) return;
        T.sx = T.W->to[T.el ? 0 : 1];
        T.sd = T.W->to[2] + E * lane();
        T.su = T.W->to[3] + E * lane();
        T.fx = T.W->from[side()] + E * (lane() - side() * K);
        T.fd = T.W->from[2] + E * lane();
        T.fu = T.W->from[3] + E * lane();
    }
    static __device__ __forceinline__ unsigned sx(const Tile& T) { return REGS ? T.sx : T.W->to[T.el ? 0 : 1]; }
    static __device__ __forceinline__ unsigned sd(const Tile& T) { return REGS ? T.sd : T.W->to[2] + E * lane(); }
    static __device__ __forceinline__ unsigned su(const Tile& T) { return REGS ? T.su : T.W->to[3] + E * lane(); }
    static __device__ __forceinline__ unsigned fx(const Tile& T) { return REGS ? T.fx : T.W->from[side()] + E * (lane() - side() * K); }
    static __device__ __forceinline__ unsigned fd(const Tile& T) { return REGS ? T.fd : T.W->from[2] + E * lane(); }
    static __device__ __forceinline__ unsigned fu(const Tile& T) { return REGS ? T.fu : T.W->from[3] + E * lane(); }
};

template <class R>
__device__ __forceinline__ V4<R> mk4(R a, R b, R c, R d) { return V4<R>{a, b, c, d}; }
// A complex number's two parts in one instruction (PK; float: f32x2, the same rounding as
// two scalar operations at half the issue slots).  A cluster's warps with columns of four
// are too few to issue at all times, and the pairs' register moves only lengthen their
// chains: 64^2 over 4 blocks 2.83 us an iteration with it, 2.69 without; over a grid 512^2
// 4.29 with it, 4.60 without.
template <int K, bool CL> constexpr bool kPacked = !(CL && K == 4);
__device__ __forceinline__ u64 bits2(float2 a) { return *reinterpret_cast<u64*>(&a); }
template <bool PK>
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    if constexpr (!PK) return make_float2(a.x + b.x, a.y + b.y);
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits2(a)), "l"(bits2(b)));
    return *reinterpret_cast<float2*>(&r);
}
template <bool PK>
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    if constexpr (!PK) return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(bits2(a)), "l"(bits2(b)), "l"(bits2(c)));
    return *reinterpret_cast<float2*>(&r);
}
template <bool PK>
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    if constexpr (!PK) return make_float2(a.x - b.x, a.y - b.y);
    return fma2<PK>(b, make_float2(-1.f, -1.f), a);
}
template <bool PK>
__device__ __forceinline__ double2 add2(double2 a, double2 b) { return a + b; }
template <bool PK>
__device__ __forceinline__ double2 sub2(double2 a, double2 b) { return a - b; }
template <bool PK>
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
    return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
template <class R>
__device__ __forceinline__ V2<R> up(const V4<R>& s) { return mk(s.x, s.y); }   // the two spin components
template <class R>
__device__ __forceinline__ V2<R> dn(const V4<R>& s) { return mk(s.z, s.w); }
template <class R>
__device__ __forceinline__ V4<R> join(V2<R> a, V2<R> b) { return mk4<R>(a.x, a.y, b.x, b.y); }

template <class R, bool PK>
__device__ __forceinline__ V2<R> half1(const V4<R>& s) { return sub2<PK>(up<R>(s), dn<R>(s)); }
template <class R, bool PK>
__device__ __forceinline__ V2<R> half2(const V4<R>& s, V2<R> u1) { return cjmul(u1, add2<PK>(up<R>(s), dn<R>(s))); }
template <class R>
__device__ __forceinline__ V2<R> half3(const V4<R>& s) { return mk(s.x - s.w, s.y + s.z); }
template <class R>
__device__ __forceinline__ V2<R> half4(const V4<R>& s, V2<R> u2) { return cjmul(u2, mk(s.x + s.w, s.y - s.z)); }

// w += the hopping terms f2 (from above) and b2 (from below): (f + b, i (f - b))
template <class R, bool PK>
__device__ __forceinline__ void hop2(V4<R>& w, V2<R> f, V2<R> b) {
    const V2<R> s = add2<PK>(add2<PK>(up<R>(w), f), b);
    w.x = s.x;
    w.y = s.y;
    w.z += b.y - f.y;
    w.w += f.x - b.x;
}

// The first half of w = g5Dw S: sends the tile's faces, then everything that
// does not come through one.  The links carry the factor -1/2.
template <class R, int K, bool CL>
__device__ __forceinline__ void stencil_inner(const Tile& T, const V4<R> (&S)[K],
                                              const V2<R> (&u1)[K], const V2<R> (&u2)[K], R m2, V2<R>* box,
                                              u64 to, unsigned seq, V4<R> (&w)[K]) {
    constexpr int E = Slots<R, K, CL>::E;
    constexpr bool PK = kPacked<K, CL>;
    if (T.h == 0) return;
    V2<R> h1[K], h2[K], h4[K];
    {   // rows
        const V2<R> lo = half3<R>(S[0]);
        if (T.dto >= 0) box[T.dto] = lo;
        else send2<CL>(to + Slots<R, K, CL>::sd(T), lo, seq);
        constexpr int J = K > 1 ? K - 2 : 0;   // tiles have K or K - 1 rows (res_plan)
        const bool full = T.h == K;
        h4[K - 1] = half4<R>(S[K - 1], u2[K - 1]);
        h4[J] = half4<R>(S[J], u2[J]);
        const V2<R> hi = mk(full ? h4[K - 1].x : h4[J].x, full ? h4[K - 1].y : h4[J].y);
        if (T.uto >= 0) box[T.uto] = hi;
        else send2<CL>(to + Slots<R, K, CL>::su(T), hi, seq);
    }
#pragma unroll
    for (int j = 0; j < K; j++) {
        h1[j] = half1<R, PK>(S[j]);
        h2[j] = half2<R, PK>(S[j], u1[j]);
        if (j + 2 < K) h4[j] = half4<R>(S[j], u2[j]);
    }
    if (T.el || T.er) {   // columns
        if (T.xto >= 0) {
#pragma unroll
            for (int j = 0; j < K; j++) box[T.xto + j] = T.el ? h1[j] : h2[j];
        } else {
#pragma unroll
            for (int j = 0; j < K; j++) send2<CL>(to + Slots<R, K, CL>::sx(T) + E * j, T.el ? h1[j] : h2[j], seq);
        }
    }
    const V2<R> mm = mk(m2, m2), mn = mk(-m2, -m2), zero = mk(R(0), R(0));
#pragma unroll
    for (int j = 0; j < K; j++) {
        V2<R> fh = mk(__shfl_sync(0xffffffffu, h1[j].x, T.srcR), __shfl_sync(0xffffffffu, h1[j].y, T.srcR));
        V2<R> b1 = mk(__shfl_sync(0xffffffffu, h2[j].x, T.srcL), __shfl_sync(0xffffffffu, h2[j].y, T.srcL));
        if (T.er) fh = zero;
        if (T.el) b1 = zero;
        const V2<R> f1 = cmul(u1[j], fh);
        w[j] = join<R>(fma2<PK>(mm, up<R>(S[j]), add2<PK>(f1, b1)), fma2<PK>(mn, dn<R>(S[j]), sub2<PK>(f1, b1)));
        // along i2 inside the tile; the bond to a missing highest row carries zeros from above only
        V2<R> f2 = zero, b2 = zero;
        if (j + 1 < K) f2 = cmul(u2[j], half3<R>(S[j + 1 < K ? j + 1 : j]));
        if (j > 0) b2 = h4[j > 0 ? j - 1 : 0];
        if (j == K - 1 && T.h < K) b2 = zero;
        hop2<R, PK>(w[j], f2, b2);
    }
}

// The second half: the faces of other tiles.  Those of other blocks are asked for
// first, `meanwhile` runs while the answers are on their way, and what has not
// arrived by then is polled.  False when a wait gave up.
template <class R, int K, bool CL, class F>
__device__ __forceinline__ bool stencil_faces(const Tile& T, const V2<R> (&u1)[K], const V2<R> (&u2)[K], V2<R>* box,
                                              u64 from, const TeamComm& C, unsigned seq, V4<R> (&w)[K], F meanwhile) {
    constexpr int BOX = ResSm<R, K>::BOX;
    constexpr bool PK = kPacked<K, CL>;
    const int lane = threadIdx.x & 31;
    V2<R>* mine = box + ((threadIdx.x >> 5) - 1) * BOX;
    Arrival<R> qx, qd, qu;
    auto ask = [&]() {
        if (T.rd) qd.template ask<CL>(from + Slots<R, K, CL>::fd(T));
        if (T.ru) qu.template ask<CL>(from + Slots<R, K, CL>::fu(T));
        if (T.rx) qx.template ask<CL>(from + Slots<R, K, CL>::fx(T));
    };
    ask();
    V2<R> lo, hi;
    if (Slots<R, K, CL>::PRE) lo = mine[2 * K + lane], hi = mine[2 * K + 32 + lane];
    meanwhile();
    if (T.h == 0) return true;
    Patience pt;
    bool ok = true;
    for (;;) {
        const bool ready = (!T.rd || qd.here(seq)) && (!T.ru || qu.here(seq)) && (!T.rx || qx.here(seq));
        if (__all_sync(0xffffffffu, ready)) break;
        if (!(ok = pt.more(C))) break;
        ask();
    }
    if (T.rx) mine[lane] = qx.val();
    __syncwarp();
    V2<R> e[K];
    if (Slots<R, K, CL>::PRE)
#pragma unroll
        for (int j = 0; j < K; j++) e[j] = mine[(T.er ? K : 0) + j];
    if (!Slots<R, K, CL>::PRE) lo = mine[2 * K + lane], hi = mine[2 * K + 32 + lane];
    if (T.rd) lo = qd.val();
    if (T.ru) hi = qu.val();
    w[0].x += lo.x;
    w[0].y += lo.y;
    w[0].z += lo.y;
    w[0].w -= lo.x;
    {   // the top row is K - 1 or K - 2; by selection, as a branch on it would index w and u2 in memory
        constexpr int J = K > 1 ? K - 2 : 0;
        const bool full = T.h == K;
        const V2<R> f = cmul(mk(full ? u2[K - 1].x : u2[J].x, full ? u2[K - 1].y : u2[J].y), hi);
        const V2<R> fa = mk(full ? f.x : R(0), full ? f.y : R(0));
        w[K - 1].x += fa.x;
        w[K - 1].y += fa.y;
        w[K - 1].z -= fa.y;
        w[K - 1].w += fa.x;
        if (K > 1) {
            const V2<R> fb = mk(full ? R(0) : f.x, full ? R(0) : f.y);
            w[J].x += fb.x;
            w[J].y += fb.y;
            w[J].z -= fb.y;
            w[J].w += fb.x;
        }
    }
    if (T.el || T.er) {
        const V2<R> sg = T.er ? mk(R(1), R(1)) : mk(R(-1), R(-1));
#pragma unroll
        for (int j = 0; j < K; j++) {
            if (j == K - 1 && T.h < K) break;   // no such row: its inbox entry is never written
            if (!Slots<R, K, CL>::PRE) e[j] = mine[(T.er ? K : 0) + j];
            if (T.er) e[j] = cmul(u1[j], e[j]);
            w[j] = join<R>(add2<PK>(up<R>(w[j]), e[j]), fma2<PK>(sg, e[j], dn<R>(w[j])));
        }
    }
    return ok;
}

template <class R, bool PK = true>
__device__ __forceinline__ R norm4(const V4<R>& a) {
    const V2<R> n = fma2<PK>(up<R>(a), up<R>(a), fma2<PK>(dn<R>(a), dn<R>(a), mk(R(0), R(0))));
    return n.x + n.y;
}
template <class R, bool PK = true>
__device__ __forceinline__ V4<R> axpy4(R a, const V4<R>& x, const V4<R>& y) {
    const V2<R> aa = mk(a, a);
    return join<R>(fma2<PK>(aa, up<R>(x), up<R>(y)), fma2<PK>(aa, dn<R>(x), dn<R>(y)));
}

// ---------------------------------------------------------------------------
// Multishift solves (MS): the base system as above, and every other shift's x and p
// in shared memory, updated by warps of their own behind the base system.
constexpr int kResShifts = QED2D_MAXPOLES;
struct ResMs {
    int n, base, nw;             // shifts, the base system's, worker warps of a block
    double d[kResShifts];        // mu_i^2 - mu_base^2
    double2* x[kResShifts];
};
struct ResMsBlock {              // the shifts' scalars of an iteration
    double a[kResShifts], b[kResShifts], z[kResShifts];
    int state[kResShifts];       // 1: x_i += a p_i, 2: p_i = z r + b p_i as well
    int flag[2];                 // how the round ended, two rounds in turn
};

// what the threads of a block share
struct ResBlock {
    int nwk;                       // worker threads
    double part[2][32 * kResWarps];   // the threads' partials of the two sums
    ResSc sc;
    int abort;                 // a wait of this block gave up
    double next;
    WarpFace face[kResWarps];
    int4 tile[kResWarps];      // first site (x, y), lanes, rows of each warp's tile
    ResRep rep;
    TeamComm C;
};

// The scalar warp (warp 0: the scheduler prefers the oldest of its warps, and this
// one is on the way of all): one step per sum, in step with the workers.  Returns the
// number of sums so far.
template <bool MIXED, bool CL, bool MS = false>
__device__ __forceinline__ unsigned res_scalar(const ResP& P, ResBlock& B, unsigned seq, u64& base0, u64& base1,
                                               const ResMs* M = nullptr, ResMsBlock* S = nullptr) {
    enum { X_BEGIN, X_RR, X_PAP, X_FENCE, X_TRUE };   // what the coming exchange sums (X_PAP in FP64: a direct iteration)
    constexpr int NV = MIXED ? 1 : 2;
    const int nw = MS ? M->nw : (int)(blockDim.x >> 5) - 1, nth = 32 * (nw + 1), lane = threadIdx.x & 31;
    // |r|^2, its inverse, the inverse of the last alpha
    double rr = 0.0, inv_rr = 0.0, inv_a = 0.0, beta = 0.0;
    double maxrr = 0.0, thr = 0.0;   // the largest |r|^2 since the last update; below thr: update
    double s = 1.0, rr64 = 0.0, bb = 0.0, tol = 0.0;
    double rr_last = 1.0, pap_last = 4.0, dir_est = 1.0;   // the last sums
    int ex = 0;   // the coming ones' fixed-point scale (team_sum_fixed)
    int k = 0, nupd = 0, fences = 0, flag = RF_GO, next = X_BEGIN;
    bool conv = false, fresh = true;
    // MS: lane i's shift; the base system's last alpha and the alpha and beta before
    double zs = 1.0, zp = 1.0, a_now = 0.0, a_last = 1.0, b_now = 0.0;
    bool act = MS && lane < M->n && lane != M->base;
    int round = 0;                  // barriers with the shift warps so far
#pragma unroll 1
    for (;;) {
        ++seq;
        const bool dead = ld_volatile_int(&B.abort) != 0;   // noted by a worker
        Sums tot{0.0, 0.0}, v;
        bool ok = true;
        bar_sync_n(1, nth);   // the workers' partials are in
        {
            double a[4] = {0.0, 0.0, 0.0, 0.0}, c[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int i = 0; i < kResWarps; i++)
                if (i < nw) {
                    a[i & 3] += B.part[0][32 * i + lane];
                    if (NV > 1) c[i & 3] += B.part[1][32 * i + lane];
                }
            v.g = (a[0] + a[1]) + (a[2] + a[3]);
            v.d = (c[0] + c[1]) + (c[2] + c[3]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                v.g += __shfl_xor_sync(0xffffffffu, v.g, o);
                if (NV > 1) v.d += __shfl_xor_sync(0xffffffffu, v.d, o);
            }
        }
        if (B.C.nb == 1) {
            tot = v;
        } else if constexpr (CL) {
            ok = cluster_sum_slots<NV>(B.C, seq, v, tot);
        } else {
            bool exact = false;
            if (next != X_BEGIN) {
                u64 bs = (seq & 1u) ? base1 : base0;
                ok = team_sum_fixed<NV>(B.C, seq, v, ex, bs, tot, next == X_RR, exact);
                if (seq & 1u) base1 = bs;
                else base0 = bs;
            }
            if (!exact && ok) ok = team_sum_slots<NV>(B.C, seq, v, tot);
        }
        double alpha = 0.0;
        const double inv_old = inv_rr;
        const bool all = MS && (next == X_BEGIN || next == X_RR);   // the shift warps join this barrier
        const bool step = MS && next == X_RR && !fresh;             // and an iteration is behind them
        if (next == X_PAP) {   // <p, (A + mu2) p>
            alpha = rr / tot.g;
            if (MIXED) pap_last = tot.g;
            flag = RF_GO;
            k++;
            next = X_RR;
        } else if (next == X_RR) {   // |r|^2; FP64: and |g5Dw r|^2
            rr_last = tot.g;
            if (!fresh && ((MIXED ? tot.g < thr : tot.g < tol) || k == P.maxiter)) {
                flag = MIXED ? RF_UPD : RF_FIN;
                next = X_FENCE;
                fences = MIXED ? 2 : 1;
                nupd += MIXED;
                conv = !MIXED && tot.g < tol;
                rr64 = MIXED ? tot.g / (s * s) : tot.g;
            } else {
                if (!fresh) beta = tot.g * inv_rr;
                if (MIXED) {
                    next = X_PAP;
                } else {
                    pap_last = tot.d;
                    const double rar = tot.d + P.mu2 * tot.g, pap = rar - beta * (tot.g * inv_a);   // beta = inv_a = 0 at first
                    const bool dir = !fresh && !(pap > 0.5 * rar);   // more subtracted than left
                    alpha = tot.g / pap;
                    dir_est = rar;
                    k++;
                    if (__builtin_expect(dir, 0)) {
                        alpha = 0.0;
                        k--;
                        flag = RF_DIR;
                        next = X_PAP;
                    }
                }
                if (fresh) maxrr = tot.g;
                fresh = false;
                rr = tot.g;
            }
        } else if (next == X_BEGIN) {   // |b|^2
            bb = rr64 = tot.g;
            tol = P.eps * bb;
            conv = bb == 0.0;
            if (MIXED && !conv) s = 1.0 / sqrt(bb);
            if (!MIXED) rr_last = bb, pap_last = 4.0 * bb;
            flag = conv ? RF_ZERO : P.guess ? RF_UPD : P.maxiter > 0 ? RF_GO : RF_STOP;
            next = P.guess ? X_FENCE : X_RR;
            fences = 1;
        } else {   // |b - (A + mu2) x|^2
            rr64 = tot.g;
            conv = tot.g < tol;
            if (conv || k == P.maxiter) {
                flag = RF_STOP;
            } else {
                flag = RF_GO;
                next = X_RR;
                if (MIXED) {
                    const double sn = 1.0 / sqrt(tot.g);
                    if (nupd) beta = (tot.g * s * s * inv_rr) * (sn / s);
                    s = sn;
                    fresh = true;
                    rr_last = 1.0;
                    pap_last = 4.0;
                } else {   // a warm start
                    rr_last = tot.g;
                    pap_last = 4.0 * tot.g;
                }
            }
        }
        if (!ok || dead) flag = RF_ABORT;
        if (lane == 0) {
            if (MIXED) {
                B.sc.cf = make_float2((float)(next == X_PAP ? beta : alpha), __int_as_float(flag));
            } else {
                B.sc.alpha = alpha;
                B.sc.beta = beta;
                B.sc.flag = flag;
            }
            B.sc.s = s;
        }
        if (all) bar_sync_n(5, blockDim.x);
        else bar_sync_n(3, nth);
        if constexpr (MS) {
            if (step) {   // the shifts' recurrences (k_cg_multishift's), lane i shift i
                const double b_new = tot.g * inv_old;
                if (act) {
                    const double zn = zs * zp * a_last / (a_now * b_now * (zp - zs) + zp * a_last * (1.0 + M->d[lane] * a_now));
                    const double q = zn / zs;
                    S->a[lane] = a_now * q;
                    S->b[lane] = b_new * q * q;
                    S->z[lane] = zn;
                    zp = zs;
                    zs = zn;
                    act = !(zn * zn * tot.g < tol);
                    S->state[lane] = act ? 2 : 1;
                } else {
                    S->state[lane] = 0;
                }
                a_last = a_now;
                b_now = b_new;
            }
            if (alpha != 0.0) a_now = alpha;   // a direct iteration's comes one sum later
            if (all) {
                if (lane == 0) S->flag[round & 1] = flag == RF_DIR ? RF_GO : flag;
                round++;
                bar_arrive_n(4, blockDim.x - 32 * nw);
            }
        }
        if (flag >= RF_STOP) break;
        // off the way from one exchange to the next
        inv_rr = 1.0 / rr;
        if (!MIXED && alpha != 0.0) inv_a = 1.0 / alpha;
        maxrr = fmax(maxrr, rr);
        thr = fmax(P.delta2 * maxrr, tol * s * s);
        if (next == X_FENCE) {
            // Exchanges that order the blocks' FP64 stores, apart from the loop's path (in it
            // they cost a 64^2 mixed CG 4%).  The fences are this warp's own: the first releases
            // what the workers stored before the barrier, the second acquires the others'.
            do {
                ++seq;
                const bool lost = ld_volatile_int(&B.abort) != 0;
                bool got = true;
                Sums zero{0.0, 0.0}, sum;
                bar_sync_n(1, nth);
                __threadfence();
                if (B.C.nb > 1) {
                    if constexpr (CL) {
                        got = cluster_sum_slots<1>(B.C, seq, zero, sum);
                    } else {
                        bool exact;
                        u64 bs = (seq & 1u) ? base1 : base0;
                        got = team_sum_fixed<NV>(B.C, seq, zero, 0, bs, sum, false, exact);
                        if (seq & 1u) base1 = bs;
                        else base0 = bs;
                    }
                }
                __threadfence();
                if (!got || lost) flag = RF_ABORT;
                else if (flag == RF_FIN) flag = RF_STOP;
                if (lane == 0) {
                    if (MIXED) B.sc.cf = make_float2(0.f, __int_as_float(flag));
                    else B.sc.flag = flag;
                }
                bar_sync_n(3, nth);
            } while (--fences > 0 && flag < RF_STOP);
            if (flag >= RF_STOP) break;
            next = X_TRUE;
        }
        ex = fixed_exponent(Sums{next == X_RR ? rr_last : next == X_PAP ? (MIXED ? pap_last : dir_est) : next == X_TRUE ? rr64 : 1.0, pap_last});
    }
    if (flag != RF_ABORT && B.C.rank == 0 && lane == 0) {
        const int it = conv ? k : P.maxiter;
        P.out[B.rep.id] = ResOut{it, conv, nupd, 0, rr64, bb};
        if (P.single) {
            DevCtl* c = P.ctl;
            c->last_iters = it;
            c->last_updates = nupd;
            c->last_conv = conv;
            c->last_relres = bb > 0.0 ? rr64 / bb : 0.0;
            c->iters_total += it;
            if (c->status == 0 && !conv) c->status = QED2D_ERR_NOT_CONVERGED;
        }
    }
    return seq;
}

// a worker's column of sites in the lattice
struct Column {
    int i1, y0, h;        // h = 0: none
    long long g0;         // site of row 0
};
__device__ __forceinline__ Column column_of(const ResBlock& B) {
    const int4 t = B.tile[(threadIdx.x >> 5) - 1];
    const int lane = threadIdx.x & 31;
    return Column{t.x + lane, t.y, lane < t.z ? t.w : 0, t.x + lane + (long long)B.rep.L1 * t.y};
}
__device__ __forceinline__ Site col_site(const Column& c, int L1, int L2, int j) {
    const long long V = (long long)L1 * L2;
    Site q;
    q.i1 = c.i1;
    q.i2 = c.y0 + j;
    q.ok = true;
    q.x = c.g0 + (long long)j * L1;
    q.xp1 = q.i1 + 1 == L1 ? q.x - (L1 - 1) : q.x + 1;
    q.xm1 = q.i1 == 0 ? q.x + (L1 - 1) : q.x - 1;
    q.xp2 = q.i2 + 1 == L2 ? (long long)q.i1 : q.x + L1;
    q.xm2 = q.i2 == 0 ? q.x + (V - L1) : q.x - L1;
    return q;
}
// workers: the thread's partials of the coming exchange
__device__ __forceinline__ void put_part(ResBlock& B, double g) {
    B.part[0][threadIdx.x - 32] = g;
    bar_arrive_n(1, B.nwk + 32);
}
__device__ __forceinline__ void put_part(ResBlock& B, double g, double d) {
    B.part[1][threadIdx.x - 32] = d;
    put_part(B, g);
}
// A warp whose wait for a face gave up leaves a note that the scalar warp finds at a
// later sum and turns into RF_ABORT for the whole block, so that all its threads leave at
// the same barrier.
__device__ __forceinline__ void note(ResBlock& B, bool ok) {
    if (!ok) *(volatile int*)&B.abort = 1;
}
// workers: the end of a sum
template <bool MIXED>
__device__ __forceinline__ int wait_scalar(ResBlock& B, bool all = false) {
    if (all) bar_sync_n(5, blockDim.x);   // MS: with the shift warps
    else bar_sync_n(3, B.nwk + 32);
    if constexpr (MIXED) return __float_as_int(B.sc.cf.y);
    else return B.sc.flag;
}

// Workers: the FP64 true residual b - (A + mu2) x, after x += x32 / s (add), and,
// where the solve goes on, the FP32 residual for the next iteration, left in x32
// (the caller takes it and clears x32).  The stencils read other blocks' x and
// t64, so an exchange follows each of them.  Runs a few times per solve, between
// iterations, when only shared memory holds anything.
template <bool MIXED>
__device__ __forceinline__ int res_update(const ResP& P, ResBlock& B, float4* x32, bool add) {
    const Column c = column_of(B);
    const int nwk = B.nwk, L1 = B.rep.L1, L2 = B.rep.L2;
    const long long V = (long long)L1 * L2, o2 = 2 * B.rep.off;
    const double m2 = B.rep.m2, mu2 = P.mu2;
    double2* xs = P.x + o2;
    double2* t64 = P.t64 + o2;
    double2* r64 = P.r64 + o2;
    const double2* bs = P.b + o2;
    const LkD L{P.U + o2, V};
    if (add) {
        const double inv_s = 1.0 / B.sc.s;
#pragma unroll 1
        for (int j = 0; j < c.h; j++) {
            const long long g = c.g0 + (long long)j * L1;
            const float4 d = x32[j * nwk];
            Pair<double> xv{__ldcg(xs + g), __ldcg(xs + g + V)};
            xv.a = xv.a + inv_s * to_d(make_float2(d.x, d.y));
            xv.b = xv.b + inv_s * to_d(make_float2(d.z, d.w));
            st_d(xs, V, g, xv);
        }
        __threadfence();
        __syncwarp();
        put_part(B, 0.0, 0.0);
        if (wait_scalar<MIXED>(B) == RF_ABORT) return RF_ABORT;
    }
#pragma unroll 1
    for (int j = 0; j < c.h; j++) {
        const Site q = col_site(c, L1, L2, j);
        st_d(t64, V, q.x, g5dw_at<double>(SpDcg{xs, V}, L, q, m2));
    }
    __threadfence();
    __syncwarp();
    put_part(B, 0.0, 0.0);
    if (wait_scalar<MIXED>(B) == RF_ABORT) return RF_ABORT;
    double n = 0.0;
#pragma unroll 1
    for (int j = 0; j < c.h; j++) {
        const Site q = col_site(c, L1, L2, j);
        const Pair<double> a = g5dw_at<double>(SpDcg{t64, V}, L, q, m2), xc = SpDcg{xs, V}.ld(q.x);
        Pair<double> rv;
        rv.a = __ldg(bs + q.x) - (a.a + mu2 * xc.a);
        rv.b = __ldg(bs + q.x + V) - (a.b + mu2 * xc.b);
        st_d(r64, V, q.x, rv);
        n += norm2(rv.a) + norm2(rv.b);
    }
    put_part(B, n, 0.0);
    const int flag = wait_scalar<MIXED>(B);
    if (flag != RF_GO || !MIXED) return flag;
    const double s = B.sc.s;
#pragma unroll 1
    for (int j = 0; j < c.h; j++) {
        const long long g = c.g0 + (long long)j * L1;
        const float2 a = to_f(s * r64[g]), d = to_f(s * r64[g + V]);
        x32[j * nwk] = mk4<float>(a.x, a.y, d.x, d.y);
    }
    return flag;
}

// Workers: |b|^2 and (mixed) the first FP32 residual, left in x32.  x = 0 without a
// guess where the solve adds to it or has nothing to do.
template <bool MIXED, bool MS = false>
__device__ __forceinline__ int res_begin(const ResP& P, ResBlock& B, float4* x32) {
    const Column c = column_of(B);
    const int nwk = B.nwk, L1 = B.rep.L1;
    const long long V = (long long)L1 * B.rep.L2, o2 = 2 * B.rep.off;
    double acc = 0.0;
#pragma unroll 1
    for (int j = 0; j < c.h; j++) {
        const long long g = o2 + c.g0 + (long long)j * L1;
        acc += norm2(__ldg(P.b + g)) + norm2(__ldg(P.b + V + g));
    }
    put_part(B, acc, 0.0);
    const int flag = wait_scalar<MIXED>(B, MS);
    if (flag == RF_ABORT || flag == RF_UPD) return flag;
    const double2 z = make_double2(0, 0);
    const double s = B.sc.s;
#pragma unroll 1
    for (int j = 0; j < c.h; j++) {
        const long long g = o2 + c.g0 + (long long)j * L1;
        if (flag == RF_ZERO || (!P.guess && (MIXED || flag != RF_GO))) {
            P.x[g] = z;
            P.x[g + V] = z;
        }
        if (flag == RF_ZERO || (!MIXED && flag == RF_STOP && !P.guess)) {   // zero source: zero solution
            P.t64[g] = z;
            P.t64[g + V] = z;
        }
        if (MIXED) {
            const float2 a = to_f(s * __ldg(P.b + g)), d = to_f(s * __ldg(P.b + V + g));
            x32[j * nwk] = mk4<float>(a.x, a.y, d.x, d.y);
        }
    }
    return flag;
}

// Workers, FP64: x (+)= the solve's, and g5Dw x, which reads other blocks' x.
__device__ __forceinline__ void res_finish(const ResP& P, ResBlock& B, const double4x* xs) {
    const Column c = column_of(B);
    const int nwk = B.nwk, L1 = B.rep.L1, L2 = B.rep.L2;
    const long long V = (long long)L1 * L2, o2 = 2 * B.rep.off;
    double2* x = P.x + o2;
#pragma unroll 1
    for (int j = 0; j < c.h; j++) {
        const long long g = c.g0 + (long long)j * L1;
        const double4x d = xs[j * nwk];
        Pair<double> v{make_double2(d.x, d.y), make_double2(d.z, d.w)};
        if (P.guess) {
            v.a = x[g] + v.a;
            v.b = x[g + V] + v.b;
        }
        st_d(x, V, g, v);
    }
    __threadfence();
    __syncwarp();
    put_part(B, 0.0, 0.0);
    if (wait_scalar<false>(B) == RF_ABORT || !P.want_g5) return;
#pragma unroll 1
    for (int j = 0; j < c.h; j++) {
        const Site q = col_site(c, L1, L2, j);
        st_d(P.t64 + o2, V, q.x, g5dw_at<double>(SpDcg{x, V}, LkD{P.U + o2, V}, q, B.rep.m2));
    }
}

// Lane 0 of a worker warp: the warp's tile and where its faces go.
template <class R, int K, bool CL>
__device__ __forceinline__ void res_place(ResBlock& B, int warp) {
    constexpr int N = Num<R>::SLOTS;
    const ResRep& L = B.rep;
    const int rank = B.C.rank, nslots = B.C.nslots;
    const int bi = rank % L.bx, bj = rank / L.bx;
    const int c0 = bi * L.ntx / L.bx, c1 = (bi + 1) * L.ntx / L.bx;
    const int r0 = bj * L.nty / L.by, r1 = (bj + 1) * L.nty / L.by;
    const int nc = c1 - c0, nr = r1 - r0;
    const int wy = warp / L.wx, wx = warp - wy * L.wx;
    if (rank >= L.bx * L.by || wx >= nc || wy >= nr) {
        B.tile[warp] = make_int4(0, 0, 0, 0);
        return;
    }
    const int tc = c0 + wx, tr = r0 + wy;
    const int x0 = (int)((long long)tc * L.L1 / L.ntx), x1 = (int)((long long)(tc + 1) * L.L1 / L.ntx);
    const int y0 = (int)((long long)tr * L.L2 / L.nty), y1 = (int)((long long)(tr + 1) * L.L2 / L.nty);
    B.tile[warp] = make_int4(x0, y0, x1 - x0, y1 - y0);
    WarpFace& W = B.face[warp];
    W.warp[0] = wx > 0 ? warp - 1 : (L.bx == 1 ? warp + nc - 1 : -1);
    W.warp[1] = wx < nc - 1 ? warp + 1 : (L.bx == 1 ? warp - (nc - 1) : -1);
    W.warp[2] = wy > 0 ? warp - L.wx : (L.by == 1 ? warp + (nr - 1) * L.wx : -1);
    W.warp[3] = wy < nr - 1 ? warp + L.wx : (L.by == 1 ? warp - (nr - 1) * L.wx : -1);
    const int nb[4] = {(bi == 0 ? L.bx - 1 : bi - 1) + L.bx * bj, (bi == L.bx - 1 ? 0 : bi + 1) + L.bx * bj,
                       bi + L.bx * (bj == 0 ? L.by - 1 : bj - 1), bi + L.bx * (bj == L.by - 1 ? 0 : bj + 1)};
    // A block's slots: left and right columns [wy][K], lower and upper rows [wx][32].
    // A face goes to the opposite side of the neighbour: its tile has this one's
    // position along the face.
    const int at[4] = {wy * K, (L.wy + wy) * K, 2 * L.wy * K + wx * 32, 2 * L.wy * K + (L.wx + wx) * 32};
    for (int d = 0; d < 4; d++) {
        if constexpr (CL) {
            W.to[d] = map_rank((unsigned)B.C.slots + 16 * N * at[d ^ 1], nb[d]);
            W.from[d] = 16 * N * at[d];
        } else {
            W.to[d] = (unsigned)(nb[d] * 2 * nslots + N * at[d ^ 1]) * 16;
            W.from[d] = (unsigned)(rank * 2 * nslots + N * at[d]) * 16;
        }
    }
}

// Returns the number of halo exchanges so far.
template <class R, int K, bool CL, bool MS = false>
__device__ __forceinline__ unsigned res_worker(const ResP& P, ResBlock& B, char* dyn, unsigned seq,
                                               V4<R>* rbuf = nullptr) {   // MS: r for the shift warps, two copies in turn
    constexpr bool MIXED = std::is_same<R, float>::value;
    constexpr int BOX = ResSm<R, K>::BOX;
    constexpr bool PK = kPacked<K, CL>;
    constexpr bool OLD = K * sizeof(R) <= 8;   // registers for r before the last update, so that p can wait
    const int nwk = B.nwk, lane = threadIdx.x & 31;
    V4<R>* xs = reinterpret_cast<V4<R>*>(dyn) + (threadIdx.x - 32);   // x: row j at xs[j * nwk]
    V4<R>* ps = xs + K * nwk;                                         // p and q likewise: A p (FP64), or t between updates (mixed)
    V4<R>* qs = ps + K * nwk;
    V2<R>* box0 = reinterpret_cast<V2<R>*>(dyn + (size_t)nwk * 3 * K * sizeof(V4<R>));
    V2<R>* box1 = box0 + (nwk >> 5) * BOX;
    if (lane == 0) res_place<R, K, CL>(B, (threadIdx.x >> 5) - 1);
    __syncwarp();
    Tile T;
    {
        const int4 t4 = B.tile[(threadIdx.x >> 5) - 1];
        T.w = t4.z;
        T.h = t4.w;
        T.el = lane == 0;
        T.er = lane == T.w - 1;
        T.srcR = min(lane + 1, 31);
        T.srcL = lane < T.w ? max(lane - 1, 0) : 31;   // lanes past the tile take lane 31's zero
        const WarpFace& F = B.face[(threadIdx.x >> 5) - 1];
        T.xto = F.warp[T.el ? 0 : 1] < 0 ? -1 : F.warp[T.el ? 0 : 1] * BOX + (T.el ? K : 0);
        T.dto = F.warp[2] < 0 ? -1 : F.warp[2] * BOX + 2 * K + 32 + lane;
        T.uto = F.warp[3] < 0 ? -1 : F.warp[3] * BOX + 2 * K + lane;
        T.W = &F;
        Slots<R, K, CL>::init(T);
        const int side = Slots<R, K, CL>::side();
        T.rx = T.h > 0 && lane < 2 * K && F.warp[side] < 0 && lane - side * K < T.h;
        T.rd = T.h > 0 && T.dto < 0;
        T.ru = T.h > 0 && T.uto < 0;
    }
    // the slots of the two exchanges of an iteration (in a cluster WarpFace::to holds addresses)
    const u64 from1 = B.C.slots, from0 = from1 + (u64)B.C.nslots * 16, to1 = CL ? 0 : from1, to0 = to1 + (u64)B.C.nslots * 16;
    const V4<R> zero = mk4<R>(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < K; j++) xs[j * nwk] = ps[j * nwk] = qs[j * nwk] = zero;
    int flag = res_begin<MIXED, MS>(P, B, reinterpret_cast<float4*>(xs));
    bool first = true;
    V2<R> u1[K], u2[K];
    V4<R> r[K], t[K], w[K];
    V4<R> ro[K];   // FP64: r before the last update
    R alpha = 0, beta = 0;
    const R m2 = (R)B.rep.m2, mu2 = (R)P.mu2;
    int m = 0;   // MS: iterations
    for (;;) {
        const double2* src = P.b;
        if (flag != RF_GO) {
            if (flag != RF_UPD) return seq;
            flag = res_update<MIXED>(P, B, reinterpret_cast<float4*>(xs), !first);
            if (flag != RF_GO) return seq;
            src = P.r64;
        }
        first = false;
        const Column c = column_of(B);
#pragma unroll
        for (int j = 0; j < K; j++) {
            u1[j] = u2[j] = mk(R(0), R(0));
            w[j] = ro[j] = zero;
            if constexpr (MIXED) {
                t[j] = qs[j * nwk];
                r[j] = xs[j * nwk];
                xs[j * nwk] = zero;
            } else {
                t[j] = r[j] = zero;
            }
            if (j < c.h) {
                const long long g = 2 * B.rep.off + c.g0 + (long long)j * B.rep.L1, V = (long long)B.rep.L1 * B.rep.L2;
                const double2 a = __ldg(P.U + g), d = __ldg(P.U + V + g);
                u1[j] = mk(R(-0.5) * (R)a.x, R(-0.5) * (R)a.y);
                u2[j] = mk(R(-0.5) * (R)d.x, R(-0.5) * (R)d.y);
                if constexpr (!MIXED) {
                    const double2 e = src[g], f = src[g + V];
                    r[j] = mk4<R>(e.x, e.y, f.x, f.y);
                }
            }
        }
        alpha = beta = 0;
        if constexpr (MIXED) {
            for (;;) {
                {
                    R f = 0;
#pragma unroll
                    for (int j = 0; j < K; j++) f += norm4<R, PK>(r[j]);
                    put_part(B, (double)f);
                }
                ++seq;   // w = g5Dw r
                stencil_inner<R, K, CL>(T, r, u1, u2, m2, box0, to0, seq, w);
                bar_sync_n(2, nwk);
                note(B, stencil_faces<R, K, CL>(T, u1, u2, box0, from0, B.C, seq, w, [&]() {   // x += alpha p of the last iteration
#pragma unroll
                    for (int j = 0; j < K; j++) xs[j * nwk] = axpy4<R, PK>(alpha, ps[j * nwk], xs[j * nwk]);
                }));
                flag = wait_scalar<MIXED>(B);
                if (flag != RF_GO) break;
                beta = B.sc.cf.x;
                {
                    R f = 0;
#pragma unroll
                    for (int j = 0; j < K; j++) {
                        t[j] = axpy4<R, PK>(beta, t[j], w[j]);
                        f += norm4<R, PK>(t[j]);
                    }
                    double d = (double)f;
                    if (mu2 != R(0)) {   // with a shift <p, A p> needs p now, else it is formed during the exchange
                        f = 0;
#pragma unroll
                        for (int j = 0; j < K; j++) {
                            const V4<R> pn = axpy4<R, PK>(beta, ps[j * nwk], r[j]);
                            ps[j * nwk] = pn;
                            f += norm4<R, PK>(pn);
                        }
                        d += P.mu2 * (double)f;
                    }
                    put_part(B, d);
                }
                ++seq;   // w = g5Dw t
                stencil_inner<R, K, CL>(T, t, u1, u2, m2, box1, to1, seq, w);
                bar_sync_n(2, nwk);
                note(B, stencil_faces<R, K, CL>(T, u1, u2, box1, from1, B.C, seq, w, [&]() {
                    if (mu2 == R(0))
#pragma unroll
                        for (int j = 0; j < K; j++) ps[j * nwk] = axpy4<R, PK>(beta, ps[j * nwk], r[j]);
                }));
                if (wait_scalar<MIXED>(B) == RF_ABORT) return seq;
                alpha = B.sc.cf.x;
#pragma unroll
                for (int j = 0; j < K; j++) {
                    if (mu2 != R(0)) w[j] = axpy4<R, PK>(mu2, ps[j * nwk], w[j]);
                    r[j] = axpy4<R, PK>(-alpha, w[j], r[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < K; j++) qs[j * nwk] = t[j];
        } else {
            bool adv = false;   // an iteration's p and x are still to be formed
            bool dir = false;   // a direct iteration: p in the place of r, which waits in qs
            for (;;) {
                ++seq;   // t = g5Dw r
                stencil_inner<R, K, CL>(T, r, u1, u2, m2, box0, to0, seq, t);
                bar_sync_n(2, nwk);
                R g = 0, d = 0;
                bool ok = stencil_faces<R, K, CL>(T, u1, u2, box0, from0, B.C, seq, t, [&]() {
#pragma unroll
                    for (int j = 0; j < K; j++) g += norm4<R, PK>(r[j]);
                });
#pragma unroll
                for (int j = 0; j < K; j++) d += norm4<R, PK>(t[j]);
                put_part(B, dir ? d + P.mu2 * g : (double)g, (double)d);
                ++seq;   // w = g5Dw t
                stencil_inner<R, K, CL>(T, t, u1, u2, m2, box1, to1, seq, w);
                bar_sync_n(2, nwk);
                ok &= stencil_faces<R, K, CL>(T, u1, u2, box1, from1, B.C, seq, w, []() {});
                note(B, ok);
                if (adv) {   // p = r_old + beta p, x += alpha p
#pragma unroll
                    for (int j = 0; j < K; j++) {
                        V4<R> pn = ps[j * nwk];
                        if constexpr (OLD) ps[j * nwk] = pn = axpy4<R, PK>(beta, pn, ro[j]);
                        xs[j * nwk] = axpy4<R, PK>(alpha, pn, xs[j * nwk]);
                    }
                }
#pragma unroll
                for (int j = 0; j < K; j++) {
                    if (mu2 != R(0)) w[j] = axpy4<R, PK>(mu2, r[j], w[j]);
                    if constexpr (OLD) ro[j] = r[j];
                    t[j] = qs[j * nwk];
                }
                flag = wait_scalar<MIXED>(B, MS && !dir);
                alpha = (R)B.sc.alpha;
                beta = (R)B.sc.beta;
                if (flag > RF_DIR) break;
                if (__builtin_expect(flag == RF_DIR, 0)) {
                    dir = true;
                    adv = false;
#pragma unroll
                    for (int j = 0; j < K; j++) {
                        qs[j * nwk] = r[j];
                        r[j] = axpy4<R, PK>(beta, ps[j * nwk], r[j]);
                    }
                    continue;
                }
                adv = true;
                m++;
#pragma unroll
                for (int j = 0; j < K; j++) {   // q = A r + beta q (direct: A p), r -= alpha q
                    V4<R> q = axpy4<R, PK>(beta, t[j], w[j]);
                    if (__builtin_expect(dir, 0)) {
                        q = w[j];
                        r[j] = ro[j] = t[j];
                    }
                    qs[j * nwk] = q;
                    if constexpr (!OLD) ps[j * nwk] = axpy4<R, PK>(beta, ps[j * nwk], r[j]);
                    r[j] = axpy4<R, PK>(-alpha, q, r[j]);
                    if constexpr (MS) rbuf[((m & 1) * K + j) * nwk + threadIdx.x - 32] = r[j];
                }
                dir = false;
            }
            if (flag == RF_FIN) res_finish(P, B, xs);
            return seq;
        }
    }
}

template <class R, int K, bool CL>
__global__ void __launch_bounds__(32 * (kResWarps + 1), 1) k_res_cg(const __grid_constant__ ResP P) {
    extern __shared__ __align__(16) char dyn[];
    __shared__ ResBlock B;
    const int team = blockIdx.x / P.nb;
    if (threadIdx.x == 0) {
        B.abort = 0;
        B.nwk = blockDim.x - 32;
        B.C.nb = P.nb;
        B.C.rank = blockIdx.x - team * P.nb;
        B.C.nslots = P.nslots;
        B.C.polls = P.polls;
        B.C.err = &P.ctl->err;
        if constexpr (CL) {
            B.C.psum = smem_u32(dyn + ResSm<R, K>::bytes((blockDim.x >> 5) - 1));
            B.C.slots = B.C.psum + 4 * kResCluster * 16;
        } else {
            B.C.slots = (u64)(P.slots + (size_t)team * P.nb * 2 * P.nslots);
            B.C.psum = (u64)(P.psum + (size_t)team * 4 * P.nb);
            B.C.acc = P.acc + kResAcc * team;
        }
    }
    if constexpr (CL) {   // no slot carries a tag yet
        ulonglong2* sl = reinterpret_cast<ulonglong2*>(dyn + ResSm<R, K>::bytes((blockDim.x >> 5) - 1));
        for (int i = threadIdx.x; i < 4 * kResCluster + 2 * P.nslots; i += blockDim.x) sl[i] = make_ulonglong2(0, 0);
        cooperative_groups::this_cluster().sync();
    }
    unsigned seq = 0;
    u64 base0 = 0, base1 = 0;
    for (int next = team; next < P.nrep;) {
        if (threadIdx.x == 0) {
            B.rep = P.reps ? P.reps[next] : P.rep0;
            if (P.m2) B.rep.m2 = P.m2[B.rep.id];
        }
        __syncthreads();
        if (threadIdx.x < 32) seq = res_scalar<std::is_same<R, float>::value, CL>(P, B, seq, base0, base1);
        else seq = res_worker<R, K, CL>(P, B, dyn, seq);
        if (CL || P.nteams >= P.nrep) break;
        __syncthreads();
        if ((std::is_same<R, float>::value ? __float_as_int(B.sc.cf.y) : B.sc.flag) == RF_ABORT) break;
        if (threadIdx.x < 32) {   // the team's first block takes the next system for the team
            ++seq;
            int n = 0;
            if (B.C.rank == 0 && threadIdx.x == 0) n = atomicAdd(P.queue, 1);
            Sums tot{(double)__shfl_sync(0xffffffffu, n, 0), 0.0};
            if (P.nb > 1 && !team_sum_slots<1>(B.C, seq, tot, tot)) tot.g = (double)P.nrep;
            if (threadIdx.x == 0) B.next = tot.g;
        }
        __syncthreads();
        next = P.nteams + (int)B.next;
    }
    if (B.C.rank == 0 && threadIdx.x == 0 && ld_volatile_int(&P.ctl->err) != 0)
        atomicCAS(&P.ctl->status, 0, QED2D_ERR_TIMEOUT);
    if constexpr (CL) cooperative_groups::this_cluster().sync();   // others may still write here
}

// ---------------------------------------------------------------------------
// host side
// A kernel's limit of dynamic shared memory belongs to the function on the device, whoever
// launches it: every launch and query asks for all that the device has beside the kernel's
// static shared memory, so that host threads with contexts of other sizes, which share the
// function, never lower the limit under one another's launches.
// (The static part is taken from the types: asking the driver costs 3 us a launch.)
inline int res_allow_smem(const void* kern, size_t static_bytes = sizeof(ResBlock)) {
    int dev = 0, optin = 0;
    QCHECK(cudaGetDevice(&dev));
    QCHECK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    QCHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                optin - (int)((static_bytes + 15) / 16 * 16)));
    return QED2D_OK;
}

inline int res_slots(const ResPlan& p, int per) { return per * (2 * p.wy * p.K + 2 * p.wx * 32); }   // of one buffer of a block

template <class R, int K>
static size_t res_smem(const ResGeom& g) {
    return ResSm<R, K>::bytes(g.nw) + (g.cl ? sizeof(ulonglong2) * (4 * kResCluster + 2 * g.nslots) : 0);
}

template <class R, int K>
static int res_clusters_k(const ResGeom& g) {
    const void* kern = (const void*)k_res_cg<R, K, true>;
    const size_t sm = res_smem<R, K>(g);
    if (res_allow_smem(kern) != QED2D_OK ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g.nb);
    cfg.blockDim = dim3(32 * (g.nw + 1));
    cfg.dynamicSmemBytes = sm;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = g.nb;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <class R, int K, bool CL>
static int res_launch_k(const ResP& P, const ResGeom& g, cudaStream_t stream) {
    const void* kern = (const void*)k_res_cg<R, K, CL>;
    const size_t sm = res_smem<R, K>(g);
    QTRY(res_allow_smem(kern));
    if (CL) QCHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(P.nb * P.nteams - g.missing);
    cfg.blockDim = dim3(32 * (g.nw + 1));
    cfg.dynamicSmemBytes = sm;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    if (CL) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = P.nb;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    QCHECK(cudaLaunchKernelEx(&cfg, k_res_cg<R, K, CL>, P));
    count_launch();
    return QED2D_OK;
}

}  // namespace qed2d
