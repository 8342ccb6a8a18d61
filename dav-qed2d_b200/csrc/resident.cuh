// resident.cuh -- the on-chip CG: the whole state of a solve (links, r, p, t, x; in
// FP32 for the mixed solver, resident.cu, in FP64 for the other, resident_f64.cu) lives in registers and shared memory for the length of the solve, and
// only halos and partial sums leave an SM.
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
// shared memory, a larger one in global memory.  A slot of exchange n is overwritten
// by exchange n + 2, which its sender starts only after every block has published
// its partial of n + 1, i.e. after the slot has been read.
//
// One iteration has two exchanges, each halo + sum: r with |r|^2, t with |t|^2.
// Both stencils run while the sum of their exchange is on its way, and so do the
// updates of p and x (in shared memory), which nothing waits for:
//   w = g5Dw r,  x += alpha p    ; beta      ; t = w + beta t
//   w = g5Dw t,  p = r + beta p  ; alpha     ; r -= alpha w
// (g5Dw is linear, so t = g5Dw p; the recurrences, the reliable updates and the
// FP64 stop rule are those of k_cg_mixed's second form).  One extra warp per block
// does the block's sum, the team's sum and the scalar recurrences.
//
// What bounds it (B200, 1.92 GHz): the exchanges.  64^2 (one cluster of 16 blocks):
// 3700 cycles an iteration, of which 2 x 1500 are sum, exchange and recurrences; 512^2
// (144 blocks): 9000, where both chains take about 4000 an exchange, the workers'
// stencil (355 instructions per site row and iteration, issue slots 44% used) and the
// sums (2600 from partial to total).  Against the grid solver with its state in L2:
// 64^2 4.85 -> 1.89 us per iteration, 128^2 5.95 -> 2.63, 256^2 7.1 -> 4.3,
// 512^2 12.3 -> 5.2 (reliable updates included).
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "resident.h"
#include "stencil.cuh"

namespace qed2d {

constexpr int kResWarps = 15;      // most worker warps of a block (with the scalar warp: 128 registers a thread)
constexpr int kResCluster = 16;    // most blocks of a cluster

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
    u64* acc;                 // fixed-point sums: [team][32] words
    int nslots;               // slots of one buffer of a block
    ResOut* out;
    DevCtl* ctl;
    int single;               // write the context's solve record
};

enum { RF_GO, RF_UPD, RF_FIN, RF_STOP, RF_ZERO, RF_ABORT };   // the last three end the solve

// what the scalar warp hands to the workers after an exchange
struct ResSc {
    double c;       // alpha or beta
    float cf;
    int flag;
    double s;       // scale of the FP32 vectors
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

// dynamic shared memory of a block: per worker warp x, p and (mixed, during updates)
// t of its sites and the inbox of faces from other warps of the block
template <class R, int K>
struct ResSm {
    static constexpr int BOX = 2 * K + 64;   // left, right columns [K], lower, upper rows [32]
    static constexpr int ARRAYS = std::is_same<R, float>::value ? 3 : 2;
    static __host__ __device__ size_t bytes(int nw) {
        return (size_t)nw * (ARRAYS * K * 32 * sizeof(V4<R>) + BOX * sizeof(V2<R>));
    }
};

// a block's place in its team
struct TeamComm {
    u64 slots;           // global halo slots of the team, or this block's in shared memory (CL)
    u64 psum;            // the team's partials, [2][receiving block][sending block], or this block's row pair (CL)
    u64* acc;            // the team's fixed-point sums: two pairs of words (not CL)
    int nb, rank, nslots;
    int* err;
};

// Bounded wait of a warp: false when *err is set or the polls run out.
struct Patience {
    unsigned n = 0;
    __device__ __forceinline__ bool more(int* err) {
        if ((++n & 255u) != 0) return true;
        const int e = ld_volatile_int(err);
        if (__any_sync(0xffffffffu, e != 0)) return false;
        if (n <= (1u << 22)) return true;
        if ((threadIdx.x & 31) == 0) atomicExch(err, 2 /* QED2D_ERR_TIMEOUT */);
        return false;
    }
};

// warp-wide: publishes this block's partial of exchange seq to every block of the
// team and returns the team's sum (same additions in the same order in every block)
__device__ __forceinline__ bool team_sum_slots(const TeamComm& C, unsigned seq, double v, double& tot) {
    const int nb = C.nb, lane = threadIdx.x & 31;
    const u64 w = (u64)__double_as_longlong(v);
    const u64 w0 = tag((unsigned)w, seq), w1 = tag((unsigned)(w >> 32), seq);
    bool ok = true;
    double s = 0.0;
    Patience pt;
    const u64 rows = C.psum + (u64)(seq & 1u) * nb * nb * 16;
#pragma unroll 1
    for (int i = lane; i < nb; i += 32) st_slot<false>(rows + ((u64)i * nb + C.rank) * 16, w0, w1);
#pragma unroll 1
    for (int i = 0; i < nb && ok; i += 32) {
        ulonglong2 q;
        for (;;) {
            q = ld_slot<false>(rows + ((u64)C.rank * nb + min(i + lane, nb - 1)) * 16);
            if (__all_sync(0xffffffffu, tagged(q, seq))) break;
            if (!(ok = pt.more(C.err))) break;
        }
        if (i + lane < nb) s += slot_double(q);
    }
    tot = warp_sum(s);
    return ok;
}

// The same in a cluster: every block's partial goes to a slot in every block's
// shared memory.  (Every warp's partial to every block, without the block's own sum
// first, measured slower: 64^2 over 16 blocks 1970 cycles from partial to sum against 1400.)
__device__ __forceinline__ bool cluster_sum_slots(const TeamComm& C, unsigned seq, double v, double& tot) {
    const int nb = C.nb, lane = threadIdx.x & 31;
    const unsigned row = (unsigned)C.psum + 16 * (seq & 1u) * kResCluster;
    const u64 w = (u64)__double_as_longlong(v);
    if (lane < nb) st_slot<true>(map_rank(row + 16 * C.rank, lane), tag((unsigned)w, seq), tag((unsigned)(w >> 32), seq));
    ulonglong2 q;
    Patience pt;
    bool ok = true;
    for (;;) {
        q = ld_slot<true>(row + 16 * min(lane, nb - 1));
        if (__all_sync(0xffffffffu, tagged(q, seq))) break;
        if (!(ok = pt.more(C.err))) break;
    }
    double s = lane < nb ? slot_double(q) : 0.0;
#pragma unroll
    for (int o = kResCluster / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    tot = __shfl_sync(0xffffffffu, s, 0);
    return ok;
}

// The same through one pair of atomic words (large teams over global memory): the
// partial in 80-bit fixed point, 40 bits a word, scaled by a power of two that every
// block derives from an earlier sum, with a count of the blocks in the top byte of
// each word.  Integer additions commute, so the sum does not depend on the order; it
// is exact to 2^-76 of that earlier sum `est` (and repeated through the slots when
// that leaves less than 52 bits of it).  The words only grow (modulo 2^64), two pairs
// in turn, so nothing is cleared; `base` is the pair's value before the exchange.
// A partial out of range (or NaN) is counted in the next byte instead, and then every
// block falls back to team_sum_slots.  Measured with 144 blocks: 1430 cycles an
// exchange, against 2970 through the slots (whose polls grow with the square of the
// team) and 2440 with an arrival counter and partials behind it.
__device__ __forceinline__ bool team_sum_fixed(const TeamComm& C, unsigned seq, double v, double est, ulonglong2& base,
                                               double& tot, bool& exact) {
    const int lane = threadIdx.x & 31;
    u64* acc = C.acc + 16 * (seq & 1u);
    const int ex = min(max((int)((u64)__double_as_longlong(est) >> 52 & 0x7ff) - 1023, -900), 900);
    ulonglong2 d = make_ulonglong2(0, 0);
    int ok = 1;
    if (lane == 0) {
        const double up = __longlong_as_double((long long)(1023 + 36 - ex) << 52);
        const double y = v * up;   // exact
        const bool fits = y < 1099511627776.0;   // 2^40; false for NaN
        const double hi = floor(y);
        const u64 h = fits ? (u64)hi : 1ull << 48, l = fits ? (u64)((y - hi) * 1099511627776.0) : 0ull;
        const u64 one = 1ull << 56;
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(acc), "l"(h + one) : "memory");
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(acc + 1), "l"(l + one) : "memory");
        unsigned n = 0;
        for (;;) {
            const ulonglong2 q = ld_slot<false>((u64)acc);
            d.x = q.x - base.x;
            d.y = q.y - base.y;
            if ((int)(d.x >> 56) == C.nb && (int)(d.y >> 56) == C.nb) {
                base = q;
                break;
            }
            if ((++n & 255u) == 0) {
                if (ld_volatile_int(C.err) != 0) ok = 0;
                else if (n > (1u << 22)) {
                    atomicExch(C.err, 2 /* QED2D_ERR_TIMEOUT */);
                    ok = 0;
                }
                if (!ok) break;
            }
        }
        const double down = __longlong_as_double((long long)(1023 - 36 + ex) << 52);
        tot = ((double)(long long)(d.x & ((1ull << 48) - 1)) +
               (double)(long long)(d.y & ((1ull << 56) - 1)) * 0x1p-40) * down;
        // no block out of range, and 52 bits left of the sum
        exact = ((d.x >> 48) & 0xff) == 0 && tot >= __longlong_as_double((long long)(1023 - 24 + ex) << 52);
    }
    tot = __shfl_sync(0xffffffffu, tot, 0);
    exact = __shfl_sync(0xffffffffu, (int)exact, 0);
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
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
    // where this thread's faces go in the block's inboxes, -1: another block
    int xto;             // the column's (el, er lanes)
    int dto, uto;        // the lower and the upper row's
};

template <class R>
__device__ __forceinline__ V4<R> mk4(R a, R b, R c, R d) { return V4<R>{a, b, c, d}; }
template <class R>
__device__ __forceinline__ V2<R> half1(const V4<R>& s) { return mk(s.x - s.z, s.y - s.w); }
template <class R>
__device__ __forceinline__ V2<R> half2(const V4<R>& s, V2<R> u1) { return cjmul(u1, mk(s.x + s.z, s.y + s.w)); }
template <class R>
__device__ __forceinline__ V2<R> half3(const V4<R>& s) { return mk(s.x - s.w, s.y + s.z); }
template <class R>
__device__ __forceinline__ V2<R> half4(const V4<R>& s, V2<R> u2) { return cjmul(u2, mk(s.x + s.w, s.y - s.z)); }

// The first half of w = g5Dw S: sends the tile's faces, then everything that
// does not come through one.  The links carry the factor -1/2.
template <class R, int K, bool CL>
__device__ __forceinline__ void stencil_inner(const Tile& T, const WarpFace& W, const V4<R> (&S)[K],
                                              const V2<R> (&u1)[K], const V2<R> (&u2)[K], R m2, V2<R>* box,
                                              const TeamComm& C, unsigned seq, V4<R> (&w)[K]) {
    const int lane = threadIdx.x & 31;
    constexpr int E = 16 * Num<R>::SLOTS;   // bytes of a face entry
    V2<R> h1[K], h2[K];
    if (T.h == 0) return;
#pragma unroll
    for (int j = 0; j < K; j++) {
        h1[j] = half1<R>(S[j]);
        h2[j] = half2<R>(S[j], u1[j]);
    }
    const u64 slots = (CL ? 0 : C.slots) + (u64)(seq & 1u) * C.nslots * 16;   // W.to holds addresses in a cluster
    {   // rows
        const V2<R> lo = half3<R>(S[0]);
        if (T.dto >= 0) box[T.dto] = lo;
        else send2<CL>(slots + W.to[2] + E * lane, lo, seq);
        constexpr int J = K > 1 ? K - 2 : 0;   // tiles have K or K - 1 rows (res_plan)
        const bool full = T.h == K;
        const V2<R> h4a = half4<R>(S[K - 1], u2[K - 1]), h4b = half4<R>(S[J], u2[J]);
        const V2<R> hi = mk(full ? h4a.x : h4b.x, full ? h4a.y : h4b.y);
        if (T.uto >= 0) box[T.uto] = hi;
        else send2<CL>(slots + W.to[3] + E * lane, hi, seq);
    }
    if (T.el || T.er) {   // columns
        if (T.xto >= 0) {
#pragma unroll
            for (int j = 0; j < K; j++) box[T.xto + j] = T.el ? h1[j] : h2[j];
        } else {
            const u64 sl = slots + W.to[T.el ? 0 : 1];
#pragma unroll
            for (int j = 0; j < K; j++) send2<CL>(sl + E * j, T.el ? h1[j] : h2[j], seq);
        }
    }
#pragma unroll
    for (int j = 0; j < K; j++) {
        V2<R> fh = mk(__shfl_sync(0xffffffffu, h1[j].x, T.srcR), __shfl_sync(0xffffffffu, h1[j].y, T.srcR));
        V2<R> b1 = mk(__shfl_sync(0xffffffffu, h2[j].x, T.srcL), __shfl_sync(0xffffffffu, h2[j].y, T.srcL));
        if (T.er) fh = mk(R(0), R(0));
        if (T.el) b1 = mk(R(0), R(0));
        const V4<R> s = S[j];
        const V2<R> f1 = cmul(u1[j], fh);
        w[j].x = m2 * s.x + (f1.x + b1.x);
        w[j].y = m2 * s.y + (f1.y + b1.y);
        w[j].z = -m2 * s.z + (f1.x - b1.x);
        w[j].w = -m2 * s.w + (f1.y - b1.y);
    }
#pragma unroll
    for (int j = 0; j + 1 < K; j++)
        if (j + 1 < T.h) {   // the bond between rows j and j + 1
            const V2<R> f2 = cmul(u2[j], half3<R>(S[j + 1])), b2 = half4<R>(S[j], u2[j]);
            w[j].x += f2.x;
            w[j].y += f2.y;
            w[j].z -= f2.y;
            w[j].w += f2.x;
            w[j + 1].x += b2.x;
            w[j + 1].y += b2.y;
            w[j + 1].z += b2.y;
            w[j + 1].w -= b2.x;
        }
}

// The second half: the faces of other tiles.  Those of other blocks are asked for
// first, `meanwhile` runs while the answers are on their way, and what has not
// arrived by then is polled.  False when a wait gave up.
template <class R, int K, bool CL, class F>
__device__ __forceinline__ bool stencil_faces(const Tile& T, const WarpFace& W, const V2<R> (&u1)[K],
                                              const V2<R> (&u2)[K], V2<R>* box, const TeamComm& C, unsigned seq,
                                              V4<R> (&w)[K], F meanwhile) {
    constexpr int BOX = ResSm<R, K>::BOX, E = 16 * Num<R>::SLOTS;
    const int lane = threadIdx.x & 31;
    V2<R>* mine = box + ((threadIdx.x >> 5) - 1) * BOX;
    const u64 slots = C.slots + (u64)(seq & 1u) * C.nslots * 16;
    const bool on = T.h > 0;
    const int side = lane >= K ? 1 : 0;   // the first 2K lanes ask for a row each of the left and right columns
    const bool rx = on && lane < 2 * K && W.warp[side] < 0 && lane - side * K < T.h;
    const bool rd = on && T.dto < 0, ru = on && T.uto < 0;
    Arrival<R> qx, qd, qu;
    auto ask = [&]() {
        if (rd) qd.template ask<CL>(slots + W.from[2] + E * lane);
        if (ru) qu.template ask<CL>(slots + W.from[3] + E * lane);
        if (rx) qx.template ask<CL>(slots + W.from[side] + E * (lane - side * K));
    };
    ask();
    meanwhile();
    if (!on) return true;
    Patience pt;
    bool ok = true;
    for (;;) {
        const bool ready = (!rd || qd.here(seq)) && (!ru || qu.here(seq)) && (!rx || qx.here(seq));
        if (__all_sync(0xffffffffu, ready)) break;
        if (!(ok = pt.more(C.err))) break;
        ask();
    }
    if (rx) mine[lane] = qx.val();
    __syncwarp();
    if (T.el || T.er) {
        const R sg = T.er ? R(1) : R(-1);
#pragma unroll
        for (int j = 0; j < K; j++) {
            if (j == K - 1 && T.h < K) break;   // no such row: its inbox entry is never written
            V2<R> e = mine[(T.er ? K : 0) + j];
            if (T.er) e = cmul(u1[j], e);
            w[j].x += e.x;
            w[j].y += e.y;
            w[j].z += sg * e.x;
            w[j].w += sg * e.y;
        }
    }
    const V2<R> lo = rd ? qd.val() : mine[2 * K + lane], hi = ru ? qu.val() : mine[2 * K + 32 + lane];
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
    return ok;
}

template <class R>
__device__ __forceinline__ R norm4(const V4<R>& a) { return a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w; }
template <class R>
__device__ __forceinline__ V4<R> axpy4(R a, const V4<R>& x, const V4<R>& y) {
    return mk4<R>(y.x + a * x.x, y.y + a * x.y, y.z + a * x.z, y.w + a * x.w);
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
    double part[32 * kResWarps];   // the threads' partials of an exchange
    ResSc sc;
    int abort;                 // a wait of this block gave up
    double next;
    WarpFace face[kResWarps];
    int4 tile[kResWarps];      // first site (x, y), lanes, rows of each warp's tile
    ResRep rep;
    TeamComm C;
};

// The scalar warp (warp 0: the scheduler prefers the oldest of its warps, and this
// one is on the way of all): one step per exchange, in step with the workers.  Returns the
// exchange it ended at.
template <bool MIXED, bool CL, bool MS = false>
__device__ __forceinline__ unsigned res_scalar(const ResP& P, ResBlock& B, unsigned seq, ulonglong2& base0,
                                               ulonglong2& base1, const ResMs* M = nullptr, ResMsBlock* S = nullptr) {
    enum { X_BEGIN, X_GUESS, X_RR, X_PAP, X_FENCE, X_TRUE };   // what the coming exchange sums
    const int nw = MS ? M->nw : (int)(blockDim.x >> 5) - 1, nth = 32 * (nw + 1), lane = threadIdx.x & 31;
    double zs = 1.0, zp = 1.0, a_last = 1.0, b_last = 0.0, a_now = 0.0;   // MS: lane i's shift; the recurrences' scalars
    bool act = MS && lane < M->n && lane != M->base;
    int round = 0;   // MS: barriers with the shift warps so far
    double rr = 0.0, inv_rr = 0.0, maxrr = 0.0, s = 1.0, beta = 0.0, rr64 = 0.0, bb = 0.0, tol = 0.0;
    double rr_last = 1.0, pap_last = 4.0;   // the last |r|^2 and <p, A p>: the fixed-point scales
    double thr = 0.0;                       // |r|^2 below it: reliable update
    int k = 0, nupd = 0, fences = 0, flag = RF_GO, next = X_BEGIN;
    bool conv = false, fresh = true;
#pragma unroll 1
    for (;;) {
        ++seq;
        const bool dead = ld_volatile_int(&B.abort) != 0;   // noted by a worker before the last barrier
        double tot = 0.0;
        bool ok = true;
        bar_sync_n(1, nth);   // the workers' partials are in
        double v = 0.0, v1 = 0.0;
#pragma unroll
        for (int i = 0; i < kResWarps; i++) {
            const double a = i < nw ? B.part[32 * i + lane] : 0.0;
            if (i & 1) v1 += a;
            else v += a;
        }
        v = warp_sum(v + v1);
        if (B.C.nb == 1) {
            tot = v;
        } else if constexpr (CL) {
            ok = cluster_sum_slots(B.C, seq, v, tot);
        } else {
            bool exact = false;
            if (next != X_BEGIN) {
                const double est = next == X_RR ? rr_last : next == X_PAP ? pap_last : next == X_TRUE ? rr64 : 1.0;
                ulonglong2 bs = (seq & 1u) ? base1 : base0;
                ok = team_sum_fixed(B.C, seq, v, est, bs, tot, exact);
                if (seq & 1u) base1 = bs;
                else base0 = bs;
            }
            if (!exact && next != X_FENCE && ok) ok = team_sum_slots(B.C, seq, v, tot);
        }
        double c = 0.0, rr_old = rr;
        const bool all = MS && (next == X_BEGIN || next == X_RR);   // the shift warps join this barrier
        const bool step = MS && next == X_RR && !fresh;             // and an iteration is behind them
        if (next == X_PAP) {   // <p, (A + mu2) p>
            c = rr / tot;   // alpha
            if (MS) a_now = c;
            pap_last = tot;
            k++;
            next = X_RR;
        } else if (next == X_RR) {   // |r|^2
            next = X_PAP;
            rr_last = tot;
            if (fresh) {
                rr = maxrr = tot;
                fresh = false;
            } else if (!MIXED && (tot < tol || k == P.maxiter)) {
                conv = tot < tol;
                rr64 = tot;
                flag = RF_FIN;
                next = X_FENCE;
                fences = 1;
            } else if (MIXED && (tot < thr || k == P.maxiter)) {
                flag = RF_UPD;
                nupd++;
                next = X_FENCE;
                fences = 2;
                rr64 = tot / (s * s);
            } else {
                beta = tot * inv_rr;
                rr = tot;
            }
            c = beta;
        } else if (next == X_FENCE) {   // orders the blocks' FP64 stores
            __threadfence();
            if (flag == RF_FIN) flag = RF_STOP;
            if (--fences == 0) next = X_TRUE;
        } else if (next == X_BEGIN) {   // |b|^2
            bb = rr64 = tot;
            tol = P.eps * bb;
            conv = bb == 0.0;
            if (MIXED && !conv) s = 1.0 / sqrt(bb);
            if (!MIXED) rr_last = bb, pap_last = 4.0 * bb;
            flag = conv ? RF_ZERO : P.guess ? RF_UPD : P.maxiter > 0 ? RF_GO : RF_STOP;
            next = P.guess ? X_FENCE : X_RR;
            fences = 1;
        } else {   // |b - (A + mu2) x|^2
            rr64 = tot;
            conv = tot < tol;
            if (conv || k == P.maxiter) {
                flag = RF_STOP;
            } else if (!MIXED) {   // a warm start
                flag = RF_GO;
                next = X_RR;
                rr_last = tot;
                pap_last = 4.0 * tot;
            } else {
                const double sn = 1.0 / sqrt(tot);
                if (nupd) beta = (tot * s * s * inv_rr) * (sn / s);
                s = sn;
                fresh = true;
                flag = RF_GO;
                next = X_RR;
                rr_last = 1.0;
                pap_last = 4.0;
            }
        }
        if (!ok || dead) flag = RF_ABORT;
        if (lane == 0) {
            if (MIXED) B.sc.cf = (float)c;
            else B.sc.c = c;
            B.sc.flag = flag;
            B.sc.s = s;
        }
        if (all) bar_sync_n(5, blockDim.x);
        else bar_sync_n(3, nth);
        if constexpr (MS) {
            const bool give_up = !all && flag == RF_ABORT && next == X_RR;   // in <p, A p>: the shift warps wait for |r|^2
            if (step) {   // the shifts' recurrences (k_cg_multishift's), lane i shift i
                const double b_new = tot / rr_old;
                if (act) {
                    const double zn = zs * zp * a_last / (a_now * b_last * (zp - zs) + zp * a_last * (1.0 + M->d[lane] * a_now));
                    const double q = zn / zs;
                    S->a[lane] = a_now * q;
                    S->b[lane] = b_new * q * q;
                    S->z[lane] = zn;
                    zp = zs;
                    zs = zn;
                    act = !(zn * zn * tot < tol);
                    S->state[lane] = act ? 2 : 1;
                } else {
                    S->state[lane] = 0;
                }
                a_last = a_now;
                b_last = b_new;
            }
            if (give_up) bar_arrive_n(5, blockDim.x);
            if (all || give_up) {
                if (lane == 0) S->flag[round & 1] = flag;
                round++;
                bar_arrive_n(4, blockDim.x - 32 * nw);
            }
        }
        if (flag >= RF_STOP) break;
        // off the way from one exchange to the next
        inv_rr = 1.0 / rr;
        maxrr = fmax(maxrr, rr);
        thr = fmax(P.delta2 * maxrr, tol * s * s);
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
// workers: the thread's partial of exchange seq
__device__ __forceinline__ void put_part(ResBlock& B, double s) {
    B.part[threadIdx.x - 32] = s;
    bar_arrive_n(1, B.nwk + 32);
}
// Workers: the end of an exchange.  A warp whose wait for a face gave up (!ok)
// leaves a note that the scalar warp finds at the next exchange and turns into
// RF_ABORT for the whole block, so that all its threads leave at the same barrier.
__device__ __forceinline__ int wait_scalar(ResBlock& B, bool ok, bool all = false) {
    if (!ok) *(volatile int*)&B.abort = 1;
    if (all) bar_sync_n(5, blockDim.x);   // MS: with the shift warps
    else bar_sync_n(3, B.nwk + 32);
    return *(volatile int*)&B.sc.flag;
}

// Workers: the FP64 true residual b - (A + mu2) x, after x += x32 / s (add), and,
// where the solve goes on, the FP32 residual for the next iteration, left in x32
// (the caller takes it and clears x32).  The stencils read other blocks' x and
// t64, so an exchange follows each of them.  Runs a few times per solve, with
// the iteration's registers put away in shared memory (t) or read again (links).
template <bool MIXED>
__device__ __forceinline__ int res_update(const ResP& P, ResBlock& B, float4* x32, unsigned& seq, bool add) {
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
        put_part(B, 0.0);
        ++seq;
        if (wait_scalar(B, true) == RF_ABORT) return RF_ABORT;
    }
#pragma unroll 1
    for (int j = 0; j < c.h; j++) {
        const Site q = col_site(c, L1, L2, j);
        st_d(t64, V, q.x, g5dw_at<double>(SpDcg{xs, V}, L, q, m2));
    }
    __threadfence();
    __syncwarp();
    put_part(B, 0.0);
    ++seq;
    if (wait_scalar(B, true) == RF_ABORT) return RF_ABORT;
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
    put_part(B, n);
    ++seq;
    const int flag = wait_scalar(B, true);
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
__device__ __forceinline__ int res_begin(const ResP& P, ResBlock& B, float4* x32, unsigned& seq) {
    const Column c = column_of(B);
    const int nwk = B.nwk, L1 = B.rep.L1;
    const long long V = (long long)L1 * B.rep.L2, o2 = 2 * B.rep.off;
    double acc = 0.0;
#pragma unroll 1
    for (int j = 0; j < c.h; j++) {
        const long long g = o2 + c.g0 + (long long)j * L1;
        acc += norm2(__ldg(P.b + g)) + norm2(__ldg(P.b + V + g));
    }
    put_part(B, acc);
    ++seq;
    const int flag = wait_scalar(B, true, MS);
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
__device__ __forceinline__ void res_finish(const ResP& P, ResBlock& B, const double4x* xs, unsigned& seq) {
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
    put_part(B, 0.0);
    ++seq;
    if (wait_scalar(B, true) == RF_ABORT || !P.want_g5) return;
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

template <class R, int K, bool CL, bool MS = false>
__device__ __forceinline__ unsigned res_worker(const ResP& P, ResBlock& B, char* dyn, unsigned seq,
                                               V4<R>* rbuf = nullptr) {   // MS: r for the shift warps, two copies in turn
    constexpr bool MIXED = std::is_same<R, float>::value;
    const int nwk = B.nwk, lane = threadIdx.x & 31;
    V4<R>* xs = reinterpret_cast<V4<R>*>(dyn) + (threadIdx.x - 32);   // x: row j at xs[j * nwk]
    V4<R>* ps = xs + K * nwk;                                         // the search direction likewise
    V4<R>* ts = ps + K * nwk;                                         // mixed: t during an update
    V2<R>* box = reinterpret_cast<V2<R>*>(dyn + (size_t)nwk * ResSm<R, K>::ARRAYS * K * sizeof(V4<R>));
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
        constexpr int BOX = ResSm<R, K>::BOX;
        const WarpFace& F = B.face[(threadIdx.x >> 5) - 1];
        T.xto = F.warp[T.el ? 0 : 1] < 0 ? -1 : F.warp[T.el ? 0 : 1] * BOX + (T.el ? K : 0);
        T.dto = F.warp[2] < 0 ? -1 : F.warp[2] * BOX + 2 * K + 32 + lane;
        T.uto = F.warp[3] < 0 ? -1 : F.warp[3] * BOX + 2 * K + lane;
    }
    const WarpFace& W = B.face[(threadIdx.x >> 5) - 1];
    const V4<R> zero = mk4<R>(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < K; j++) {
        xs[j * nwk] = ps[j * nwk] = zero;
        if (MIXED) ts[j * nwk] = zero;
    }
    int flag = res_begin<MIXED, MS>(P, B, reinterpret_cast<float4*>(xs), seq);
    bool first = true;
    V2<R> u1[K], u2[K];
    V4<R> r[K], t[K], w[K];
    R alpha = 0;
    const R m2 = (R)B.rep.m2, mu2 = (R)P.mu2;
    for (;;) {
        const double2* src = P.b;
        if (flag != RF_GO) {
            if (flag != RF_UPD) return seq;
            flag = res_update<MIXED>(P, B, reinterpret_cast<float4*>(xs), seq, !first);
            if (flag != RF_GO) return seq;
            src = P.r64;
        }
        first = false;
        const Column c = column_of(B);
#pragma unroll
        for (int j = 0; j < K; j++) {
            u1[j] = u2[j] = mk(R(0), R(0));
            w[j] = zero;
            if constexpr (MIXED) {
                t[j] = ts[j * nwk];
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
        for (;;) {
            {
                R f = 0;
#pragma unroll
                for (int j = 0; j < K; j++) f += norm4<R>(r[j]);
                put_part(B, (double)f);
                ++seq;
            }
            stencil_inner<R, K, CL>(T, W, r, u1, u2, m2, box, B.C, seq, w);
            bar_sync_n(2, nwk);
            bool ok = stencil_faces<R, K, CL>(T, W, u1, u2, box, B.C, seq, w, [&]() {   // x += alpha p of the last iteration
#pragma unroll
                for (int j = 0; j < K; j++) xs[j * nwk] = axpy4<R>(alpha, ps[j * nwk], xs[j * nwk]);
            });
            flag = wait_scalar(B, ok, MS);
            if (flag != RF_GO) break;
            const R beta = MIXED ? (R)B.sc.cf : (R)B.sc.c;
            {
                R f = 0;
#pragma unroll
                for (int j = 0; j < K; j++) {
                    t[j] = axpy4<R>(beta, t[j], w[j]);
                    f += norm4<R>(t[j]);
                }
                double d = (double)f;
                if (mu2 != R(0)) {   // with a shift <p, A p> needs p now, else it is formed during the exchange
                    f = 0;
#pragma unroll
                    for (int j = 0; j < K; j++) {
                        const V4<R> pn = axpy4<R>(beta, ps[j * nwk], r[j]);
                        ps[j * nwk] = pn;
                        f += norm4<R>(pn);
                    }
                    d += P.mu2 * (double)f;
                }
                put_part(B, d);
                ++seq;
            }
            stencil_inner<R, K, CL>(T, W, t, u1, u2, m2, box, B.C, seq, w);
            bar_sync_n(2, nwk);
            ok = stencil_faces<R, K, CL>(T, W, u1, u2, box, B.C, seq, w, [&]() {
                if (mu2 == R(0))
#pragma unroll
                    for (int j = 0; j < K; j++) ps[j * nwk] = axpy4<R>(beta, ps[j * nwk], r[j]);
            });
            if (wait_scalar(B, ok) == RF_ABORT) {
                if (MS) bar_arrive_n(5, blockDim.x);   // the shift warps wait there
                return seq;
            }
            alpha = MIXED ? (R)B.sc.cf : (R)B.sc.c;
#pragma unroll
            for (int j = 0; j < K; j++) {
                if (mu2 != R(0)) w[j] = axpy4<R>(mu2, ps[j * nwk], w[j]);
                r[j] = axpy4<R>(-alpha, w[j], r[j]);
                if constexpr (MS) rbuf[(((seq >> 1) & 1) * K + j) * nwk + threadIdx.x - 32] = r[j];
            }
        }
        alpha = 0;
        if constexpr (MIXED) {
#pragma unroll
            for (int j = 0; j < K; j++) ts[j * nwk] = t[j];
        } else {
            if (flag == RF_FIN) res_finish(P, B, xs, seq);
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
        B.C.err = &P.ctl->err;
        if constexpr (CL) {
            B.C.psum = smem_u32(dyn + ResSm<R, K>::bytes((blockDim.x >> 5) - 1));
            B.C.slots = B.C.psum + 2 * kResCluster * 16;
        } else {
            B.C.slots = (u64)(P.slots + (size_t)team * P.nb * 2 * P.nslots);
            B.C.psum = (u64)(P.psum + (size_t)team * 2 * P.nb * P.nb);
            B.C.acc = P.acc + 32 * team;
        }
    }
    if constexpr (CL) {   // no slot carries a tag yet
        ulonglong2* sl = reinterpret_cast<ulonglong2*>(dyn + ResSm<R, K>::bytes((blockDim.x >> 5) - 1));
        for (int i = threadIdx.x; i < 2 * (kResCluster + P.nslots); i += blockDim.x) sl[i] = make_ulonglong2(0, 0);
        cooperative_groups::this_cluster().sync();
    }
    unsigned seq = 0;
    ulonglong2 base0 = make_ulonglong2(0, 0), base1 = base0;
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
        if (B.sc.flag == RF_ABORT) break;
        ++seq;   // the team's first block takes the next system for the team
        if (threadIdx.x < 32) {
            int n = 0;
            if (B.C.rank == 0 && threadIdx.x == 0) n = atomicAdd(P.queue, 1);
            double tot = (double)__shfl_sync(0xffffffffu, n, 0);
            if (P.nb > 1 && !team_sum_slots(B.C, seq, tot, tot)) tot = (double)P.nrep;
            if (threadIdx.x == 0) B.next = tot;
        }
        __syncthreads();
        next = P.nteams + (int)B.next;
    }
    if (B.C.rank == 0 && threadIdx.x == 0 && ld_volatile_int(B.C.err) != 0)
        atomicCAS(&P.ctl->status, 0, QED2D_ERR_TIMEOUT);
    if constexpr (CL) cooperative_groups::this_cluster().sync();   // others may still write here
}

// ---------------------------------------------------------------------------
// host side
inline int res_slots(const ResPlan& p, int per) { return per * (2 * p.wy * p.K + 2 * p.wx * 32); }   // of one buffer of a block

template <class R, int K>
static size_t res_smem(const ResPlan& p) {
    return ResSm<R, K>::bytes(p.wx * p.wy) +
           (p.cl ? sizeof(ulonglong2) * 2 * (kResCluster + res_slots(p, Num<R>::SLOTS)) : 0);
}

template <class R, int K>
static int res_clusters_k(const ResPlan& plan) {
    const void* kern = (const void*)k_res_cg<R, K, true>;
    const size_t sm = res_smem<R, K>(plan);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(plan.blocks());
    cfg.blockDim = dim3(32 * (plan.wx * plan.wy + 1));
    cfg.dynamicSmemBytes = sm;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = plan.blocks();
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
static int res_launch_k(const ResP& P, const ResPlan& plan, cudaStream_t stream) {
    const void* kern = (const void*)k_res_cg<R, K, CL>;
    const size_t sm = res_smem<R, K>(plan);
    QCHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    if (CL) QCHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(P.nb * P.nteams);
    cfg.blockDim = dim3(32 * (plan.wx * plan.wy + 1));
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
