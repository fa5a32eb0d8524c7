// Level sweep of the transient forward solve, in state-major layout.
//
// Replaces the transient half of solver::solve_nonterminal_part
// (cuda/src/solver.cu:205-300) and its block-triangular solve
// (cuda/src/linear_system_solve.cu:249-325, 492-626) for the forward form: the expected
// occupation z of the transient states solves (Q - A) z = x0, and terminal SCC t
// receives y_t = x0(t) + sum over edges u -> v, u transient, v in t, of rate * z_u.
// That is L x0 of the reference without forming L.
//
// The transient block is lower triangular in the topological order of the condensation:
// an SCC receives flow only from SCCs of higher level and never from another SCC of its
// own level.  Level groups are solved one after another, sources first, and inside a
// group every SCC is an independent diagonal block.  Per group:
//   - singleton SCCs only: z_v = b_v / q_v;
//   - otherwise BiCGStab on the odd-parity Schur complement.  Every edge flips one bit, so
//     the graph is bipartite by popcount parity and the even rows are eliminated exactly.
//     The right preconditioner is the Schur diagonal.  Where an SCC is solved depends on its
//     larger parity and the number of systems K:
//       up to kSccMaxRows rows: one CTA per (SCC, few systems), vectors on chip (k_sw_scc);
//       up to kSccMaxCluster times as many: a cluster per (SCC, system) for K >=
//       kSccClusterMin, else the group is one block of a cooperative grid (kSccGrid);
//       beyond: the cooperative grid for K <= 32; for more systems the row kernels, one
//       launch per step, SCC by SCC, and the group's other SCCs and singletons as above.
//     k_sw_scc is FP64 throughout; the row kernels' inner iterations are FP64
//     (ESL_METHOD_DIRECT) or FP32 (ESL_METHOD_MIXED) inside FP64 iterative refinement on
//     the true residual.
//
// Layout: every vector is [row][system], the Kp (K rounded up to 32) systems of a row
// contiguous.  A warp handles 32 systems of one state, so every neighbour gather reads a
// contiguous run of 32 values however scattered the group's states are among the 2^n.
// Rows are "slots": the transient states numbered group by group, even-parity states of
// a group first, then odd.  The row structure (state, out-mask, predecessor lists) is
// read once per row and shared by every system.  Rates are staged per CTA in shared
// memory as [rate index][system lane].
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <type_traits>
#include <vector>

#include <cub/device/device_scan.cuh>
#include <nvtx3/nvToolsExt.h>

#include "esl_internal.h"
#include "scc_plan.h"

namespace esl {
namespace {

constexpr int kSwT = 256;            // threads per row kernel
constexpr int kSwLocalMax = 512;     // largest SCC of a kind-1 group
constexpr int kSwPoll = 4;           // Krylov iterations launched between convergence polls
// Poll windows in flight: the host reads the running count of window c - (depth - 1)
// after queueing window c, so a late host leaves the GPU idle only after it has fallen
// depth - 1 windows behind.  Windows queued past convergence cost little (tiles whose
// systems have stopped exit at once).
constexpr int kSwPollDepth = 3;
static_assert(kSwPollDepth >= 2 && kSwPollDepth <= 4, "the context holds four poll events and count slots");
constexpr double kSwAcceptRel = 1e-8;  // stagnating systems are accepted at this relative residual
constexpr int kSwStall = 30;         // inner iterations without halving the residual before an inner solve stops
// The same for the FP64 inner solves of grid-wide groups.  BiCGStab's residual there has
// plateaus of up to ~90 iterations that end by themselves, and a restart discards the
// Krylov space: on the largest group of the n=20 network, 30 cost three refinement rounds
// and 376 iterations, 100 two rounds and 220 (512 rate sets, FP64 replica on the host).
constexpr int kSwStall64 = 100;

// per-system flags
constexpr int SW_DONE = 1;   // group solve finished for this system
constexpr int SW_FAIL = 2;   // finished without meeting the acceptance residual
constexpr int SW_RUN = 4;    // runs an inner solve in this refinement step
constexpr int SW_IDONE = 8;  // its inner solve has stopped

// per-system scalar arrays (doubles), each Kp long
// C_GAM0..2: the deflation scalar gamma(x) of the operator applications of the true
// residual, of v = A p and of t = A s (deflated groups only); C_D0..2 take the
// accumulations of the undeflated products there, which nothing reads.
enum Scal { C_BB, C_RR64, C_PREV, C_RHO, C_R0V, C_TS, C_TT, C_RR, C_RN, C_BETA, C_OMEGA, C_TARGET, C_BEST, C_SCALE,
            C_R0T, C_GAM0, C_GAM1, C_GAM2, C_D0, C_D1, C_D2, C_NSCAL };
// per-system int arrays
enum IScal { I_FLAGS, I_ITERS, I_NOIMP, I_TOTAL, I_STALL, I_NISCAL };

struct SwGroup {
    uint32_t beg, ne, no;  // first slot, even rows, odd rows
    uint32_t ob;           // first odd slot (beg + ne, except in a piece of a group)
    int kind;              // 0 singletons, 1 SCCs of at most kSwLocalMax states, 2 larger ones (their
                           // odd rows are the learned warm start's targets)
    int max_scc;
    uint64_t nin;          // in-group predecessor entries of the group's rows
    uint32_t s0, ns;       // the group's SCCs of >= 2 states: range in SweepPlan::scc
    uint32_t sh0, nsh;     // their shapes: range in SweepPlan::shapes
    uint32_t l0, nlarge;   // those beyond a cluster (the first ones): range in SweepPlan::large
    uint32_t most;         // most rows of one parity of an SCC (0: singletons only)
    bool resident;         // every one of them fits a CTA or a cluster of k_sw_scc
    bool split;            // one of them needs a cluster
    uint32_t singles;      // rows that are SCCs of their own
    int term;              // terminal plan: the terminal SCC of the group (-1 otherwise)
    uint32_t pos0;         // terminal plan: position of the SCC's first state in the order
};

struct SweepPlan {
    uint32_t M = 0, max_rows = 0, max_even = 0, max_odd = 0;
    int TS = 0;
    std::vector<SwGroup> groups;
    DevBuf<uint2> rows;                  // per slot: (state, out-mask)
    DevBuf<uint4> desc;                  // per slot: (state, out-mask, first in-group entry, count)
    DevBuf<uint32_t> ig_ptr, ig_ent;     // predecessors inside the group: slot << 6 | rate index
    DevBuf<uint32_t> og_ptr, og_ent;     // predecessors in earlier groups
    DevBuf<uint32_t> tp_ptr, tp_ent;     // transient predecessors of terminal position p
    // SCCs of >= 2 states in the order of scc_sort_key: (first even slot, even rows, first odd
    // slot, odd rows); an SCC's even and odd slots are one run each.  The host keeps their
    // shapes, and the places of those beyond a cluster: a network may have millions of SCCs.
    DevBuf<uint4> scc;
    DevBuf<uint64_t> scc_key;  // (while the plan is built)
    std::vector<SccShape> shapes;
    std::vector<uint4> large;
    // Predecessors of the rows of SCCs solved by one CTA (k_sw_scc), by slices of 32 rows of
    // one parity: scc_sl = an SCC's first even and first odd slice, sl = a slice's (lines,
    // first line of ell).  Line j holds entries 4j .. 4j + 3 of 32 rows, 16 bytes a row; a narrow
    // SCC's (scc_narrow) are as wide as the parity has rows and sl holds their place in ell,
    // behind those of the others.  An entry is the
    // local row of the other parity << 9 | rate index << 3, so that masked and shifted they
    // are byte offsets (row * 8 after >> 6); past a row's last entry the local row is the
    // other parity's row count.  In an SCC split over a cluster the local row is the owner's
    // rank << 13 | its row there, and past the last entry the own rank's row kSccMaxRows.
    DevBuf<uint2> scc_sl, sl;
    DevBuf<uint4> ell;
    // terminal plan: per slot, the state's position in the reordering
    DevBuf<uint32_t> pos;
    // backward plan of the whole transient part: per slot, the in-mask among transient states
    DevBuf<uint32_t> rev;
    // the terminal SCCs above kDenseTerminalMax states, one deflated grid group each
    // (slots of their own; in-group predecessor lists only), or null
    SweepPlan* term = nullptr;
    SweepPlan() = default;
    SweepPlan(const SweepPlan&) = delete;
    SweepPlan& operator=(const SweepPlan&) = delete;
    ~SweepPlan() { delete term; }
};

void free_plan_sweep(void* p) { delete static_cast<SweepPlan*>(p); }

struct SwArgs {
    int n, K, Kp, nrhs, KT;
    const double* rateT;     // [2n][Kp], rateT[j * Kp + k] = rate j of system k (0 past K)
    const uint2* rows;
    const uint4* desc;       // per slot: (state, out-mask, first in-group entry, in-group count)
    const uint32_t* ig_ptr;
    const uint32_t* ig_ent;
    // rows: ne even ones from slot beg, no odd ones from slot ob
    uint32_t beg, ob, ne, no;
    const int* flags;        // per-system flags or null
    // FP64 out-rate sums of the group's rows, [row][Kp], or null (then recomputed from
    // the out-masks): q of the odd rows and 1 / q of the even rows
    const double* Qo;
    const double* IQe;
    // Deflated groups (a terminal SCC): per-system accumulator of gamma(x) = sum of the
    // odd-row vector plus sum of its even-row elimination, or null; u_o = q_o * inv_s.
    double* gam;
    double inv_s;
};

// slot of row r of a group (even rows first)
__device__ __forceinline__ uint32_t sw_slot(const SwArgs& a, uint32_t r) { return r < a.ne ? a.beg + r : a.ob + (r - a.ne); }

// A tile is KT systems of one row handled by TR = KT / S threads, S systems per thread:
// thread `lane` of the row owns the adjacent systems k = lane * S, ..., k + S - 1 of the
// tile, so that its S values of a row are one vector load.  TR >= 32, so the 32 lanes of
// a warp always share one row.
struct Tile {
    int lane, rsub, RB, KT, TR, k;
};

template <int S = 1>
__device__ __forceinline__ Tile tile_of(int KT) {
    Tile t;
    t.KT = KT;
    t.TR = KT / S;
    t.RB = blockDim.x / t.TR;
    t.lane = threadIdx.x % t.TR;
    t.rsub = threadIdx.x / t.TR;
    t.k = blockIdx.y * KT + t.lane * S;
    return t;
}

// S adjacent values of a row (8- or 4-byte elements), one vector load when S == 2
template <int S, class TX>
__device__ __forceinline__ void load_s(const TX* __restrict__ p, TX (&v)[S]) {
    if constexpr (S == 2 && sizeof(TX) == 8) {
        const double2 w = *reinterpret_cast<const double2*>(p);
        v[0] = (TX)w.x;
        v[1] = (TX)w.y;
    } else if constexpr (S == 2 && sizeof(TX) == 4) {
        const float2 w = *reinterpret_cast<const float2*>(p);
        v[0] = (TX)w.x;
        v[1] = (TX)w.y;
    } else {
#pragma unroll
        for (int q = 0; q < S; q++) v[q] = p[q];
    }
}

template <class T>
__device__ __forceinline__ void sw_rates(T* s, const SwArgs& a, const Tile& t) {
    const int k0 = blockIdx.y * t.KT;
    const int tot = 2 * a.n * t.KT;
    for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
        const int j = idx / t.KT, l = idx - j * t.KT;
        s[idx] = (T)a.rateT[(size_t)j * a.Kp + k0 + l];
    }
    __syncthreads();
}

// out-rates of state v (out-mask f) for this thread's S systems
template <int S, class T>
__device__ __forceinline__ void sw_qs(const T* s, uint32_t v, uint32_t f, const Tile& t, T (&q)[S]) {
#pragma unroll
    for (int j = 0; j < S; j++) q[j] = 0;
    while (f) {
        const int i = __ffs(f) - 1;
        f &= f - 1;
        const T* r = s + (2 * i + ((v >> i) & 1u)) * t.KT + t.lane * S;
#pragma unroll
        for (int j = 0; j < S; j++) q[j] += r[j];
    }
}

template <class T>
__device__ __forceinline__ T sw_q(const T* s, uint32_t v, uint32_t f, const Tile& t) {
    T q[1];
    sw_qs<1>(s, v, f, t, q);
    return q[0];
}

// Predecessor entries are (slot << 6) | rate index, the rate index of the edge being
// 2i + b for a flip of bit i out of a source whose bit i is b (rates are
// [up_0, down_0, up_1, ...]).
constexpr int kEntShift = 6;
__device__ __forceinline__ uint32_t ent_slot(uint32_t e) { return e >> kEntShift; }
__device__ __forceinline__ int ent_rate(uint32_t e) { return (int)(e & 63u); }

__device__ __forceinline__ bool sw_skip(const SwArgs& a, int k) {
    if (k >= a.K) return true;
    if (!a.flags) return false;
    const int f = a.flags[k];
    return !(f & SW_RUN) || (f & SW_IDONE);
}

// acc[j] += sum over the predecessor entries ent[p0 .. p0 + cnt) of a row of
// rate(entry) * X[ent_slot(entry) - base][system j], in entry order.  With MASK false,
// systems with act[j] == false accumulate whatever their rows hold (their acc must then
// be left unused by the caller); with MASK true they add zero.  All 32 lanes of a
// warp handle the same row, so the row's entries (at most n <= 26) arrive in one
// coalesced load and are broadcast by shuffles, and the gathers are issued four entries
// at a time.  Every lane of the warp must call it; systems with act[j] == false load
// nothing.
template <int S, class TC, class TX, bool MASK = true>
__device__ __forceinline__ void sw_gathers_m(const TC* s, const Tile& t, int Kp, uint32_t mine, int cnt,
                                             const TX* __restrict__ X, uint32_t base, const bool (&act)[S],
                                             TC (&acc)[S]) {
    const TX* Xk = X + t.k;
    const TC* sk = s + t.lane * S;
    bool any = false;
#pragma unroll
    for (int q = 0; q < S; q++) any |= act[q];
    // a thread loads its S adjacent values of a row together (inactive ones are read and
    // then ignored: they share the load)
    int j = 0;
    for (; j + 4 <= cnt; j += 4) {
        uint32_t e[4];
        TX x[4][S];
#pragma unroll
        for (int u = 0; u < 4; u++) e[u] = __shfl_sync(0xffffffffu, mine, j + u);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const TX* row = Xk + (size_t)(ent_slot(e[u]) - base) * Kp;
            if (any) {
                load_s<S, TX>(row, x[u]);
            } else {
#pragma unroll
                for (int q = 0; q < S; q++) x[u][q] = (TX)0;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            TC r[S];
            load_s<S, TC>(sk + ent_rate(e[u]) * t.KT, r);
#pragma unroll
            for (int q = 0; q < S; q++) acc[q] += r[q] * ((!MASK || act[q]) ? (TC)x[u][q] : (TC)0);
        }
    }
    for (; j < cnt; j++) {
        const uint32_t e = __shfl_sync(0xffffffffu, mine, j);
        const TX* row = Xk + (size_t)(ent_slot(e) - base) * Kp;
        TX x[S];
        if (any) {
            load_s<S, TX>(row, x);
        } else {
#pragma unroll
            for (int q = 0; q < S; q++) x[q] = (TX)0;
        }
        TC r[S];
        load_s<S, TC>(sk + ent_rate(e) * t.KT, r);
#pragma unroll
        for (int q = 0; q < S; q++) acc[q] += r[q] * ((!MASK || act[q]) ? (TC)x[q] : (TC)0);
    }
}

template <int S, class TC, class TX, bool MASK = true>
__device__ __forceinline__ void sw_gathers(const TC* s, const Tile& t, int Kp, const uint32_t* __restrict__ ent,
                                           uint32_t p0, int cnt, const TX* __restrict__ X, uint32_t base,
                                           const bool (&act)[S], TC (&acc)[S]) {
    const int lane = threadIdx.x & 31;
    const uint32_t mine = lane < cnt ? __ldg(ent + p0 + lane) : 0u;
    sw_gathers_m<S, TC, TX, MASK>(s, t, Kp, mine, cnt, X, base, act, acc);
}

template <class TC, class TX>
__device__ __forceinline__ TC sw_gather(const TC* s, const Tile& t, int Kp, const uint32_t* __restrict__ ent,
                                        uint32_t p0, int cnt, const TX* __restrict__ X, uint32_t base, bool act,
                                        TC acc) {
    const bool a1[1] = {act};
    TC c1[1] = {acc};
    sw_gathers<1, TC, TX>(s, t, Kp, ent, p0, cnt, X, base, a1, c1);
    return c1[0];
}

// Block-wide sums of NV per-thread values for each of this thread's S systems, added
// atomically to dst[v][system] by the first row of the CTA.
template <int NV, int S = 1>
__device__ __forceinline__ void sw_reduce(const double (&v)[NV][S], double* const (&dst)[NV], const Tile& t, int K) {
    __shared__ double red[NV * S * kSwT];
#pragma unroll
    for (int j = 0; j < NV; j++)
#pragma unroll
        for (int q = 0; q < S; q++) red[(j * S + q) * kSwT + threadIdx.x] = v[j][q];
    __syncthreads();
    if (t.rsub == 0) {
#pragma unroll
        for (int j = 0; j < NV; j++)
#pragma unroll
            for (int q = 0; q < S; q++) {
                const int k = t.k + q;
                if (k >= K) continue;
                double acc = 0.0;
                for (int r = 0; r < t.RB; r++) acc += red[(j * S + q) * kSwT + r * t.TR + t.lane];
                if (acc != 0.0) atomicAdd(dst[j] + k, acc);
            }
    }
}

// ---- right-hand sides -------------------------------------------------------------------
// b_v = x0(v) + inflow from transient states of earlier groups, for every row of the
// group; DIRECT groups store z_v = b_v / q_v in Z, others b into the group buffer Bv.
template <bool DIRECT>
__global__ void __launch_bounds__(kSwT) k_sw_rhs(SwArgs a, const uint32_t* __restrict__ og_ptr,
                                                 const uint32_t* __restrict__ og_ent, const double* __restrict__ x0,
                                                 size_t x0_ld, double* __restrict__ Z, double* __restrict__ Bv) {
    extern __shared__ double s_rate[];
    const Tile t = tile_of(a.KT);
    sw_rates(s_rate, a, t);
    const bool act = t.k < a.K;
    if (__all_sync(0xffffffffu, !act)) return;
    const uint32_t cnt = a.ne + a.no;
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < cnt; r += gridDim.x * t.RB) {
        const uint32_t slot = sw_slot(a, r);
        const uint2 row = a.rows[slot];
        const uint32_t v = row.x;
        const uint32_t p0 = og_ptr[slot];
        double acc = act ? x0[(size_t)(t.k % a.nrhs) * x0_ld + v] : 0.0;
        acc = sw_gather<double, double>(s_rate, t, a.Kp, og_ent, p0, (int)(og_ptr[slot + 1] - p0), Z, 0u, act, acc);
        if (!act) continue;
        if (DIRECT)
            Z[(size_t)slot * a.Kp + t.k] = acc / sw_q(s_rate, v, row.y, t);
        else
            Bv[(size_t)r * a.Kp + t.k] = acc;
    }
}

// Schur diagonal on the odd rows: dS_o = q_o - sum over in-group e with e -> o and o -> e
// of rate(e -> o) rate(o -> e) / q_e.
__global__ void __launch_bounds__(kSwT) k_sw_diag(SwArgs a, double* __restrict__ dS64, float* __restrict__ dS32) {
    extern __shared__ double s_rate[];
    const Tile t = tile_of(a.KT);
    sw_rates(s_rate, a, t);
    if (t.k >= a.K) return;
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
        const uint32_t slot = a.ob + r;
        const uint2 row = a.rows[slot];
        const uint32_t o = row.x;
        double d = sw_q(s_rate, o, row.y, t);
        for (uint32_t e = a.ig_ptr[slot]; e < a.ig_ptr[slot + 1]; e++) {
            const uint32_t ent = a.ig_ent[e];
            const int ri = ent_rate(ent);
            if (!((row.y >> (ri >> 1)) & 1u)) continue;  // no edge o -> e
            const uint2 re = a.rows[ent_slot(ent)];
            // rate(e -> o) is the entry's; rate(o -> e) flips the same bit the other way
            d -= s_rate[ri * t.KT + t.lane] * s_rate[(ri ^ 1) * t.KT + t.lane] / sw_q(s_rate, re.x, re.y, t);
        }
        dS64[(size_t)r * a.Kp + t.k] = d;
        if (dS32) dS32[(size_t)r * a.Kp + t.k] = (float)d;
    }
}

// Out-rate sums of a grid group's rows, once per group: Qo = q of the odd rows, IQe =
// 1 / q of the even rows, so that the operator kernels read one value per row and system
// instead of summing the rates of the out-mask.
__global__ void __launch_bounds__(kSwT) k_sw_qrows(SwArgs a, double* __restrict__ Qo, double* __restrict__ IQe) {
    extern __shared__ double s_rate[];
    const Tile t = tile_of(a.KT);
    sw_rates(s_rate, a, t);
    if (t.k >= a.K) return;
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.ne + a.no; r += gridDim.x * t.RB) {
        const uint2 row = a.rows[sw_slot(a, r)];
        const double q = sw_q(s_rate, row.x, row.y, t);
        if (r < a.ne)
            IQe[(size_t)r * a.Kp + t.k] = 1.0 / q;
        else
            Qo[(size_t)(r - a.ne) * a.Kp + t.k] = q;
    }
}

// Even-row elimination: W_e = (C_e + sum over in-group odd predecessors o of
// rate(o -> e) X_o) / q_e.  C (FP64, even rows of the group buffer) and X may be null.
// S systems per thread.
// DEFL: also adds the sum of the written W over the even rows into a.gam (FP64, the
// deflated operator of a terminal SCC).
template <int S, class TX, class TW, class TC, bool DEFL = false>
__global__ void __launch_bounds__(kSwT) k_sw_elim(SwArgs a, const double* __restrict__ C, const TX* __restrict__ X,
                                                  TW* __restrict__ W) {
    extern __shared__ unsigned char s_raw[];
    TC* s_rate = reinterpret_cast<TC*>(s_raw);
    const Tile t = tile_of<S>(a.KT);
    sw_rates(s_rate, a, t);
    bool act[S];
    bool any = false;
    double wsum[S];
#pragma unroll
    for (int q = 0; q < S; q++) {
        act[q] = !sw_skip(a, t.k + q);
        any |= act[q];
        wsum[q] = 0.0;
    }
    // the gathers shuffle across the warp: a warp runs the row loop if any lane is active
    const bool wany = __any_sync(0xffffffffu, any);
    if (!DEFL && !wany) return;
    const uint32_t obase = a.ob;
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < (wany ? a.ne : 0u); r += gridDim.x * t.RB) {
        // (state, out-mask, first entry, count) in one load
        const uint4 d = a.desc[a.beg + r];
        const size_t idx = (size_t)r * a.Kp + t.k;
        TC acc[S];
#pragma unroll
        for (int q = 0; q < S; q++) acc[q] = (C && act[q]) ? (TC)C[idx + q] : (TC)0;
        // acc of an inactive system is never stored: no masking in the gathers
        if (X) sw_gathers<S, TC, TX, false>(s_rate, t, a.Kp, a.ig_ent, d.z, (int)d.w, X, obase, act, acc);
        if (sizeof(TC) == 8 && a.IQe) {
#pragma unroll
            for (int q = 0; q < S; q++)
                if (act[q]) {
                    const TW w = (TW)(acc[q] * (TC)__ldcs(a.IQe + idx + q));
                    W[idx + q] = w;
                    if (DEFL) wsum[q] += (double)w;
                }
        } else {
            TC qv[S];
            sw_qs<S>(s_rate, d.x, d.y, t, qv);
#pragma unroll
            for (int q = 0; q < S; q++)
                if (act[q]) {
                    const TW w = (TW)(acc[q] / qv[q]);
                    W[idx + q] = w;
                    if (DEFL) wsum[q] += (double)w;
                }
        }
    }
    if (DEFL) {
        double v[1][S];
#pragma unroll
        for (int q = 0; q < S; q++) v[0][q] = wsum[q];
        double* const dst[1] = {a.gam};
        sw_reduce<1, S>(v, dst, t, a.K);
    }
}

// Odd-row operator.  y = q X - sum over in-group even predecessors e of rate(e -> o) W_e.
//   MODE 0: Y = B + sum(rate W)          (reduced rhs, FP64), acc0 += Y^2
//   MODE 1: Y = B - y                    (true residual, FP64), acc0 += Y^2
//   MODE 2: Y = y                        acc0 += AUX . Y   (AUX = r0)
//   MODE 3: Y = y                        acc0 += Y . (AUX X), acc1 += Y . Y   (AUX = dS)
//   MODE 4: (no output)                  acc0 += y . B, acc1 += y . y   (B = reduced rhs)
//   MODE 6: as MODE 3, and acc2 += R0x . Y (so that the next beta is known before the
//           x / r update: beta = -(r0 . t) / (r0 . v))
// S systems per thread.  X, AUX and Y are streamed (evict-first) so that the gathered W
// keeps its place in L2.
// DEFL (MODE 1, 2 and 6): also adds the sum of X over the odd rows into a.gam; Y is
// then the undeflated product, which k_sw_defl_fin completes.
template <int S, int MODE, class T, bool DEFL = false>
__global__ void __launch_bounds__(kSwT) k_sw_apply(SwArgs a, const T* __restrict__ X, const T* __restrict__ W,
                                                   const double* __restrict__ B, const T* __restrict__ AUX,
                                                   T* __restrict__ Y, double* acc0, double* acc1,
                                                   const T* __restrict__ R0x, double* acc2) {
    extern __shared__ unsigned char s_raw[];
    T* s_rate = reinterpret_cast<T*>(s_raw);
    const Tile t = tile_of<S>(a.KT);
    sw_rates(s_rate, a, t);
    double d0[S], d1[S], d2[S], dg[S];
    bool act[S];
    bool any = false;
#pragma unroll
    for (int q = 0; q < S; q++) {
        d0[q] = d1[q] = d2[q] = dg[q] = 0.0;
        const int k = t.k + q;
        act[q] = !((MODE >= 2) ? sw_skip(a, k) : (k >= a.K));
        any |= act[q];
    }
    if (__any_sync(0xffffffffu, any)) {
        for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
            const uint4 d = a.desc[a.ob + r];  // (state, out-mask, first entry, count)
            const size_t idx = (size_t)r * a.Kp + t.k;
            T flow[S];
#pragma unroll
            for (int q = 0; q < S; q++) flow[q] = 0;
            sw_gathers<S, T, T, false>(s_rate, t, a.Kp, a.ig_ent, d.z, (int)d.w, W, a.beg, act, flow);
            T qv[S];
            if (MODE != 0) {
                if (sizeof(T) == 8 && a.Qo) {
#pragma unroll
                    for (int q = 0; q < S; q++) qv[q] = act[q] ? (T)__ldcs(a.Qo + idx + q) : (T)0;
                } else {
                    sw_qs<S>(s_rate, d.x, d.y, t, qv);
                }
            }
#pragma unroll
            for (int q = 0; q < S; q++) {
                if (!act[q]) continue;
                const size_t i = idx + q;
                if (MODE == 0) {
                    const double y = B[i] + (double)flow[q];
                    Y[i] = (T)y;
                    d0[q] += y * y;
                } else {
                    const T x = __ldcs(X + i);
                    if (DEFL) dg[q] += (double)x;
                    const T y = qv[q] * x - flow[q];
                    if (MODE == 1) {
                        const double res = B[i] - (double)y;
                        Y[i] = (T)res;
                        d0[q] += res * res;
                    } else if (MODE == 2) {
                        __stcs(Y + i, y);
                        d0[q] += (double)__ldcs(AUX + i) * (double)y;
                    } else if (MODE == 4) {
                        d0[q] += (double)y * B[i];
                        d1[q] += (double)y * (double)y;
                    } else {
                        __stcs(Y + i, y);
                        d0[q] += (double)y * ((double)__ldcs(AUX + i) * (double)x);
                        d1[q] += (double)y * (double)y;
                        if (MODE == 6) d2[q] += (double)__ldcs(R0x + i) * (double)y;
                    }
                }
            }
        }
    }
    if (DEFL && MODE == 6) {
        double v[4][S];
#pragma unroll
        for (int q = 0; q < S; q++) {
            v[0][q] = d0[q];
            v[1][q] = d1[q];
            v[2][q] = d2[q];
            v[3][q] = dg[q];
        }
        double* const dst[4] = {acc0, acc1, acc2, a.gam};
        sw_reduce<4, S>(v, dst, t, a.K);
    } else if (DEFL) {
        double v[2][S];
#pragma unroll
        for (int q = 0; q < S; q++) {
            v[0][q] = d0[q];
            v[1][q] = dg[q];
        }
        double* const dst[2] = {acc0, a.gam};
        sw_reduce<2, S>(v, dst, t, a.K);
    } else if (MODE == 6) {
        double v[3][S];
#pragma unroll
        for (int q = 0; q < S; q++) {
            v[0][q] = d0[q];
            v[1][q] = d1[q];
            v[2][q] = d2[q];
        }
        double* const dst[3] = {acc0, acc1, acc2};
        sw_reduce<3, S>(v, dst, t, a.K);
    } else if (MODE == 3 || MODE == 4) {
        double v[2][S];
#pragma unroll
        for (int q = 0; q < S; q++) {
            v[0][q] = d0[q];
            v[1][q] = d1[q];
        }
        double* const dst[2] = {acc0, acc1};
        sw_reduce<2, S>(v, dst, t, a.K);
    } else {
        double v[1][S];
#pragma unroll
        for (int q = 0; q < S; q++) v[0][q] = d0[q];
        double* const dst[1] = {acc0};
        sw_reduce<1, S>(v, dst, t, a.K);
    }
}

// ---- paired-row Schur operator for 32-system tiles ---------------------------------------
// The largest level groups run 32-system tiles (their gathered slice must stay in L2), and
// with one system per lane a warp spends ~13 instructions per system and predecessor entry
// on the entry shuffle, the address, the load, the rate look-up and the select.  Here a
// half warp serves one row and each lane two adjacent systems, so a warp runs two rows at
// once and every instruction of the gather loop serves four (row, system) pairs: the
// row value and the rate are 16-byte loads.  The two rows' entry counts differ; the loop
// runs to the larger count and the other half's gathers are predicated off.  FP64, no
// deflation, out-rate sums from SwArgs::Qo / IQe.  Tile layout: KT = 32, S = 2, TR = 16
// (tile_of<2>(32): rsub = threadIdx.x / 16, lane = threadIdx.x % 16).

// Entries past a row's count are padded with a dummy entry, (base << 6) | 2n: gathered
// row 0 (always in range) times rate row 2n, a row of zeros the kernels append to the
// rate table.  So the gather loop needs no predicates; a padded term adds 0 * x.

// acc[q] += sum over the entries of this half warp's row (m0: lane l16 holds entry l16,
// m1: entry 16 + l16, both padded) of rate(entry) * X[entry row] for this lane's two
// systems; cmax = the larger count of the warp's two rows (warp-uniform).  O32: the
// gathered vector's element offsets fit in 32 bits.  The sums of inactive systems take
// whatever their rows hold and are never stored.
template <bool O32>
__device__ __forceinline__ void pr_gathers(const double* s_rate, const Tile& t, int Kp, uint32_t m0, uint32_t m1,
                                           int cmax, const double* __restrict__ X, uint32_t base,
                                           double (&acc)[2]) {
    const double* Xk = X + t.k;
    const double* sk = s_rate + t.lane * 2;
    auto term = [&](uint32_t e) {
        const uint32_t row = ent_slot(e) - base;
        const double* xp = O32 ? Xk + row * (uint32_t)Kp : Xk + (size_t)row * Kp;
        const double2 x = *reinterpret_cast<const double2*>(xp);
        const double2 r = *reinterpret_cast<const double2*>(sk + ent_rate(e) * 32);
        acc[0] += r.x * x.x;
        acc[1] += r.y * x.y;
    };
    const int c16 = min(cmax, 16);
    int j = 0;
    // two entries per step: measured faster than four (fewer registers, more warps)
    for (; j + 2 <= c16; j += 2) {
        uint32_t e[2];
#pragma unroll
        for (int u = 0; u < 2; u++) e[u] = __shfl_sync(0xffffffffu, m0, j + u, 16);
#pragma unroll
        for (int u = 0; u < 2; u++) term(e[u]);
    }
    for (; j < c16; j++) term(__shfl_sync(0xffffffffu, m0, j, 16));
    for (j = 16; j < cmax; j++) term(__shfl_sync(0xffffffffu, m1, j - 16, 16));
}

// this half warp's row r: its padded entries 0..15 (m0) and 16..31 (m1), and the larger
// entry count of the warp's two rows
struct PrRow {
    uint32_t m0, m1;
    int cnt, cmax;
};
__device__ __forceinline__ PrRow pr_row(const SwArgs& a, uint32_t rowbase, uint32_t r, uint32_t count,
                                        uint32_t dummy) {
    PrRow p;
    const uint32_t l16 = threadIdx.x & 15;
    uint2 zw = make_uint2(0u, 0u);
    if (r < count) zw = __ldg(reinterpret_cast<const uint2*>(a.desc + rowbase + r) + 1);
    p.cnt = (int)zw.y;
    p.m0 = l16 < zw.y ? __ldg(a.ig_ent + zw.x + l16) : dummy;
    p.m1 = l16 + 16 < zw.y ? __ldg(a.ig_ent + zw.x + 16 + l16) : dummy;
    p.cmax = max(p.cnt, __shfl_xor_sync(0xffffffffu, p.cnt, 16));
    return p;
}

// rate table of a paired-row kernel: sw_rates plus the zero row 2n of padded entries
__device__ __forceinline__ void pr_rates(double* s_rate, const SwArgs& a, const Tile& t) {
    if (threadIdx.x < 32) s_rate[2 * a.n * 32 + threadIdx.x] = 0.0;
    sw_rates(s_rate, a, t);
}

// Paired-row k_sw_elim: W_e = (sum rate X) / q_e over the group's even rows.
// 8 CTAs per SM (32 registers, a few bytes of spill): measured faster than 6 CTAs
// without spill
template <bool O32>
__global__ void __launch_bounds__(kSwT, 8) k_sw_elim_pr(SwArgs a, const double* __restrict__ X,
                                                     double* __restrict__ W) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    double* s_rate = reinterpret_cast<double*>(s_raw);
    const Tile t = tile_of<2>(32);
    pr_rates(s_rate, a, t);
    bool act[2];
    act[0] = !sw_skip(a, t.k);
    act[1] = !sw_skip(a, t.k + 1);
    const bool any = act[0] || act[1];
    if (!__any_sync(0xffffffffu, any)) return;
    const uint32_t count = a.ne, rs = gridDim.x * t.RB, obase = a.ob;
    // the warp's two rows are rw and rw + 1; the loop condition is warp-uniform
    for (uint32_t rw = blockIdx.x * t.RB + (t.rsub & ~1); rw < count; rw += rs) {
        const uint32_t r = rw + (t.rsub & 1);
        const PrRow p = pr_row(a, a.beg, r, count, (obase << kEntShift) | (uint32_t)(2 * a.n));
        double acc[2] = {0.0, 0.0};
        pr_gathers<O32>(s_rate, t, a.Kp, p.m0, p.m1, p.cmax, X, obase, acc);
        if (r < count) {
            const size_t idx = (size_t)r * a.Kp + t.k;
            const double2 iq = __ldcs(reinterpret_cast<const double2*>(a.IQe + idx));
            if (act[0]) W[idx] = acc[0] * iq.x;
            if (act[1]) W[idx + 1] = acc[1] * iq.y;
        }
    }
}

// Paired-row k_sw_apply, MODE 2 (Y = y, acc0 += AUX . Y, AUX = r0) and MODE 6 (Y = y,
// acc0 += Y . (AUX X), AUX = dS, acc1 += Y . Y, acc2 += R0x . Y); q_o from Qo.
template <int MODE, bool O32>
__global__ void __launch_bounds__(kSwT) k_sw_apply_pr(SwArgs a, const double* __restrict__ X,
                                                      const double* __restrict__ W, const double* __restrict__ AUX,
                                                      double* __restrict__ Y, double* acc0, double* acc1,
                                                      const double* __restrict__ R0x, double* acc2) {
    static_assert(MODE == 2 || MODE == 6, "paired-row apply: MODE 2 or 6");
    extern __shared__ __align__(16) unsigned char s_raw[];
    double* s_rate = reinterpret_cast<double*>(s_raw);
    const Tile t = tile_of<2>(32);
    pr_rates(s_rate, a, t);
    double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0}, d2[2] = {0.0, 0.0};
    bool act[2];
    act[0] = !sw_skip(a, t.k);
    act[1] = !sw_skip(a, t.k + 1);
    const bool any = act[0] || act[1];
    if (__any_sync(0xffffffffu, any)) {
        const uint32_t count = a.no, rs = gridDim.x * t.RB, rowbase = a.ob;
        for (uint32_t rw = blockIdx.x * t.RB + (t.rsub & ~1); rw < count; rw += rs) {
            const uint32_t r = rw + (t.rsub & 1);
            const PrRow p = pr_row(a, rowbase, r, count, (a.beg << kEntShift) | (uint32_t)(2 * a.n));
            double flow[2] = {0.0, 0.0};
            pr_gathers<O32>(s_rate, t, a.Kp, p.m0, p.m1, p.cmax, W, a.beg, flow);
            if (r >= count) continue;
            const size_t i = (size_t)r * a.Kp + t.k;
            const double2 qv = __ldcs(reinterpret_cast<const double2*>(a.Qo + i));
            const double2 x = __ldcs(reinterpret_cast<const double2*>(X + i));
            const double2 aux = __ldcs(reinterpret_cast<const double2*>(AUX + i));
            const double y0 = qv.x * x.x - flow[0], y1 = qv.y * x.y - flow[1];
            if (MODE == 2) {
                if (act[0]) {
                    __stcs(Y + i, y0);
                    d0[0] += aux.x * y0;
                }
                if (act[1]) {
                    __stcs(Y + i + 1, y1);
                    d0[1] += aux.y * y1;
                }
            } else {
                const double2 r0 = __ldcs(reinterpret_cast<const double2*>(R0x + i));
                if (act[0]) {
                    __stcs(Y + i, y0);
                    d0[0] += y0 * (aux.x * x.x);
                    d1[0] += y0 * y0;
                    d2[0] += r0.x * y0;
                }
                if (act[1]) {
                    __stcs(Y + i + 1, y1);
                    d0[1] += y1 * (aux.y * x.y);
                    d1[1] += y1 * y1;
                    d2[1] += r0.y * y1;
                }
            }
        }
    }
    if (MODE == 6) {
        double v[3][2] = {{d0[0], d0[1]}, {d1[0], d1[1]}, {d2[0], d2[1]}};
        double* const dst[3] = {acc0, acc1, acc2};
        sw_reduce<3, 2>(v, dst, t, a.K);
    } else {
        double v[1][2] = {{d0[0], d0[1]}};
        double* const dst[1] = {acc0};
        sw_reduce<1, 2>(v, dst, t, a.K);
    }
}

// ---- deflated operator of a terminal SCC -------------------------------------------------
// For a terminal SCC C the stationary vector solves (-K_C + u 1^T) pi = u, whose only
// solution is the normalised kernel of K_C whenever 1^T u != 0 (1^T K_C = 0), and whose
// matrix keeps every eigenvalue of -K_C except 0, which moves to 1^T u.  With u zero on
// the even rows the even rows still eliminate exactly, and on the odd rows the system
// becomes S x + u gamma(x) = u with gamma(x) = 1^T x + 1^T W(x), W the even-row
// elimination.  Here u_o = q_o / s (s = states of the SCC), so 1^T u is about the mean
// out-rate.  k_sw_elim / k_sw_apply<DEFL> accumulate gamma; this kernel adds gamma u to
// the product (MODE 2, 6) or subtracts it from the residual (MODE 1) and forms the
// products of that MODE (see k_sw_apply) on the completed vector.
template <int MODE>
__global__ void __launch_bounds__(kSwT) k_sw_defl_fin(SwArgs a, double* __restrict__ Y, const double* __restrict__ X,
                                                      const double* __restrict__ AUX, const double* __restrict__ R0x,
                                                      const double* __restrict__ gam, double* acc0, double* acc1,
                                                      double* acc2) {
    const Tile t = tile_of(a.KT);
    const bool act = MODE == 1 ? t.k < a.K : !sw_skip(a, t.k);
    double d0 = 0.0, d1 = 0.0, d2 = 0.0;
    if (act) {
        const double g = gam[t.k];
        for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
            const size_t i = (size_t)r * a.Kp + t.k;
            const double u = a.Qo[i] * a.inv_s;
            if (MODE == 1) {
                const double y = Y[i] - g * u;
                Y[i] = y;
                d0 += y * y;
            } else {
                const double y = Y[i] + g * u;
                Y[i] = y;
                if (MODE == 2) {
                    d0 += AUX[i] * y;
                } else {
                    d0 += y * (AUX[i] * X[i]);
                    d1 += y * y;
                    d2 += R0x[i] * y;
                }
            }
        }
    }
    if (MODE == 6) {
        double v[3][1] = {{d0}, {d1}, {d2}};
        double* const dst[3] = {acc0, acc1, acc2};
        sw_reduce<3>(v, dst, t, a.K);
    } else {
        double v[1][1] = {{d0}};
        double* const dst[1] = {acc0};
        sw_reduce<1>(v, dst, t, a.K);
    }
}

// Right-hand side of a deflated group in the group buffer: 0 on the even rows, u_o =
// q_o / s on the odd rows.
__global__ void __launch_bounds__(kSwT) k_sw_defl_rhs(SwArgs a, double* __restrict__ Bv) {
    extern __shared__ double s_rate[];
    const Tile t = tile_of(a.KT);
    sw_rates(s_rate, a, t);
    if (t.k >= a.K) return;
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.ne + a.no; r += gridDim.x * t.RB) {
        const uint2 row = a.rows[sw_slot(a, r)];
        Bv[(size_t)r * a.Kp + t.k] = r < a.ne ? 0.0 : sw_q(s_rate, row.x, row.y, t) * a.inv_s;
    }
}

// Terminal kernel of a deflated group into Rb[k][position]: the group's slots (both
// parities, solved in Z) at their positions in the reordering, and their sum per system.
__global__ void __launch_bounds__(kSwT) k_sw_term_out(SwArgs a, const uint32_t* __restrict__ pos,
                                                      const double* __restrict__ Z, int TS, double* __restrict__ Rb,
                                                      double* sums) {
    const Tile t = tile_of(a.KT);
    double d = 0.0;
    if (t.k < a.K) {
        for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.ne + a.no; r += gridDim.x * t.RB) {
            const uint32_t slot = sw_slot(a, r);
            const double v = Z[(size_t)slot * a.Kp + t.k];
            Rb[(size_t)t.k * TS + pos[slot]] = v;
            d += v;
        }
    }
    double v[1][1] = {{d}};
    double* const dst[1] = {sums};
    sw_reduce<1>(v, dst, t, a.K);
}

// Rb[k][p0 .. p0 + count) /= sums[k]
__global__ void k_sw_term_norm(int K, int TS, uint32_t p0, uint32_t count, const double* __restrict__ sums,
                               double* __restrict__ Rb) {
    const int k = blockIdx.y;
    if (k >= K) return;
    const double inv = sums[k] != 0.0 ? 1.0 / sums[k] : 0.0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
        Rb[(size_t)k * TS + p0 + i] *= inv;
}

// ---- compaction of running systems --------------------------------------------------------
// A system tile runs until its slowest system stops, so once the running systems fit in
// fewer tiles they are moved to the leading columns of every per-system array (a
// physical permutation of each row's system run, so that the kernels keep their
// coalesced [row][system] access) and the grid shrinks.  cperm maps the compacted
// column to the original system; the inverse permutation restores every array before
// the inner solve's result is committed.
constexpr int kCompactMaxKp = 1024;  // a row's systems are permuted in shared memory
constexpr int kPermWarps = 4;

__device__ __forceinline__ bool sw_running(int f) { return (f & SW_RUN) && !(f & SW_IDONE); }

__global__ void k_sw_iota(int n, int* __restrict__ p) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) p[k] = k;
}

// Stable partition of the columns [0, Kc): running systems first.  p2[new] = old column;
// cperm[new] = cperm[old].  One CTA.
__global__ void __launch_bounds__(1024) k_sw_perm_build(int Kc, const int* __restrict__ flags, int* __restrict__ cperm,
                                                        int* __restrict__ p2) {
    __shared__ int s_run[kCompactMaxKp / 32 + 1], s_stop[kCompactMaxKp / 32 + 1];
    __shared__ int s_old[kCompactMaxKp];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int nch = (Kc + 31) / 32;
    for (int k = threadIdx.x; k < Kc; k += blockDim.x) s_old[k] = cperm[k];
    for (int c = warp; c < nch; c += nw) {
        const int k = c * 32 + lane;
        const bool valid = k < Kc;
        const bool run = valid && sw_running(flags[k]);
        const unsigned m = __ballot_sync(0xFFFFFFFFu, run), v = __ballot_sync(0xFFFFFFFFu, valid);
        if (lane == 0) {
            s_run[c] = __popc(m);
            s_stop[c] = __popc(v & ~m);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int ra = 0, sa = 0;
        for (int c = 0; c < nch; c++) {
            const int r = s_run[c], q = s_stop[c];
            s_run[c] = ra;
            s_stop[c] = sa;
            ra += r;
            sa += q;
        }
        s_run[nch] = ra;
    }
    __syncthreads();
    const int total = s_run[nch];
    for (int c = warp; c < nch; c += nw) {
        const int k = c * 32 + lane;
        const bool valid = k < Kc;
        const bool run = valid && sw_running(flags[k]);
        const unsigned m = __ballot_sync(0xFFFFFFFFu, run), v = __ballot_sync(0xFFFFFFFFu, valid);
        const unsigned lt = (1u << lane) - 1u;
        if (valid) {
            const int pos = run ? s_run[c] + __popc(m & lt) : total + s_stop[c] + __popc(v & ~m & lt);
            p2[pos] = k;
            cperm[pos] = s_old[k];
        }
    }
}

struct PermArr {
    void* p;
    uint32_t rows;
    int esize;  // 4 or 8 bytes
};
struct PermList {
    PermArr a[16];
};

// Array blockIdx.y, each of its rows (stride Kp): forward row[k] = row_old[p[k]], inverse
// row[p[k]] = row_old[k], for k < Kc.  One warp per row, the row staged in shared memory.
__global__ void __launch_bounds__(kPermWarps * 32) k_sw_row_perm(PermList L, int Kp, int Kc, const int* __restrict__ p,
                                                                 int inverse) {
    extern __shared__ double s_rowbuf[];
    const PermArr A = L.a[blockIdx.y];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* sm = s_rowbuf + (size_t)warp * Kc;
    for (uint32_t r = blockIdx.x * kPermWarps + warp; r < A.rows; r += gridDim.x * kPermWarps) {
        if (A.esize == 8) {
            double* row = static_cast<double*>(A.p) + (size_t)r * Kp;
            for (int k = lane; k < Kc; k += 32) sm[k] = row[k];
            __syncwarp();
            for (int k = lane; k < Kc; k += 32) {
                if (inverse)
                    row[p[k]] = sm[k];
                else
                    row[k] = sm[p[k]];
            }
        } else {
            float* row = static_cast<float*>(A.p) + (size_t)r * Kp;
            float* sf = reinterpret_cast<float*>(sm);
            for (int k = lane; k < Kc; k += 32) sf[k] = row[k];
            __syncwarp();
            for (int k = lane; k < Kc; k += 32) {
                if (inverse)
                    row[p[k]] = sf[k];
                else
                    row[k] = sf[p[k]];
            }
        }
        __syncwarp();
    }
}

// ---- BiCGStab vector steps (odd rows; scalars per system) --------------------------------
struct SwScalPtr {
    double* c[C_NSCAL];
    int* i[I_NISCAL];
};

template <class T>
__global__ void __launch_bounds__(kSwT) k_sw_s(SwArgs a, SwScalPtr sc, const T* __restrict__ R, const T* __restrict__ V,
                                               const T* __restrict__ dS, T* __restrict__ SH) {
    const Tile t = tile_of(a.KT);
    if (sw_skip(a, t.k)) return;
    const double r0v = sc.c[C_R0V][t.k];
    const T alpha = r0v != 0.0 ? (T)(sc.c[C_RHO][t.k] / r0v) : (T)0;
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
        const size_t idx = (size_t)r * a.Kp + t.k;
        SH[idx] = (R[idx] - alpha * V[idx]) / dS[idx];
    }
}

// x / r update fused with the next search direction.  With alpha = rho / (r0 . v),
// omega = (t . s) / (t . t) and, from r0 . s = 0, beta = -(r0 . t) / (r0 . v):
//   D += alpha PH + omega SH,  R = s - omega t,  PH = (R + beta (dS PH - omega V)) / dS.
// A system that stops at this iteration gets a direction it never uses.
template <class T>
__global__ void __launch_bounds__(kSwT) k_sw_xrp(SwArgs a, SwScalPtr sc, T* __restrict__ PH,
                                                 const T* __restrict__ SH, const T* __restrict__ dS,
                                                 const T* __restrict__ TT, const T* __restrict__ R0,
                                                 const T* __restrict__ V, T* __restrict__ D, T* __restrict__ R) {
    const Tile t = tile_of(a.KT);
    double d0 = 0.0, d1 = 0.0;
    if (!sw_skip(a, t.k)) {
        const double r0v = sc.c[C_R0V][t.k], tt = sc.c[C_TT][t.k];
        const T alpha = r0v != 0.0 ? (T)(sc.c[C_RHO][t.k] / r0v) : (T)0;
        const T omega = tt > 0.0 ? (T)(sc.c[C_TS][t.k] / tt) : (T)0;
        const T beta = r0v != 0.0 ? (T)(-sc.c[C_R0T][t.k] / r0v) : (T)0;
        for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
            const size_t idx = (size_t)r * a.Kp + t.k;
            const T sh = __ldcs(SH + idx), ph = PH[idx], d = __ldcs(dS + idx);
            __stcs(D + idx, __ldcs(D + idx) + alpha * ph + omega * sh);
            const T rn = d * sh - omega * __ldcs(TT + idx);
            __stcs(R + idx, rn);
            PH[idx] = (rn + beta * (d * ph - omega * __ldcs(V + idx))) / d;
            d0 += (double)rn * (double)rn;
            d1 += (double)__ldcs(R0 + idx) * (double)rn;
        }
    }
    double v[2][1] = {{d0}, {d1}};
    double* const dst[2] = {sc.c[C_RR], sc.c[C_RN]};
    sw_reduce<2>(v, dst, t, a.K);
}

// k_sw_s and k_sw_xrp for FP64 with two adjacent systems per thread (tile_of<2>: 16-byte
// loads and stores, half the instructions per value; any KT >= 32).  Stores are made for
// running systems only, as in the one-system kernels.
__device__ __forceinline__ void st2(double* p, double v0, double v1, bool a0, bool a1) {
    if (a0 && a1) {
        __stcs(reinterpret_cast<double2*>(p), make_double2(v0, v1));
    } else {
        if (a0) p[0] = v0;
        if (a1) p[1] = v1;
    }
}

__global__ void __launch_bounds__(kSwT) k_sw_s2(SwArgs a, SwScalPtr sc, const double* __restrict__ R,
                                                const double* __restrict__ V, const double* __restrict__ dS,
                                                double* __restrict__ SH) {
    const Tile t = tile_of<2>(a.KT);
    const bool a0 = !sw_skip(a, t.k), a1 = !sw_skip(a, t.k + 1);
    if (!a0 && !a1) return;
    double al[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int k = min(t.k + q, a.Kp - 1);
        const double r0v = sc.c[C_R0V][k];
        al[q] = r0v != 0.0 ? sc.c[C_RHO][k] / r0v : 0.0;
    }
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
        const size_t idx = (size_t)r * a.Kp + t.k;
        const double2 rv = __ldcs(reinterpret_cast<const double2*>(R + idx));
        const double2 vv = __ldcs(reinterpret_cast<const double2*>(V + idx));
        const double2 dv = __ldcs(reinterpret_cast<const double2*>(dS + idx));
        st2(SH + idx, (rv.x - al[0] * vv.x) / dv.x, (rv.y - al[1] * vv.y) / dv.y, a0, a1);
    }
}

__global__ void __launch_bounds__(kSwT) k_sw_xrp2(SwArgs a, SwScalPtr sc, double* __restrict__ PH,
                                                  const double* __restrict__ SH, const double* __restrict__ dS,
                                                  const double* __restrict__ TT, const double* __restrict__ R0,
                                                  const double* __restrict__ V, double* __restrict__ D,
                                                  double* __restrict__ R) {
    const Tile t = tile_of<2>(a.KT);
    const bool a0 = !sw_skip(a, t.k), a1 = !sw_skip(a, t.k + 1);
    double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
    if (a0 || a1) {
        double al[2], om[2], be[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int k = min(t.k + q, a.Kp - 1);
            const double r0v = sc.c[C_R0V][k], tt = sc.c[C_TT][k];
            al[q] = r0v != 0.0 ? sc.c[C_RHO][k] / r0v : 0.0;
            om[q] = tt > 0.0 ? sc.c[C_TS][k] / tt : 0.0;
            be[q] = r0v != 0.0 ? -sc.c[C_R0T][k] / r0v : 0.0;
        }
        for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
            const size_t idx = (size_t)r * a.Kp + t.k;
            const double2 sh = __ldcs(reinterpret_cast<const double2*>(SH + idx));
            const double2 ph = *reinterpret_cast<const double2*>(PH + idx);
            const double2 d = __ldcs(reinterpret_cast<const double2*>(dS + idx));
            const double2 dd = __ldcs(reinterpret_cast<const double2*>(D + idx));
            const double2 tv = __ldcs(reinterpret_cast<const double2*>(TT + idx));
            const double2 vv = __ldcs(reinterpret_cast<const double2*>(V + idx));
            const double2 r0 = __ldcs(reinterpret_cast<const double2*>(R0 + idx));
            st2(D + idx, dd.x + al[0] * ph.x + om[0] * sh.x, dd.y + al[1] * ph.y + om[1] * sh.y, a0, a1);
            const double rn0 = d.x * sh.x - om[0] * tv.x, rn1 = d.y * sh.y - om[1] * tv.y;
            st2(R + idx, rn0, rn1, a0, a1);
            const double p0 = (rn0 + be[0] * (d.x * ph.x - om[0] * vv.x)) / d.x;
            const double p1 = (rn1 + be[1] * (d.y * ph.y - om[1] * vv.y)) / d.y;
            if (a0 && a1) {
                *reinterpret_cast<double2*>(PH + idx) = make_double2(p0, p1);
            } else {
                if (a0) PH[idx] = p0;
                if (a1) PH[idx + 1] = p1;
            }
            if (a0) {
                d0[0] += rn0 * rn0;
                d1[0] += r0.x * rn0;
            }
            if (a1) {
                d0[1] += rn1 * rn1;
                d1[1] += r0.y * rn1;
            }
        }
    }
    double v[2][2] = {{d0[0], d0[1]}, {d1[0], d1[1]}};
    double* const dst[2] = {sc.c[C_RR], sc.c[C_RN]};
    sw_reduce<2, 2>(v, dst, t, a.K);
}

// Scalar step after each iteration; one CTA; writes the number of running systems.
__global__ void k_sw_scal(int K, SwScalPtr sc, int max_iters, int stall_max, int* active) {
    __shared__ int s_cnt;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    int cnt = 0;
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        int f = sc.i[I_FLAGS][k];
        if (!(f & SW_RUN) || (f & SW_IDONE)) continue;
        const int it = ++sc.i[I_ITERS][k];
        sc.i[I_TOTAL][k]++;
        const double rho = sc.c[C_RHO][k], r0v = sc.c[C_R0V][k], ts = sc.c[C_TS][k], tt = sc.c[C_TT][k];
        const double rr = sc.c[C_RR][k], rn = sc.c[C_RN][k];
        const double alpha = r0v != 0.0 ? rho / r0v : 0.0;
        const double omega = tt > 0.0 ? ts / tt : 0.0;
        if (rr < 0.5 * sc.c[C_BEST][k]) {
            sc.c[C_BEST][k] = rr;
            sc.i[I_STALL][k] = 0;
        } else {
            sc.i[I_STALL][k]++;
        }
        const bool stop = !(rr > sc.c[C_TARGET][k]) || it >= max_iters || r0v == 0.0 || omega == 0.0 ||
                          rn == 0.0 || !isfinite(rr) || !isfinite(alpha) || sc.i[I_STALL][k] >= stall_max;
        if (stop) {
            sc.i[I_FLAGS][k] = f | SW_IDONE;
        } else {
            sc.c[C_BETA][k] = (rn / rho) * (alpha / omega);
            sc.c[C_OMEGA][k] = omega;
            sc.c[C_RHO][k] = rn;
            cnt++;
        }
        sc.c[C_R0V][k] = sc.c[C_TS][k] = sc.c[C_TT][k] = sc.c[C_RR][k] = sc.c[C_RN][k] = sc.c[C_R0T][k] = 0.0;
        sc.c[C_GAM1][k] = sc.c[C_GAM2][k] = 0.0;
    }
    atomicAdd(&s_cnt, cnt);
    __syncthreads();
    if (threadIdx.x == 0) *active = s_cnt;
}

// Decide, per system, whether another refinement step runs; writes the count.
__global__ void k_sw_outer(int K, SwScalPtr sc, double tol2, double inner_rel2, double accept2, int outer,
                           int max_refine, int* active) {
    __shared__ int s_cnt;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    int cnt = 0;
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        int f = sc.i[I_FLAGS][k];
        if (f & SW_DONE) continue;
        const double rr = sc.c[C_RR64][k], b2 = sc.c[C_BB][k];
        if (!(b2 > 0.0) || rr <= tol2 * b2) {
            sc.i[I_FLAGS][k] = SW_DONE;
            continue;
        }
        if (outer > 0 && !(rr < 0.25 * sc.c[C_PREV][k])) sc.i[I_NOIMP][k]++;
        // A system whose refinement stagnates has reached what FP64 delivers for it and
        // is accepted within the acceptance residual; one that runs out of refinement
        // steps while still improving has missed its budget and goes to the fallback.
        if (sc.i[I_NOIMP][k] >= 2 || !isfinite(rr)) {
            sc.i[I_FLAGS][k] = (rr <= accept2 * b2) ? SW_DONE : (SW_DONE | SW_FAIL);
            continue;
        }
        if (outer >= max_refine) {
            sc.i[I_FLAGS][k] = SW_DONE | SW_FAIL;
            continue;
        }
        // the inner solve works on the residual scaled to unit norm
        const double scale = 1.0 / sqrt(rr);
        sc.i[I_FLAGS][k] = SW_RUN;
        sc.i[I_ITERS][k] = 0;
        sc.c[C_PREV][k] = rr;
        sc.c[C_SCALE][k] = scale;
        sc.c[C_RHO][k] = 1.0;
        sc.c[C_BETA][k] = 0.0;
        sc.c[C_OMEGA][k] = 1.0;
        sc.c[C_TARGET][k] = fmax(inner_rel2, 0.01 * tol2 * b2 * scale * scale);
        sc.c[C_BEST][k] = 1.0;
        sc.i[I_STALL][k] = 0;
        sc.c[C_R0V][k] = sc.c[C_TS][k] = sc.c[C_TT][k] = sc.c[C_RR][k] = sc.c[C_RN][k] = sc.c[C_R0T][k] = 0.0;
        sc.c[C_GAM1][k] = sc.c[C_GAM2][k] = 0.0;
        cnt++;
    }
    atomicAdd(&s_cnt, cnt);
    __syncthreads();
    if (threadIdx.x == 0) *active = s_cnt;
}

// start of an inner solve: R = R0 = (T) (R64 * scale), PH = R / dS (the first search
// direction), D = V = 0
template <class T>
__global__ void __launch_bounds__(kSwT) k_sw_start(SwArgs a, const double* __restrict__ scale,
                                                   const double* __restrict__ R64, const T* __restrict__ dS,
                                                   T* __restrict__ R, T* __restrict__ R0, T* __restrict__ D,
                                                   T* __restrict__ PH, T* __restrict__ V) {
    const Tile t = tile_of(a.KT);
    if (sw_skip(a, t.k)) return;
    const double sk = scale[t.k];
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
        const size_t idx = (size_t)r * a.Kp + t.k;
        const T x = (T)(R64[idx] * sk);
        R[idx] = x;
        R0[idx] = x;
        D[idx] = 0;
        PH[idx] = x / dS[idx];
        V[idx] = 0;
    }
}

template <class T>
__global__ void __launch_bounds__(kSwT) k_sw_commit(SwArgs a, const double* __restrict__ scale,
                                                    const T* __restrict__ D, double* __restrict__ X64) {
    const Tile t = tile_of(a.KT);
    if (t.k >= a.K || !(a.flags[t.k] & SW_RUN)) return;
    const double nrm = 1.0 / scale[t.k];
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
        const size_t idx = (size_t)r * a.Kp + t.k;
        X64[idx] += nrm * (double)D[idx];
    }
}

// Starting iterate of the odd rows.  A row without in-group predecessors is a singleton
// SCC: its value bS / dS is exact.  Other rows take the warm start (K x N, by state) or 0.
__global__ void __launch_bounds__(kSwT) k_sw_init(SwArgs a, const double* __restrict__ warm, size_t warm_ld,
                                                  const double* __restrict__ bS, const double* __restrict__ dS,
                                                  double* __restrict__ X64) {
    const Tile t = tile_of(a.KT);
    if (t.k >= a.K) return;
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB) {
        const uint32_t slot = a.ob + r;
        const size_t idx = (size_t)r * a.Kp + t.k;
        double x;
        if (a.ig_ptr[slot] == a.ig_ptr[slot + 1])
            x = bS[idx] / dS[idx];
        else
            x = warm ? warm[(size_t)t.k * warm_ld + a.rows[slot].x] : 0.0;
        X64[idx] = x;
    }
}

// X *= alpha_k = (S X . b) / (S X . S X): the least-squares multiple of the warm start,
// whose residual is never larger than that of a zero start
__global__ void __launch_bounds__(kSwT) k_sw_warm_scale(SwArgs a, const double* __restrict__ yb,
                                                        const double* __restrict__ yy, double* __restrict__ X64) {
    const Tile t = tile_of(a.KT);
    if (t.k >= a.K) return;
    const double alpha = yy[t.k] > 0.0 ? yb[t.k] / yy[t.k] : 0.0;
    for (uint32_t r = blockIdx.x * t.RB + t.rsub; r < a.no; r += gridDim.x * t.RB)
        X64[(size_t)r * a.Kp + t.k] *= alpha;
}

// ---- SCC-resident refinement --------------------------------------------------------------
// One CTA (a team of its warps, a cluster or a cooperative grid: see the modes below) solves
// one SCC for KS systems (a power of two chosen per SCC) from right-hand side to result: the two vectors the operator gathers (the search direction and its
// even-row elimination) stay in shared memory, a thread's own rows in registers, and the
// CTA stops with its own systems.  A Krylov iteration is bounded by its chain of FP64
// reductions, barriers and shared-memory gathers (3.9 us at 256 rows, 27 us at 4,096)
// instead of L2 latency and launches.  Against the launch per step (SCCs above 512 states)
// and the CTA-local solve on global vectors that it replaces: n=12 x 64 rate sets 14.7 ->
// 1.5 ms, n=17 x 185 systems 64.6 -> 14.9 ms, one n=22 solve 277 -> 61 ms.
//
// A work item is (SCC, tile of KS systems) and has a team of warps; a CTA holds several
// teams of small SCCs, each with a barrier and a part of shared memory of its own, because
// a group may have thousands of them beside one of 512 rows, whose CTAs fill an SM each.
// The SCCs of a launch are listed largest first and cut into buckets of equal KS and team
// size.  CTAs past the last item serve the group's singleton SCCs (rows without in-group
// predecessors): z = b / q.
// Most CTAs that share an SCC beyond kSccMaxRows rows of a parity.  512 systems: SCCs of 16K states (two) 11.2 -> 6 ms and
// of 26K to 31K (four) 31 -> 28 and 22 -> 14 ms against the row kernels; of 53K to 58K states
// (eight) 31 -> 38 and 64 -> 78 ms.
constexpr int kSccMaxCluster = 4;
constexpr uint32_t kSccClusterRows = kSccMaxRows * kSccMaxCluster;
struct SccArgs {
    SwArgs a;
    const uint4* scc;  // the launch's SCCs: (first even slot, even rows, first odd slot, odd rows)
    const uint2 *scc_sl, *sl;  // see SweepPlan
    const uint4* ell;
    SccBucket b[kSccBuckets];
    int nb;
    uint32_t ctas;     // CTAs before those of the singleton rows
    const uint32_t *og_ptr, *og_ent;
    const double* x0;
    size_t x0_ld;
    const double* warm;  // K x N warm start by state, or null
    size_t warm_ld;
    const uint32_t* rev; // per slot, flips whose reverse of the row's entries exists (null: the out-mask)
    double* Z;           // [slot][Kp]
    double* own[kOwnCount];  // group-sized scratch, see SccOwn (kSccBig: the first five)
    unsigned* bar;       // kSccGrid: barrier arrivals (0 before the launch), and a failure flag
    unsigned polls, missing;  // kSccGrid: bound of a barrier wait; arrivals that never come (a test's)
    double* part;        // kSccGrid: 2 x CTAs x 3 x KS partial sums
    double tol2, accept2;
    int max_iters, max_outer, stall;
    unsigned long long* ratio;  // per system: max over SCCs of final |r|^2 / |b|^2 (bits of a double >= 0)
    int* fail;                  // per system: 1 once an SCC stays above the acceptance residual
    int *iters, *refines;       // the group's most inner iterations and refinement steps
    // deflated (terminal) groups: kernels into Rb[k][pos[slot]], normalised to sum 1
    const uint32_t* pos;
    double* Rb;
    int TS;
};

// Barrier of a cooperative launch (target: the arrivals it waits for).  A wait is bounded: past
// the bound it sets the failure flag, which ends the other CTAs' waits too.  A CTA whose wait
// ended that way is gone: it takes no part in later barriers and sums and leaves its loops, so
// that the CTAs that still run read nothing that it wrote afterwards into their decisions.  Its
// threads learn of it through a flag that changes only between the two __syncthreads of a
// wait: read outside of them it is the same for all.
__device__ __forceinline__ volatile int& grid_gone() {
    __shared__ int s_gone;
    return *const_cast<volatile int*>(&s_gone);
}
__device__ __forceinline__ void grid_wait(const SccArgs& g, unsigned& target) {
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == 0 && !grid_gone()) {
        __threadfence();
        atomicAdd(g.bar, 1u);
        unsigned n = 0;
        while ((int)(*(volatile unsigned*)g.bar - target) < 0) {
            if (*(volatile unsigned*)(g.bar + 1)) {
                grid_gone() = 1;
                break;
            }
            if (++n > g.polls) atomicExch(g.bar + 1, 1u);
        }
        __threadfence();
    }
    __syncthreads();
}

// a team's barrier: `threads` of the CTA, named by the team
struct SccTeam {
    int id, threads, tid;
};
__device__ __forceinline__ void scc_sync(const SccTeam& m) {
    if (m.threads == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(m.id), "r"(m.threads) : "memory");
}

// The row gathers are bound by the instructions they issue (77% of issue slots at 18
// instructions per entry when entries were loaded, tested and decoded one by one): four
// entries come in one load, untested, already scaled to byte offsets, and shared memory is
// addressed in 32 bits.
__device__ __forceinline__ double lds_f64(uint32_t addr) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t shared_addr(const double* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// byte offsets of an entry's rate and gathered row in arrays of 1 << lks systems
__device__ __forceinline__ uint32_t ell_rate(uint32_t e, int lks) { return (e & 0x1F8u) << lks; }
__device__ __forceinline__ uint32_t ell_row(uint32_t e, int lks) { return (e >> 6 & ~7u) << lks; }
// acc += sum over four entries of rate * X (shared addresses, this thread's system included)
__device__ __forceinline__ void ell_add(double& acc, const uint4& e, uint32_t X, uint32_t rate, int lks) {
    const double r0 = lds_f64(rate + ell_rate(e.x, lks)), x0 = lds_f64(X + ell_row(e.x, lks));
    const double r1 = lds_f64(rate + ell_rate(e.y, lks)), x1 = lds_f64(X + ell_row(e.y, lks));
    const double r2 = lds_f64(rate + ell_rate(e.z, lks)), x2 = lds_f64(X + ell_row(e.z, lks));
    const double r3 = lds_f64(rate + ell_rate(e.w, lks)), x3 = lds_f64(X + ell_row(e.w, lks));
    acc += r0 * x0;
    acc += r1 * x1;
    acc += r2 * x2;
    acc += r3 * x3;
}

// The same of an SCC split over a cluster (one system): the entry's row is in the shared
// memory of CTA e >> 22 of the cluster.
__device__ __forceinline__ double lds_cluster(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    double v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote));
    return v;
}
__device__ __forceinline__ void ell_add_cluster(double& acc, const uint4& e, uint32_t X, uint32_t rate) {
    const double r0 = lds_f64(rate + (e.x & 0x1F8u)), x0 = lds_cluster(X + (e.x >> 6 & 0xFFF8u), e.x >> 22);
    const double r1 = lds_f64(rate + (e.y & 0x1F8u)), x1 = lds_cluster(X + (e.y >> 6 & 0xFFF8u), e.y >> 22);
    const double r2 = lds_f64(rate + (e.z & 0x1F8u)), x2 = lds_cluster(X + (e.z >> 6 & 0xFFF8u), e.z >> 22);
    const double r3 = lds_f64(rate + (e.w & 0x1F8u)), x3 = lds_cluster(X + (e.w >> 6 & 0xFFF8u), e.w >> 22);
    acc += r0 * x0;
    acc += r1 * x1;
    acc += r2 * x2;
    acc += r3 * x3;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Sums of NV values over a team's threads of one system; every thread of a system gets
// the same bits.  `red` holds NV x warps x KS doubles; calls without a barrier in between
// must use different buffers.  Both levels are butterflies, the values interleaved: each
// thread adding up the warps' partial sums itself took 3,000 cycles a value at 32 warps,
// two thirds of an iteration.
template <int NV>
__device__ __forceinline__ void scc_sum(double* red, int lks, const SccTeam& m, double (&v)[NV]) {
    const int lane = m.tid & 31, warp = m.tid >> 5, KS = 1 << lks, total = (m.threads >> 5) << lks;
    for (int o = 16; o >= KS; o >>= 1)
#pragma unroll
        for (int j = 0; j < NV; j++) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
    if (lane < KS)
#pragma unroll
        for (int j = 0; j < NV; j++) red[j * total + (warp << lks) + lane] = v[j];
    scc_sync(m);
    // lane l takes the partial sums l, l + 32, ... of its system l % KS
#pragma unroll
    for (int j = 0; j < NV; j++) v[j] = lane < total ? red[j * total + lane] : 0.0;
    for (int w = lane + 32; w < total; w += 32)
#pragma unroll
        for (int j = 0; j < NV; j++) v[j] += red[j * total + w];
    for (int o = 16; o >= KS; o >>= 1)
#pragma unroll
        for (int j = 0; j < NV; j++) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
}

// out-rate sum of state v (out-mask f) for system s
__device__ __forceinline__ double scc_q(const double* rate, uint32_t v, uint32_t f, int lks, int s) {
    double q = 0.0;
    while (f) {
        const int i = __ffs(f) - 1;
        f &= f - 1;
        q += rate[((2 * i + (int)((v >> i) & 1u)) << lks) | s];
    }
    return q;
}

// Singleton rows of a group, z = (x0 + inflow from earlier groups) / q.  KW = min(32, K
// rounded up to a power of two) adjacent lanes serve the systems of one row, so that
// small batches fill the warp with rows.
__device__ __forceinline__ void scc_singles(const SccArgs& g, uint32_t cta, uint32_t ctas) {
    const SwArgs& a = g.a;
    int lw = 0;
    while (lw < 5 && (1 << lw) < a.K) lw++;
    const int KW = 1 << lw;
    const uint32_t rows = a.ne + a.no, tiles = (uint32_t)((a.K + KW - 1) >> lw), rpb = blockDim.x >> lw;
    for (uint64_t u = (uint64_t)cta * rpb + (threadIdx.x >> lw); u < (uint64_t)rows * tiles; u += (uint64_t)ctas * rpb) {
        const uint32_t t = (uint32_t)(u / rows), r = (uint32_t)(u - (uint64_t)t * rows);
        const int k = (int)(t << lw) + (int)(threadIdx.x & (KW - 1));
        if (k >= a.K) continue;
        const uint32_t slot = sw_slot(a, r);
        const uint4 d = a.desc[slot];
        if (d.w) continue;  // in an SCC of two or more states
        double acc = g.x0[(size_t)(k % a.nrhs) * g.x0_ld + d.x];
        const uint32_t p1 = g.og_ptr[slot + 1];
        for (uint32_t p = g.og_ptr[slot]; p < p1; p += 4) {
            uint32_t e[4];
            double z[4], r4[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) e[u] = p + u < p1 ? __ldg(g.og_ent + p + u) : 0u;
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                z[u] = p + u < p1 ? g.Z[(size_t)ent_slot(e[u]) * a.Kp + k] : 0.0;
                r4[u] = __ldg(a.rateT + (size_t)ent_rate(e[u]) * a.Kp + k);
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; u++)
                if (p + u < p1) acc += r4[u] * z[u];
        }
        double q = 0.0;
        for (uint32_t f = d.y; f; f &= f - 1) {
            const int i = __ffs(f) - 1;
            q += __ldg(a.rateT + (size_t)(2 * i + (int)((d.x >> i) & 1u)) * a.Kp + k);
        }
        g.Z[(size_t)slot * a.Kp + k] = acc / q;
    }
}

// Own-row vectors of a thread.  One row per thread (BIG false): registers.  Else values of
// an array, indexed [row << lks | s], that only this thread touches.
template <bool BIG>
struct SccVec {
    double reg;
    double* mem;
    __device__ __forceinline__ double get(int idx) const { return BIG ? mem[idx] : reg; }
    __device__ __forceinline__ void set(int idx, double x) {
        if (BIG) mem[idx] = x;
        else reg = x;
    }
};

// 1 / x to about an ulp: two Newton steps from a single-precision reciprocal (not finite
// where x is outside its range; the elimination's residual check then rejects the result)
__device__ __forceinline__ double scc_recip(double x) {
    double r = (double)(1.0f / (float)x);
    r = fma(r, fma(-x, r, 1.0), r);
    return fma(r, fma(-x, r, 1.0), r);
}

// kSccSmall: SCCs of at most kSccThreads rows of either parity, a thread per row and
// system, everything but the gathered vectors in registers, the row's first entries included.
// kSccBig: several rows per thread; r, v, p, t and 1 / q in shared memory, r0, d, the
// Schur diagonal, q and the right-hand side in memory (streamed, an item's own run).
// kSccCluster: kSccBig over a cluster of up to kSccMaxCluster CTAs for one system, each with
// kSccMaxRows rows of either parity; gathers read the owner's shared memory, sums are
// exchanged through it (a network of two SCCs of 16,384 states, 64 and 16 systems: 8.1 ->
// 5.5 ms).
// kSccGrid: the whole group, all systems (at most 32), by the whole grid of a cooperative
// launch; every vector in memory as [row][KS].  For groups beyond a CTA's shared memory when
// there are at most 32 systems: the row kernels would move 32 / K times the bytes and launch
// seven kernels per iteration (n=22, one system, 11 groups of 16K to 370K rows: 24 -> 4 ms;
// split over two or more tiles it is no faster than the row kernels, 58K rows x 512 systems
// 144 against 65 ms).
// DEFL: the deflated operator of a terminal SCC (see k_sw_defl_fin): S x + u gamma(x),
// u_o = q_o / s, whose gamma is summed at the barrier that the elimination ends with anyway.
enum { kSccSmall, kSccBig, kSccGrid, kSccCluster };
template <int MODE, bool DEFL>
__global__ void __launch_bounds__(MODE == kSccSmall ? kSccThreads : kSccThreadsBig, 1)
    k_sw_scc(const __grid_constant__ SccArgs g) {
    constexpr bool CLUSTER = MODE == kSccCluster, BIG = MODE == kSccBig || CLUSTER, GRID = MODE == kSccGrid,
                   MEM = BIG || GRID;
    uint32_t rank = 0, ranks = 1;
    if (CLUSTER) {
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    }
    extern __shared__ double s_all[];
    const SwArgs& a = g.a;
    if (!GRID && !CLUSTER && blockIdx.x >= g.ctas) {
        if (!DEFL) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            scc_singles(g, blockIdx.x - g.ctas, gridDim.x - g.ctas);
        }
        return;
    }
    int bk = 0;
    while (!CLUSTER && bk + 1 < g.nb && blockIdx.x >= g.b[bk + 1].cta0) bk++;
    const SccBucket& bu = g.b[bk];
    const int lteam = MEM ? 10 : bu.lteam;
    const SccTeam team = {MEM ? 0 : (int)(threadIdx.x >> lteam), 1 << lteam, (int)(threadIdx.x & ((1u << lteam) - 1u))};
    const uint32_t item = GRID ? 0u : CLUSTER ? blockIdx.x / ranks : BIG ? blockIdx.x - bu.cta0 : (blockIdx.x - bu.cta0) * bu.teams + team.id;
    if (!MEM && (team.id >= bu.teams || item >= bu.items)) return;
    double* s_scc = MEM ? s_all : s_all + (size_t)team.id * bu.stride;
    const int lks = bu.lks, KS = 1 << lks;
    const uint32_t tiles = (uint32_t)((a.K + KS - 1) >> lks), tile = item % tiles;
    const uint4 sc = GRID ? make_uint4(a.beg, a.ne, a.ob, a.no) : g.scc[bu.scc0 + item / tiles];
    uint2 first = GRID ? make_uint2(0u, 0u) : g.scc_sl[bu.scc0 + item / tiles];
    // the rates, in flight with the SCC's description
    const int nact = team.threads;
    double* rate = s_scc;
#pragma unroll 4
    for (int idx = team.tid; idx < (2 * a.n) << lks; idx += nact)
        rate[idx] = a.rateT[(size_t)(idx >> lks) * a.Kp + (size_t)tile * KS + (idx & (KS - 1))];
    uint32_t ev0 = sc.x, od0 = sc.z;
    int se = (int)sc.y, so = (int)sc.w;
    const double inv_s = 1.0 / (double)(se + so);
    if (CLUSTER) {
        // this CTA's rows
        const int r0 = (int)rank * kSccMaxRows;
        ev0 += r0;
        od0 += r0;
        first.x += r0 / 32;
        first.y += r0 / 32;
        se = min(max(se - r0, 0), kSccMaxRows);
        so = min(max(so - r0, 0), kSccMaxRows);
    }
    // rows that the arrays are laid out for: the same in every CTA of a cluster
    const int le_rows = CLUSTER ? kSccMaxRows : se, lo_rows = CLUSTER ? kSccMaxRows : so, sm = max(le_rows, lo_rows);
    const int s = team.tid & (KS - 1);
    const int rs = ((GRID ? (int)blockIdx.x * nact : 0) + team.tid) >> lks, RS = ((GRID ? (int)gridDim.x : 1) * nact) >> lks;
    const int k = (int)tile * KS + s;
    const size_t Kp = a.Kp;
    const bool act = k < a.K;
    // both with a zero row past the last, for the entries that a row of a slice lacks
    double* A = GRID ? g.own[kOwnA] : rate + ((size_t)(2 * a.n) << lks);  // odd rows: the vector whose product is formed
    double* W = GRID ? g.own[kOwnW] : A + ((size_t)(sm + 1) << lks);      // even rows: its elimination
    double* red0 = GRID ? rate + ((size_t)(2 * a.n) << lks) : W + ((size_t)(le_rows + 1) << lks);
    double* red1 = red0 + ((size_t)(2 * (nact >> 5)) << lks);
    double* red2 = red1 + ((size_t)(3 * (nact >> 5)) << lks);
    SccVec<MEM> R, V, P, T, IQ, R0, D, dS, q, BS;
    if constexpr (GRID) {
        R0.mem = g.own[kOwnR0];
        D.mem = g.own[kOwnD];
        dS.mem = g.own[kOwnDS];
        q.mem = g.own[kOwnQ];
        BS.mem = g.own[kOwnBS];
        R.mem = g.own[kOwnR];
        V.mem = g.own[kOwnV];
        P.mem = g.own[kOwnP];
        T.mem = g.own[kOwnT];
        IQ.mem = g.own[kOwnIQ];
    }
    if constexpr (BIG) {
        R.mem = red2 + ((size_t)(nact >> 5) << lks);
        V.mem = R.mem + ((size_t)lo_rows << lks);
        P.mem = V.mem + ((size_t)lo_rows << lks);
        T.mem = P.mem + ((size_t)lo_rows << lks);
        IQ.mem = T.mem + ((size_t)lo_rows << lks);
        // the SCC's block of odd rows x Kp of a group vector, tile by tile (row by row there)
        const size_t o = (size_t)(sc.z - a.beg - a.ne) * Kp + (size_t)tile * KS * sc.w + (CLUSTER ? rank * kSccMaxRows : 0);
        R0.mem = g.own[kOwnR0] + o;
        D.mem = g.own[kOwnD] + o;
        dS.mem = g.own[kOwnDS] + o;
        q.mem = g.own[kOwnQ] + o;
        BS.mem = g.own[kOwnBS] + o;
    }
    // line j of a slice of even or odd rows
    const bool narrow = !MEM && scc_narrow(sc.y, sc.w);
    auto line_at = [&](const uint2& sl, uint32_t j, uint32_t rows) {
        return g.ell + (narrow ? (size_t)(sl.y + j * rows) : (size_t)(sl.y + j) * 32);
    };
    // one row per thread: its first two lines stay in registers
    uint4 ee[2], eo[2];
    uint2 le = make_uint2(0u, 0u), lo = make_uint2(0u, 0u);
    uint2 row_e = le, row_o = le, og_e = le, og_o = le;
    if (!MEM) {
        if (rs < se) le = __ldg(g.sl + first.x + (rs >> 5));
        if (rs < so) lo = __ldg(g.sl + first.y + (rs >> 5));
        // and so do the rows and the first entries from earlier groups
        if (rs < se) {
            row_e = a.rows[ev0 + rs];
            if (!DEFL) og_e = make_uint2(g.og_ptr[ev0 + rs], g.og_ptr[ev0 + rs + 1]);
        }
        if (rs < so) {
            row_o = a.rows[od0 + rs];
            if (!DEFL) og_o = make_uint2(g.og_ptr[od0 + rs], g.og_ptr[od0 + rs + 1]);
        }
        for (int j = 0; j < 2; j++) {
            if (j < (int)le.x) ee[j] = __ldg(line_at(le, j, sc.y) + (rs & 31));
            if (j < (int)lo.x) eo[j] = __ldg(line_at(lo, j, sc.w) + (rs & 31));
        }
    }
    const uint32_t rate_at = shared_addr(rate + s);
    // fn(row, index) of the own rows below count
    auto each = [&](int count, auto fn) {
        if constexpr (MEM) {
            for (int r = rs; r < count; r += RS) fn(r, (r << lks) | s);
        } else if (rs < count) {
            fn(rs, (rs << lks) | s);
        }
    };
    // fn(row, index, sum over its entries of X) of the own even or odd rows; with several,
    // the next line, of the same row or the next one, is in flight while one is summed
    auto gather = [&](auto even, const double* X, auto fn) {
        constexpr bool EVEN = decltype(even)::value;
        const int count = EVEN ? se : so;
        [[maybe_unused]] const uint32_t xs = GRID ? 0u : shared_addr(X + s);
        if constexpr (GRID) {
            const uint32_t base = EVEN ? od0 : ev0;
            for (int r = rs; r < count; r += RS) {
                const uint2 zw = __ldg(reinterpret_cast<const uint2*>(a.desc + (EVEN ? ev0 : od0) + r) + 1);
                double acc = 0.0;
                for (uint32_t j = 0; j < zw.y; j += 8) {
                    uint32_t e[8];
                    double x[8];
#pragma unroll
                    for (uint32_t u = 0; u < 8; u++) e[u] = j + u < zw.y ? __ldg(a.ig_ent + zw.x + j + u) : 0u;
#pragma unroll
                    for (uint32_t u = 0; u < 8; u++)
                        x[u] = j + u < zw.y ? __ldcg(X + ((size_t)(ent_slot(e[u]) - base) << lks) + s) : 0.0;
#pragma unroll
                    for (uint32_t u = 0; u < 8; u++) acc += rate[(ent_rate(e[u]) << lks) | s] * x[u];
                }
                fn(r, (r << lks) | s, acc);
            }
        } else if constexpr (BIG) {
            auto add = [&](double& acc, const uint4& e) {
                if constexpr (CLUSTER) ell_add_cluster(acc, e, xs, rate_at);
                else ell_add(acc, e, xs, rate_at, lks);
            };
            if (rs >= count) return;
            const uint2* sl = g.sl + (EVEN ? first.x : first.y);
            const uint2 none = make_uint2(0u, 0u);
            uint2 cur = __ldg(sl + (rs >> 5)), nxt = rs + RS < count ? __ldg(sl + ((rs + RS) >> 5)) : none;
            const uint4* line = g.ell + (size_t)cur.y * 32 + (rs & 31);
            uint4 e = cur.x ? __ldg(line) : make_uint4(0u, 0u, 0u, 0u);
            for (int r = rs; r < count; r += RS) {
                const uint4* line2 = g.ell + (size_t)nxt.y * 32 + ((r + RS) & 31);
                const uint32_t next_lines = nxt.x;
                uint32_t left = cur.x;
                double acc = 0.0;
                uint4 f = e;
                while (left > 1) {
                    line += 32;
                    f = __ldg(line);
                    add(acc, e);
                    e = f;
                    left--;
                }
                if (next_lines) f = __ldg(line2);
                cur = nxt;
                nxt = r + 2 * RS < count ? __ldg(sl + ((r + 2 * RS) >> 5)) : none;
                if (left) add(acc, e);
                e = f;
                line = line2;
                fn(r, (r << lks) | s, acc);
            }
        } else if (rs < count) {
            const uint2 l = EVEN ? le : lo;
            double acc = 0.0;
            if (l.x > 0) ell_add(acc, EVEN ? ee[0] : eo[0], xs, rate_at, lks);
            if (l.x > 1) ell_add(acc, EVEN ? ee[1] : eo[1], xs, rate_at, lks);
            for (uint32_t j = 2; j < l.x; j++)  // (not narrow)
                ell_add(acc, __ldg(g.ell + (size_t)(l.y + j) * 32 + (rs & 31)), xs, rate_at, lks);
            fn(rs, (rs << lks) | s, acc);
        }
    };
    constexpr auto even_rows = std::true_type{};
    constexpr auto odd_rows = std::false_type{};
    // barrier of all threads of the item, and sums over them (see scc_sum); a grid's CTAs
    // add up their sums in one order, so that they take the same decisions
    unsigned target = g.missing;
    auto gone = [&]() {
        if constexpr (GRID) return grid_gone() != 0;
        else return false;
    };
    if constexpr (GRID)
        if (threadIdx.x == 0) grid_gone() = 0;
    auto sync = [&]() {
        if constexpr (GRID) grid_wait(g, target);
        else if constexpr (CLUSTER) cluster_sync();
        else scc_sync(team);
    };
    unsigned sums = 0;
    auto sum = [&](double* red, auto& v) {
        constexpr int NV = (int)(sizeof(v) / sizeof(double));
        scc_sum<NV>(red, lks, team, v);
        if constexpr (CLUSTER) {
            // the CTAs' sums, added in rank order by every thread
            __shared__ double s_xch[2][3];
            double* x = s_xch[sums++ & 1u];
            if (team.tid == 0)
#pragma unroll
                for (int j = 0; j < NV; j++) x[j] = v[j];
            cluster_sync();
            const uint32_t at = shared_addr(x);
#pragma unroll
            for (int j = 0; j < NV; j++) {
                v[j] = 0.0;
                for (uint32_t c = 0; c < ranks; c++) v[j] += lds_cluster(at + 8 * j, c);
            }
        }
        if constexpr (GRID) {
            double* part = g.part + (size_t)(sums++ & 1u) * ((size_t)gridDim.x * 3 << lks);
            if (team.tid < KS && !gone())  // (a return here instead spills 50 bytes a thread)
#pragma unroll
                for (int j = 0; j < NV; j++) __stcg(part + ((size_t)(blockIdx.x * 3 + j) << lks) + s, v[j]);
            grid_wait(g, target);
#pragma unroll
            for (int j = 0; j < NV; j++) v[j] = 0.0;
            for (int c = team.tid >> lks; c < (int)gridDim.x; c += nact >> lks)
#pragma unroll
                for (int j = 0; j < NV; j++) v[j] += __ldcg(part + ((size_t)(c * 3 + j) << lks) + s);
            scc_sum<NV>(red, lks, team, v);
            __syncthreads();  // red is free again
        }
    };
    if (!GRID && rs == 0) {
        A[(le_rows << lks) | s] = 0.0;
        W[(le_rows << lks) | s] = 0.0;
    }
    // (four entries in flight: small groups are chains of such round trips to L2)
    auto rhs = [&](uint2 og, uint32_t v) {
        double acc = g.x0[(size_t)(k % a.nrhs) * g.x0_ld + v];
        const uint32_t p1 = og.y;
        for (uint32_t p = og.x; p < p1; p += 4) {
            uint32_t e[4];
            double z[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) e[u] = p + u < p1 ? __ldg(g.og_ent + p + u) : 0u;
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) z[u] = p + u < p1 ? g.Z[(size_t)ent_slot(e[u]) * Kp + k] : 0.0;
#pragma unroll
            for (uint32_t u = 0; u < 4; u++)
                if (p + u < p1) acc += rate[(ent_rate(e[u]) << lks) | s] * z[u];
        }
        return acc;
    };
    auto og_of = [&](uint32_t slot) { return make_uint2(g.og_ptr[slot], g.og_ptr[slot + 1]); };
    // From here on this launch reads what earlier ones of the sweep wrote (and lets the next
    // one start up to this point, which only reads the plan and the rates).
    if (!GRID) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    if (GRID) __syncthreads();
    else sync();
    // even rows: 1 / q (in A too, for the Schur diagonal), and b / q, kept in Z until the end
    each(se, [&](int r, int idx) {
        const uint32_t slot = ev0 + r;
        const uint2 d = MEM ? a.rows[slot] : row_e;
        const double iq = 1.0 / scc_q(rate, d.x, d.y, lks, s);
        IQ.set(idx, iq);
        A[idx] = iq;
        double w = 0.0;
        if (!DEFL && act) {
            w = rhs(MEM ? og_of(slot) : og_e, d.x) * iq;
            g.Z[(size_t)slot * Kp + k] = w;
        }
        W[idx] = w;
    });
    if (!DEFL)
        each(so, [&](int r, int idx) {
            R.set(idx, !act ? 0.0 : MEM ? rhs(og_of(od0 + r), a.rows[od0 + r].x) : rhs(og_o, row_o.x));
        });
    sync();
    // odd rows: q, Schur diagonal, reduced right-hand side, starting iterate
    double sum1[1] = {0.0};
    gather(odd_rows, W, [&](int r, int idx, double inflow) {
        const uint32_t slot = od0 + r;
        const uint2 d = MEM ? a.rows[slot] : row_o;
        const double qv = scc_q(rate, d.x, d.y, lks, s);
        double dv = qv;
        // rate(e -> o) rate(o -> e) / q_e where both edges exist: the reverse flips the same bit
        const uint32_t both = g.rev ? g.rev[slot] : d.y;
        auto diag = [&](uint32_t ri, double iq) {
            if ((both >> (ri >> 1)) & 1u) dv -= rate[(ri << lks) | s] * rate[((ri ^ 1u) << lks) | s] * iq;
        };
        if constexpr (GRID) {
            const uint4 full = a.desc[slot];
            for (uint32_t j = full.z; j < full.z + full.w; j++) {
                const uint32_t e = __ldg(a.ig_ent + j);
                diag((uint32_t)ent_rate(e), __ldcg(A + ((size_t)(ent_slot(e) - ev0) << lks) + s));
            }
        } else {
            const uint2 sl = __ldg(g.sl + first.y + (r >> 5));
            for (uint32_t j = 0; j < 4 * sl.x; j++) {
                const uint32_t e =
                    __ldg(reinterpret_cast<const uint32_t*>(line_at(sl, j / 4, sc.w) + (r & 31)) + j % 4);
                diag(e >> 3 & 63u, CLUSTER ? lds_cluster(shared_addr(A) + (e >> 6 & 0xFFF8u), e >> 22) : A[((e >> 9) << lks) | s]);
            }
        }
        q.set(idx, qv);
        dS.set(idx, dv);
        const double b = DEFL ? qv * inv_s : R.get(idx) + inflow;
        sum1[0] += b * b;
        R.set(idx, b);
        BS.set(idx, b);
        if (act) g.Z[(size_t)slot * Kp + k] = !DEFL && g.warm ? g.warm[(size_t)k * g.warm_ld + d.x] : 0.0;
    });
    const bool dense = !MEM && !DEFL && scc_dense(so, g.max_iters);
    const int ld = scc_dense_ld(so);
    double* M = red2 + ((size_t)(nact >> 5) << lks);  // [row][column], the right-hand side last
    double* pivot = M + ((size_t)(so * ld) << lks);   // 1 / pivot of this and the next step
    auto at = [&](int r, int c) -> double& { return M[((r * ld + c) << lks) | s]; };
    if (!MEM && dense && rs < so) {
        // own row of the Schur complement: q_o - sum over e of rate(e -> o) / q_e rate(o' -> e)
        for (int c = 0; c < so; c++) at(rs, c) = 0.0;
        at(rs, rs) = q.get(0);
        at(rs, so) = R.get(0);
        for (uint32_t j = 0; j < lo.x; j++) {
            const uint4 e4 = __ldg(line_at(lo, j, sc.w) + (rs & 31));
            const uint32_t es[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint32_t er = es[u] >> 9;
                if ((int)er == se) break;
                const double w = rate[((es[u] >> 3 & 63u) << lks) | s] * A[(er << lks) | s];
                const uint2 sl = __ldg(g.sl + first.x + (er >> 5));
                for (uint32_t i = 0; i < sl.x; i++) {
                    const uint4 f4 = __ldg(line_at(sl, i, sc.y) + (er & 31));
                    const uint32_t fs[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
                    for (int x = 0; x < 4; x++)
                        if ((int)(fs[x] >> 9) != so)
                            at(rs, (int)(fs[x] >> 9)) -= w * rate[((fs[x] >> 3 & 63u) << lks) | s];
                }
            }
        }
        if (rs == 0) pivot[s] = scc_recip(at(0, 0));
    }
    sum(red1, sum1);
    const double b2 = sum1[0];
    if (!GRID && rs == 0) A[(lo_rows << lks) | s] = 0.0;  // 1 / q of an even row until here
    if (!MEM && dense) {
        // Gauss-Jordan without pivoting (the rows of an M-matrix, diagonally dominant by
        // columns); the true residual below decides whether it is good enough
        for (int j = 0; j < so; j++) {
            if (rs < so && rs != j) {
                const double f = at(rs, j) * pivot[((j & 1) << lks) | s];
                const double x = at(rs, j + 1) - f * at(j, j + 1);
                at(rs, j + 1) = x;
                if (rs == j + 1) pivot[(((j + 1) & 1) << lks) | s] = scc_recip(x);
#pragma unroll 4
                for (int c = j + 2; c <= so; c++) at(rs, c) -= f * at(j, c);
            }
            scc_sync(team);
        }
        if (rs < so && act) g.Z[(size_t)(od0 + rs) * Kp + k] = at(rs, so) / at(rs, rs);
    }
    double gamma = 0.0;
    // W = elimination of A (and gamma(A)), with the barrier after it
    auto elim = [&]() {
        double gm[1] = {0.0};
        gather(even_rows, A, [&](int, int idx, double sum) {
            const double w = sum * IQ.get(idx);
            W[idx] = w;
            if (DEFL) gm[0] += w;
        });
        if (DEFL) {
            each(so, [&](int, int idx) { gm[0] += A[idx]; });
            sum(red2, gm);
            gamma = gm[0];
        } else {
            sync();
        }
    };
    // fn(index, own odd row's value of the operator applied to A)
    auto apply = [&](auto fn) {
        gather(odd_rows, W, [&](int, int idx, double sum) {
            const double qv = q.get(idx);
            double y = qv * A[idx] - sum;
            if (DEFL) y += gamma * (qv * inv_s);
            fn(idx, y);
        });
    };
    auto load_x = [&]() {
        each(so, [&](int r, int idx) { A[idx] = act ? g.Z[(size_t)(od0 + r) * Kp + k] : 0.0; });
        sync();
    };
    bool done = !act || !(b2 > 0.0), failed = false;
    const bool warm = !DEFL && !dense && g.warm != nullptr;
    if (warm) {
        // least-squares multiple (S x . b) / (S x . S x) of the warm start: its residual is
        // never larger than that of a zero start
        load_x();
        elim();
        double v[2] = {0.0, 0.0};
        apply([&](int idx, double y) {
            v[0] += y * BS.get(idx);
            v[1] += y * y;
        });
        sum(red0, v);
        const double al = v[1] > 0.0 ? v[0] / v[1] : 0.0;
        if (act) each(so, [&](int r, int) { g.Z[(size_t)(od0 + r) * Kp + k] *= al; });
    }
    double prev = 0.0, rr = b2;
    int noimp = 0, its = 0;
    int outer = 0;  // refinement steps taken
    for (;; outer++) {
        if (outer > 0 || warm || dense) {
            // true residual r = b - S x
            load_x();
            elim();
            double v[1] = {0.0};
            apply([&](int idx, double y) {
                const double res = BS.get(idx) - y;
                R.set(idx, res);
                v[0] += res * res;
            });
            sum(red1, v);
            rr = v[0];
            if (dense && outer == 0 && act && !(rr < b2)) {
                // a zero start is better (a singular block, overflow), and the answer where
                // the SCC gets no mass (b2 == 0: done already, whatever the pivots were)
                each(so, [&](int r, int idx) {
                    g.Z[(size_t)(od0 + r) * Kp + k] = 0.0;
                    R.set(idx, BS.get(idx));
                });
                rr = b2;
            }
        }
        if (!done) {
            if (rr <= g.tol2 * b2) {
                done = true;
            } else {
                if (outer > 0 && !(rr < 0.25 * prev)) noimp++;
                if (noimp >= 2 || !isfinite(rr)) {
                    // stagnation: accepted within the acceptance residual
                    done = true;
                    failed = !(rr <= g.accept2 * b2);
                } else if (outer >= g.max_outer) {
                    // out of refinement steps while still improving: the fallback redoes it
                    done = true;
                    failed = true;
                }
            }
        }
        // every warp holds every system of the CTA, and its sums are the same everywhere
        if (!__any_sync(0xffffffffu, !done)) break;
        prev = rr;
        const bool started = !done;
        bool run = started;
        const double nrm = sqrt(rr), scale = nrm > 0.0 ? 1.0 / nrm : 0.0;
        const double target = fmax(1e-26, 0.01 * g.tol2 * b2 * scale * scale);
        // BiCGStab on the residual scaled to unit norm, right preconditioner dS; the next
        // search direction needs no barrier of its own: beta = -(r0 . t) / (r0 . v)
        each(so, [&](int, int idx) {
            const double x = R.get(idx) * scale;
            R.set(idx, x);
            R0.set(idx, x);
            D.set(idx, 0.0);
            A[idx] = x / dS.get(idx);
        });
        sync();
        double rho = 1.0, best = 1.0;
        int it = 0, stall = 0;
        while (!gone() && __any_sync(0xffffffffu, run)) {
            elim();
            double v1[1] = {0.0};
            apply([&](int idx, double y) {
                V.set(idx, y);
                v1[0] += R0.get(idx) * y;
            });
            sum(red0, v1);
            const double r0v = v1[0], alpha = r0v != 0.0 ? rho / r0v : 0.0;
            each(so, [&](int, int idx) {
                P.set(idx, A[idx]);
                A[idx] = (R.get(idx) - alpha * V.get(idx)) / dS.get(idx);
            });
            sync();
            elim();
            double v3[3] = {0.0, 0.0, 0.0};
            apply([&](int idx, double y) {
                T.set(idx, y);
                v3[0] += y * (dS.get(idx) * A[idx]);
                v3[1] += y * y;
                v3[2] += R0.get(idx) * y;
            });
            sum(red1, v3);
            const double omega = v3[1] > 0.0 ? v3[0] / v3[1] : 0.0, beta = r0v != 0.0 ? -v3[2] / r0v : 0.0;
            double v2[2] = {0.0, 0.0};
            each(so, [&](int, int idx) {
                const double sh = A[idx], ph = P.get(idx), d = dS.get(idx);
                if (run) D.set(idx, D.get(idx) + (alpha * ph + omega * sh));
                const double rv = d * sh - omega * T.get(idx);
                R.set(idx, rv);
                v2[0] += rv * rv;
                v2[1] += R0.get(idx) * rv;
                A[idx] = (rv + beta * (d * ph - omega * V.get(idx))) / d;
            });
            sum(red0, v2);
            if (run) {
                it++;
                if (v2[0] < 0.5 * best) {
                    best = v2[0];
                    stall = 0;
                } else {
                    stall++;
                }
                run = !(!(v2[0] > target) || it >= g.max_iters || r0v == 0.0 || omega == 0.0 || v2[1] == 0.0 ||
                        !isfinite(v2[0]) || !isfinite(alpha) || stall >= g.stall);
                rho = v2[1];
            }
        }
        if (gone()) break;
        its += it;
        if (started) each(so, [&](int r, int idx) { g.Z[(size_t)(od0 + r) * Kp + k] += nrm * D.get(idx); });
    }
    if (gone()) return;  // the call fails
    // even rows from the odd solution
    load_x();
    double total[1] = {0.0};
    gather(even_rows, A, [&](int r, int idx, double sum) {
        const double w = sum * IQ.get(idx);
        if (DEFL) {
            W[idx] = w;
            total[0] += w;
        } else if (act) {
            g.Z[(size_t)(ev0 + r) * Kp + k] += w;
        }
    });
    if (DEFL) {
        each(so, [&](int, int idx) { total[0] += A[idx]; });
        sum(red1, total);
        const double inv = total[0] != 0.0 ? 1.0 / total[0] : 0.0;
        if (act) {
            each(se, [&](int r, int idx) { g.Rb[(size_t)k * g.TS + g.pos[ev0 + r]] = W[idx] * inv; });
            each(so, [&](int r, int idx) { g.Rb[(size_t)k * g.TS + g.pos[od0 + r]] = A[idx] * inv; });
        }
    }
    if (CLUSTER) cluster_sync();  // no CTA leaves while others may read its shared memory
    if (act && rs == 0 && rank == 0) {
        atomicMax(g.ratio + k, (unsigned long long)__double_as_longlong(b2 > 0.0 ? rr / b2 : 0.0));
        if (failed) g.fail[k] = 1;
        atomicMax(g.iters, its);
        atomicMax(g.refines, outer);
    }
}

// ---- terminal masses ----------------------------------------------------------------------
// y[k][t] += x0(v) + sum over transient predecessors u of v of rate(u -> v) z_u, v in t
__global__ void __launch_bounds__(kSwT) k_sw_term(SwArgs a, int TS, const int32_t* __restrict__ order,
                                                  const int32_t* __restrict__ term_of,
                                                  const uint32_t* __restrict__ tp_ptr,
                                                  const uint32_t* __restrict__ tp_ent, const double* __restrict__ x0,
                                                  size_t x0_ld, const double* __restrict__ Z, int T,
                                                  double* __restrict__ y) {
    extern __shared__ double s_rate[];
    const Tile t = tile_of(a.KT);
    sw_rates(s_rate, a, t);
    if (t.k >= a.K) return;
    for (int p = blockIdx.x * t.RB + t.rsub; p < TS; p += gridDim.x * t.RB) {
        const uint32_t v = (uint32_t)order[p];
        double acc = x0[(size_t)(t.k % a.nrhs) * x0_ld + v];
        for (uint32_t e = tp_ptr[p]; e < tp_ptr[p + 1]; e++) {
            const uint32_t ent = tp_ent[e];
            acc += s_rate[ent_rate(ent) * t.KT + t.lane] * Z[(size_t)ent_slot(ent) * a.Kp + t.k];
        }
        atomicAdd(&y[(size_t)t.k * T + term_of[v]], acc);
    }
}

// occ[k][state of slot] = Z[slot][k]: a 32 x 32 transpose through shared memory
__global__ void __launch_bounds__(256) k_sw_occupation(uint32_t M, int K, int Kp, size_t N, const uint2* __restrict__ rows,
                                                       const double* __restrict__ Z, double* __restrict__ occ) {
    __shared__ double tile[32][33];
    __shared__ uint32_t st[32];
    const uint32_t s0 = blockIdx.x * 32;
    const int k0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (threadIdx.x < 32 && s0 + threadIdx.x < M) st[threadIdx.x] = rows[s0 + threadIdx.x].x;
    for (int r = ty; r < 32; r += 8)
        if (s0 + r < M) tile[r][tx] = Z[(size_t)(s0 + r) * Kp + k0 + tx];
    __syncthreads();
    for (int c = ty; c < 32; c += 8) {
        const int k = k0 + c;
        if (k < K && s0 + tx < M) occ[(size_t)k * N + st[tx]] = tile[tx][c];
    }
}

__global__ void k_sw_rate_table(int n, int K, int Kp, int nrhs, const double* __restrict__ rates,
                                double* __restrict__ rateT) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (k >= Kp) return;
    rateT[(size_t)j * Kp + k] = k < K ? rates[(size_t)(k / nrhs) * 2 * n + j] : 0.0;
}

// ---- host side ------------------------------------------------------------------------------
enum SwSlot { W_Z, W_RATET, W_BV, W_BS, W_R64, W_DS64, W_DS32, W_W64, W_WT, W_R, W_R0, W_PH, W_V, W_SH, W_TT,
              W_D, W_SCAL, W_ISCAL, W_CNT, W_LOC, W_QO, W_IQE, W_PERM, W_PART, W_COUNT };

bool debug_on();

// Terminal plan: one grid group per terminal SCC above kDenseTerminalMax states, its
// even-parity states first; predecessor entries only from the same SCC (a terminal SCC
// receives edges from transient states too, which its kernel does not see).
int build_terminal_plan(const std::vector<int32_t>& order, const std::vector<int32_t>& offsets, int T,
                        const std::vector<uint32_t>& F, const std::vector<uint32_t>& G, cudaStream_t s,
                        SweepPlan*& out) {
    out = nullptr;
    bool any = false;
    for (int t = 0; t < T; t++) any |= offsets[t + 1] - offsets[t] > kDenseTerminalMax;
    if (!any) return ESL_OK;
    auto* TP = new SweepPlan();
    std::vector<uint32_t> tslot(F.size(), 0xFFFFFFFFu);
    std::vector<uint2> rows;
    std::vector<uint32_t> pos;
    for (int t = 0; t < T; t++) {
        const int sz = offsets[t + 1] - offsets[t];
        if (sz <= kDenseTerminalMax) continue;
        SwGroup g{};
        g.beg = (uint32_t)rows.size();
        g.kind = 2;
        g.max_scc = sz;
        g.term = t;
        g.pos0 = (uint32_t)offsets[t];
        for (int par = 0; par < 2; par++) {
            for (int p = offsets[t]; p < offsets[t + 1]; p++) {
                const uint32_t v = (uint32_t)order[p];
                if ((uint32_t)(__builtin_popcount(v) & 1) != (uint32_t)par) continue;
                tslot[v] = (uint32_t)rows.size();
                rows.push_back(make_uint2(v, F[v]));
                pos.push_back((uint32_t)p);
            }
            (par ? g.no : g.ne) = (uint32_t)rows.size() - g.beg - (par ? g.ne : 0);
        }
        g.s0 = (uint32_t)TP->groups.size();
        g.ns = 1;
        TP->max_rows = std::max(TP->max_rows, g.ne + g.no);
        TP->max_even = std::max(TP->max_even, g.ne);
        TP->max_odd = std::max(TP->max_odd, g.no);
        TP->groups.push_back(g);
    }
    const uint32_t M = (uint32_t)rows.size();
    TP->M = M;
    std::vector<uint32_t> ig_ptr(M + 1, 0), ig;
    for (uint32_t sl = 0; sl < M; sl++) {
        const uint32_t v = rows[sl].x;
        uint32_t in = G[v];
        while (in) {
            const int i = __builtin_ctz(in);
            in &= in - 1;
            const uint32_t su = tslot[v ^ (1u << i)];
            if (su == 0xFFFFFFFFu) continue;  // a transient predecessor
            ig.push_back((su << 6) | (2u * (uint32_t)i + (((v >> i) & 1u) ^ 1u)));
        }
        ig_ptr[sl + 1] = (uint32_t)ig.size();
    }
    for (SwGroup& g : TP->groups) g.nin = ig_ptr[g.beg + g.ne + g.no] - ig_ptr[g.beg];
    std::vector<uint4> desc(M);
    for (uint32_t sl = 0; sl < M; sl++)
        desc[sl] = make_uint4(rows[sl].x, rows[sl].y, ig_ptr[sl], ig_ptr[sl + 1] - ig_ptr[sl]);
    int rc = ESL_OK;
    auto up = [&](auto& d, const auto& h) {
        if (rc != ESL_OK) return;
        rc = d.alloc(std::max<size_t>(h.size(), 1));
        if (rc == ESL_OK && !h.empty() &&
            cudaMemcpyAsync(d.get(), h.data(), h.size() * sizeof(h[0]), cudaMemcpyHostToDevice, s) != cudaSuccess)
            rc = fail(ESL_ERR_CUDA, "terminal plan upload failed");
    };
    up(TP->rows, rows);
    up(TP->desc, desc);
    up(TP->ig_ptr, ig_ptr);
    up(TP->ig_ent, ig);
    up(TP->pos, pos);
    if (rc == ESL_OK && cudaStreamSynchronize(s) != cudaSuccess) rc = fail(ESL_ERR_CUDA, "terminal plan upload failed");
    if (rc != ESL_OK) {
        delete TP;
        return rc;
    }
    out = TP;
    return ESL_OK;
}

int finish_scc_list(esl_ctx* ctx, SweepPlan* P, const std::vector<uint4>* list);

// The lines of SweepPlan::sl and ell made on the host from the predecessor lists, in place of
// those that finish_scc_list made.
int host_lines(esl_ctx* ctx, SweepPlan* P, const std::vector<uint32_t>& ig_ptr, const std::vector<uint32_t>& ig) {
    uint32_t count = 0;
    for (const SwGroup& g : P->groups) count += g.ns;
    if (count == 0 || !P->sl.get()) return ESL_OK;
    cudaStream_t s = ctx->stream;
    std::vector<uint4> scc(count), wide, narrow;
    ESL_CUDA(cudaMemcpyAsync(scc.data(), P->scc.get(), (size_t)count * sizeof(uint4), cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaStreamSynchronize(s));
    std::vector<uint2> sl;
    std::vector<uint8_t> is_narrow;
    for (const uint4& c : scc) {
        if (std::max(c.y, c.w) > kSccClusterRows) continue;
        const bool nar = scc_narrow(c.y, c.w), split = std::max(c.y, c.w) > (uint32_t)kSccMaxRows;
        for (int par = 0; par < 2; par++) {
            const uint32_t slot0 = par ? c.z : c.x, rows = par ? c.w : c.y, other = par ? c.x : c.z,
                           others = par ? c.y : c.w;
            for (uint32_t r0 = 0; r0 < rows; r0 += 32) {
                const uint32_t here = std::min(32u, rows - r0), width = nar ? here : 32u;
                uint32_t most = 0;
                for (uint32_t r = r0; r < r0 + here; r++) most = std::max(most, ig_ptr[slot0 + r + 1] - ig_ptr[slot0 + r]);
                const uint32_t lines = (most + 3) / 4;
                std::vector<uint4>& out = nar ? narrow : wide;
                sl.push_back(make_uint2(lines, (uint32_t)(nar ? out.size() : out.size() / 32)));
                is_narrow.push_back(nar);
                const uint32_t none = split ? r0 / kSccMaxRows << 13 | (uint32_t)kSccMaxRows : others;
                for (uint32_t j = 0; j < lines; j++)
                    for (uint32_t l = 0; l < width; l++) {
                        uint32_t e[4];
                        for (uint32_t u = 0; u < 4; u++) {
                            const uint32_t p = l < here ? ig_ptr[slot0 + r0 + l] + 4 * j + u : 0;
                            if (l < here && p < ig_ptr[slot0 + r0 + l + 1]) {
                                const uint32_t x = ig[p], r = (x >> 6) - other;
                                e[u] = (split ? (r / kSccMaxRows) << 13 | r % kSccMaxRows : r) << 9 | (x & 63u) << 3;
                            } else {
                                e[u] = none << 9;
                            }
                        }
                        out.push_back(make_uint4(e[0], e[1], e[2], e[3]));
                    }
            }
        }
    }
    for (size_t i = 0; i < sl.size(); i++)
        if (is_narrow[i]) sl[i].y += (uint32_t)wide.size();
    wide.insert(wide.end(), narrow.begin(), narrow.end());
    ESL_TRY(P->sl.alloc(sl.size()));
    ESL_TRY(P->ell.alloc(wide.size()));
    ESL_CUDA(cudaMemcpyAsync(P->sl.get(), sl.data(), sl.size() * sizeof(uint2), cudaMemcpyHostToDevice, s));
    ESL_CUDA(cudaMemcpyAsync(P->ell.get(), wide.data(), wide.size() * sizeof(uint4), cudaMemcpyHostToDevice, s));
    ESL_CUDA(cudaStreamSynchronize(s));
    return ESL_OK;
}

// The plan built on the host from copies of the net's arrays: the reference the device
// builder (build_plan_device) is checked against, bit for bit.
int build_plan_host(esl_ctx* ctx, const esl_net* net, SweepPlan*& out) {
    out = nullptr;
    cudaStream_t s = ctx->stream;
    const auto t_start = std::chrono::steady_clock::now();
    const size_t N = (size_t)net->N;
    const int n_sccs = net->n_sccs, T = net->T;
    std::vector<int32_t> order(N), offsets(n_sccs + 1), levels(std::max(n_sccs, 1)), term_of(N);
    std::vector<uint32_t> F(N), G(N);
    ESL_CUDA(cudaMemcpyAsync(order.data(), net->order.get(), N * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaMemcpyAsync(offsets.data(), net->offsets.get(), (n_sccs + 1) * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaMemcpyAsync(levels.data(), net->levels.get(), n_sccs * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaMemcpyAsync(term_of.data(), net->term_of.get(), N * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaMemcpyAsync(F.data(), net->F.get(), N * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaMemcpyAsync(G.data(), net->G.get(), N * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaStreamSynchronize(s));

    auto* P = new SweepPlan();
    const int TS = offsets[T];
    P->TS = TS;
    const uint32_t M = (uint32_t)(N - (size_t)TS);
    P->M = M;
    std::vector<uint32_t> slot_of(N, 0xFFFFFFFFu);
    std::vector<uint2> rows;
    rows.reserve(M);
    std::vector<uint4> list;  // SCCs of >= 2 states
    for (int c = T; c < n_sccs;) {
        int c1 = c, mx = 0;
        while (c1 < n_sccs && levels[c1] == levels[c]) {
            mx = std::max(mx, offsets[c1 + 1] - offsets[c1]);
            c1++;
        }
        SwGroup g{};
        g.beg = (uint32_t)rows.size();
        g.max_scc = mx;
        g.term = -1;
        g.kind = mx == 1 ? 0 : (mx <= kSwLocalMax ? 1 : 2);
        for (int par = 0; par < 2; par++) {
            for (int p = offsets[c]; p < offsets[c1]; p++) {
                const uint32_t v = (uint32_t)order[p];
                if ((uint32_t)(__builtin_popcount(v) & 1) != (uint32_t)par) continue;
                slot_of[v] = (uint32_t)rows.size();
                rows.push_back(make_uint2(v, F[v]));
            }
            (par ? g.no : g.ne) = (uint32_t)rows.size() - g.beg - (par ? g.ne : 0);
        }
        g.s0 = (uint32_t)list.size();
        uint32_t er = 0, orr = 0;  // rows of the SCCs before, of either parity
        for (int cc = c; cc < c1; cc++) {
            uint32_t ne = 0, no = 0;
            for (int p = offsets[cc]; p < offsets[cc + 1]; p++)
                (__builtin_popcount((uint32_t)order[p]) & 1 ? no : ne)++;
            if (ne + no >= 2) list.push_back(make_uint4(g.beg + er, ne, g.beg + g.ne + orr, no));
            er += ne;
            orr += no;
        }
        g.ns = (uint32_t)list.size() - g.s0;
        P->max_rows = std::max(P->max_rows, g.ne + g.no);
        P->max_even = std::max(P->max_even, g.ne);
        P->max_odd = std::max(P->max_odd, g.no);
        P->groups.push_back(g);
        c = c1;
    }
    // Predecessor lists, built by host threads in two passes over slot ranges (count,
    // then fill at the prefix offsets) so that the entries come out in slot order.
    std::vector<uint32_t> gend(M);  // end slot of each slot's group
    for (const SwGroup& g : P->groups)
        for (uint32_t sl = g.beg; sl < g.beg + g.ne + g.no; sl++) gend[sl] = g.beg + g.ne + g.no;
    std::vector<uint32_t> gbeg(M);
    for (const SwGroup& g : P->groups)
        for (uint32_t sl = g.beg; sl < g.beg + g.ne + g.no; sl++) gbeg[sl] = g.beg;
    std::vector<uint32_t> ig_ptr(M + 1, 0), og_ptr(M + 1, 0), ig, og;
    const int nth = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    auto for_slots = [&](auto fn) {
        std::vector<std::thread> th;
        const uint32_t per = (M + nth - 1) / nth;
        for (int t = 0; t < nth; t++) {
            const uint32_t a0 = std::min<uint32_t>(M, t * per), a1 = std::min<uint32_t>(M, a0 + per);
            th.emplace_back([=, &fn]() { fn(a0, a1); });
        }
        for (auto& x : th) x.join();
    };
    auto visit = [&](uint32_t sl, auto emit) {
        const uint32_t v = rows[sl].x;
        uint32_t in = G[v];
        while (in) {
            const int i = __builtin_ctz(in);
            in &= in - 1;
            const uint32_t su = slot_of[v ^ (1u << i)];
            if (su == 0xFFFFFFFFu) continue;  // a terminal state has no edge out of its SCC
            // source bit i is the complement of v's
            const uint32_t ri = 2u * (uint32_t)i + (((v >> i) & 1u) ^ 1u);
            emit(su >= gbeg[sl] && su < gend[sl], (su << 6) | ri);
        }
    };
    for_slots([&](uint32_t a0, uint32_t a1) {
        for (uint32_t sl = a0; sl < a1; sl++) {
            uint32_t ci = 0, co = 0;
            visit(sl, [&](bool inside, uint32_t) { (inside ? ci : co)++; });
            ig_ptr[sl + 1] = ci;
            og_ptr[sl + 1] = co;
        }
    });
    for (uint32_t sl = 0; sl < M; sl++) {
        ig_ptr[sl + 1] += ig_ptr[sl];
        og_ptr[sl + 1] += og_ptr[sl];
    }
    ig.resize(ig_ptr[M]);
    og.resize(og_ptr[M]);
    for_slots([&](uint32_t a0, uint32_t a1) {
        for (uint32_t sl = a0; sl < a1; sl++) {
            uint32_t pi = ig_ptr[sl], po = og_ptr[sl];
            visit(sl, [&](bool inside, uint32_t e) {
                if (inside)
                    ig[pi++] = e;
                else
                    og[po++] = e;
            });
        }
    });
    for (SwGroup& g : P->groups) g.nin = ig_ptr[g.beg + g.ne + g.no] - ig_ptr[g.beg];
    std::vector<uint32_t> tp_ptr{0}, tp;
    for (int p = 0; p < TS; p++) {
        const uint32_t v = (uint32_t)order[p];
        uint32_t in = G[v];
        while (in) {
            const int i = __builtin_ctz(in);
            in &= in - 1;
            const uint32_t su = slot_of[v ^ (1u << i)];
            if (su != 0xFFFFFFFFu) tp.push_back((su << 6) | (2u * (uint32_t)i + (((v >> i) & 1u) ^ 1u)));
        }
        tp_ptr.push_back((uint32_t)tp.size());
    }
    int rc = ESL_OK;
    auto up32 = [&](DevBuf<uint32_t>& d, const std::vector<uint32_t>& h) {
        if (rc != ESL_OK) return;
        rc = d.alloc(h.size());
        if (rc == ESL_OK && !h.empty() &&
            cudaMemcpyAsync(d.get(), h.data(), h.size() * 4, cudaMemcpyHostToDevice, s) != cudaSuccess)
            rc = fail(ESL_ERR_CUDA, "sweep plan upload failed");
    };
    if (rc == ESL_OK) rc = P->rows.alloc(rows.size());
    if (rc == ESL_OK && !rows.empty() &&
        cudaMemcpyAsync(P->rows.get(), rows.data(), rows.size() * sizeof(uint2), cudaMemcpyHostToDevice, s) !=
            cudaSuccess)
        rc = fail(ESL_ERR_CUDA, "sweep plan upload failed");
    up32(P->ig_ptr, ig_ptr);
    {
        std::vector<uint4> desc(M);
        for (uint32_t sl = 0; sl < M; sl++)
            desc[sl] = make_uint4(rows[sl].x, rows[sl].y, ig_ptr[sl], ig_ptr[sl + 1] - ig_ptr[sl]);
        if (rc == ESL_OK) rc = P->desc.alloc(std::max<uint32_t>(M, 1));
        if (rc == ESL_OK && M &&
            cudaMemcpyAsync(P->desc.get(), desc.data(), (size_t)M * sizeof(uint4), cudaMemcpyHostToDevice, s) !=
                cudaSuccess)
            rc = fail(ESL_ERR_CUDA, "sweep plan upload failed");
        if (rc == ESL_OK && cudaStreamSynchronize(s) != cudaSuccess) rc = fail(ESL_ERR_CUDA, "sweep plan upload failed");
    }
    up32(P->ig_ent, ig);
    up32(P->og_ptr, og_ptr);
    up32(P->og_ent, og);
    up32(P->tp_ptr, tp_ptr);
    up32(P->tp_ent, tp);
    if (rc == ESL_OK && cudaStreamSynchronize(s) != cudaSuccess) rc = fail(ESL_ERR_CUDA, "sweep plan upload failed");
    if (rc == ESL_OK) rc = finish_scc_list(ctx, P, &list);
    if (rc == ESL_OK) rc = host_lines(ctx, P, ig_ptr, ig);
    if (rc == ESL_OK) rc = build_terminal_plan(order, offsets, T, F, G, s, P->term);
    if (rc != ESL_OK) {
        delete P;
        return rc;
    }
    if (debug_on())
        fprintf(stderr, "[esl-sweep] plan: %zu groups, %u slots, %.1f ms on the host\n", P->groups.size(), P->M,
                std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count());
    out = P;
    return ESL_OK;
}

// ---- the level-sweep plan built on the device --------------------------------------------
// The same plan as build_plan_host, from the net's device arrays by scans and scatters:
// transient positions p' = p - TS (the reordering from the first transient SCC), SCCs
// c' = c - T.  A level group is a run of transient SCCs of one level; a group's slots are
// its positions, even-parity states first (in position order), then odd.
constexpr uint32_t kNoSlot = 0xFFFFFFFFu;

// per transient SCC: group-start flag, size; the SCC's first position is marked
__global__ void k_pl_sccs(int T, int NT, int TS, const int32_t* __restrict__ offsets, const int32_t* __restrict__ levels,
                          uint32_t* __restrict__ gflag, uint32_t* __restrict__ ssize, uint32_t* __restrict__ pos_head) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= NT) return;
    const int cc = T + c;
    gflag[c] = (c == 0 || levels[cc] != levels[cc - 1]) ? 1u : 0u;
    ssize[c] = (uint32_t)(offsets[cc + 1] - offsets[cc]);
    pos_head[offsets[cc] - TS] = 1u;
}

// first SCC of every group (gid_incl: inclusive scan of the group-start flags)
__global__ void k_pl_gfirst(int NT, const uint32_t* __restrict__ gflag, const uint32_t* __restrict__ gid_incl,
                            uint32_t* __restrict__ gfirst) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= NT) return;
    if (gflag[c]) gfirst[gid_incl[c] - 1] = (uint32_t)c;
    if (c == NT - 1) gfirst[gid_incl[c]] = (uint32_t)NT;
}

// even-parity flag per transient position (the scan's input has one more, zero, entry)
__global__ void k_pl_even(uint32_t M, int TS, const int32_t* __restrict__ order, uint32_t* __restrict__ ev) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > M) return;
    ev[p] = p < M ? ((__popc((uint32_t)order[TS + p]) & 1) == 0 ? 1u : 0u) : 0u;
}

// Group g (one warp): info[g] = (first position, even rows, odd rows, kind, largest SCC,
// first SCC, SCCs of >= 2 states).
__global__ void k_pl_groups(int T, int TS, const int32_t* __restrict__ offsets, const uint32_t* __restrict__ gid_incl,
                            int NT, const uint32_t* __restrict__ gfirst, const uint32_t* __restrict__ ssize,
                            const uint32_t* __restrict__ E, uint32_t* __restrict__ info) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int G = (int)gid_incl[NT - 1];
    if (warp >= G) return;
    const uint32_t c0 = gfirst[warp], c1 = gfirst[warp + 1];
    const uint32_t p0 = (uint32_t)(offsets[T + c0] - TS), p1 = (uint32_t)(offsets[T + c1] - TS);
    uint32_t mx = 0, n2 = 0;
    for (uint32_t c = c0 + lane; c < c1; c += 32) {
        const uint32_t sz = ssize[c];
        mx = max(mx, sz);
        if (sz >= 2) n2++;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        n2 += __shfl_xor_sync(0xFFFFFFFFu, n2, o);
    }
    const uint32_t kind = mx == 1 ? 0u : (mx <= (uint32_t)kSwLocalMax ? 1u : 2u);
    if (lane == 0) {
        const uint32_t ne = E[p1] - E[p0];
        uint32_t* o = info + (size_t)warp * 8;
        o[0] = p0;
        o[1] = ne;
        o[2] = (p1 - p0) - ne;
        o[3] = kind;
        o[4] = mx;
        o[5] = c0;
        o[6] = n2;
    }
}

// SCCs of >= 2 states in list order (idx: exclusive scan of their flags)
__global__ void k_pl_scc2(int NT, const uint32_t* __restrict__ ssize, uint32_t* __restrict__ flag) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c > NT) return;
    flag[c] = (c < NT && ssize[c] >= 2) ? 1u : 0u;
}
__global__ void k_pl_scc_list(int NT, int T, int TS, const int32_t* __restrict__ offsets,
                              const uint32_t* __restrict__ gid_incl, const uint32_t* __restrict__ ssize,
                              const uint32_t* __restrict__ E, const uint32_t* __restrict__ info,
                              const uint32_t* __restrict__ idx, uint4* __restrict__ out,
                              uint64_t* __restrict__ key) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= NT || ssize[c] < 2) return;
    const uint32_t* in = info + (size_t)(gid_incl[c] - 1) * 8;
    const uint32_t p0 = in[0], ne = in[1], cs = (uint32_t)(offsets[T + c] - TS), ce = cs + ssize[c];
    const uint32_t er = E[cs] - E[p0], se = E[ce] - E[cs];
    out[idx[c]] = make_uint4(p0 + er, se, p0 + ne + (cs - p0) - er, ssize[c] - se);
    key[idx[c]] = scc_sort_key(gid_incl[c] - 1, se, ssize[c] - se);
}

// slot of every transient position: rows, slot_of (by state), group of each slot
__global__ void k_pl_slots(uint32_t M, int TS, const int32_t* __restrict__ order, const uint32_t* __restrict__ F,
                           const uint32_t* __restrict__ E, const uint32_t* __restrict__ sccpos,
                           const uint32_t* __restrict__ gid_incl, const uint32_t* __restrict__ info,
                           uint2* __restrict__ rows, uint32_t* __restrict__ slot_of, uint32_t* __restrict__ slot_grp) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= M) return;
    const uint32_t c = sccpos[p] - 1;
    const uint32_t g = gid_incl[c] - 1;
    const uint32_t* in = info + (size_t)g * 8;
    const uint32_t p0 = in[0], ne = in[1];
    const uint32_t v = (uint32_t)order[TS + p];
    const bool even = (__popc(v) & 1) == 0;
    const uint32_t er = E[p] - E[p0];
    const uint32_t slot = p0 + (even ? er : ne + (p - p0) - er);
    rows[slot] = make_uint2(v, F[v]);
    slot_of[v] = slot;
    slot_grp[slot] = g;
}

// predecessor entries of a slot: (slot << 6) | rate index, in bit order; COUNT: only
// count those inside / outside the slot's group
template <bool COUNT>
__global__ void k_pl_preds(uint32_t M, const uint2* __restrict__ rows, const uint32_t* __restrict__ G,
                           const uint32_t* __restrict__ slot_of, const uint32_t* __restrict__ slot_grp,
                           const uint32_t* __restrict__ info, uint32_t* __restrict__ cnt_in, uint32_t* __restrict__ cnt_out,
                           const uint32_t* __restrict__ ig_ptr, const uint32_t* __restrict__ og_ptr,
                           uint32_t* __restrict__ ig, uint32_t* __restrict__ og, uint4* __restrict__ desc) {
    const uint32_t sl = blockIdx.x * blockDim.x + threadIdx.x;
    if (sl >= M) return;
    const uint2 row = rows[sl];
    const uint32_t v = row.x;
    const uint32_t* in = info + (size_t)slot_grp[sl] * 8;
    const uint32_t gb = in[0], ge = in[0] + in[1] + in[2];
    uint32_t ci = 0, co = 0;
    const uint32_t pi0 = COUNT ? 0u : ig_ptr[sl], po0 = COUNT ? 0u : og_ptr[sl];
    uint32_t g = G[v];
    while (g) {
        const int i = __ffs(g) - 1;
        g &= g - 1;
        const uint32_t su = slot_of[v ^ (1u << i)];
        if (su == kNoSlot) continue;  // a terminal state has no edge out of its SCC
        const bool inside = su >= gb && su < ge;
        if (!COUNT) {
            const uint32_t e = (su << kEntShift) | (2u * (uint32_t)i + (((v >> i) & 1u) ^ 1u));
            if (inside)
                ig[pi0 + ci] = e;
            else
                og[po0 + co] = e;
        }
        (inside ? ci : co)++;
    }
    if (COUNT) {
        cnt_in[sl] = ci;
        cnt_out[sl] = co;
    } else {
        desc[sl] = make_uint4(v, row.y, pi0, ci);
    }
}

// transient predecessors of the terminal positions
template <bool COUNT>
__global__ void k_pl_tpreds(int TS, const int32_t* __restrict__ order, const uint32_t* __restrict__ G,
                            const uint32_t* __restrict__ slot_of, uint32_t* __restrict__ cnt,
                            const uint32_t* __restrict__ tp_ptr, uint32_t* __restrict__ tp) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= TS) return;
    const uint32_t v = (uint32_t)order[p];
    uint32_t g = G[v], c = 0;
    const uint32_t b = COUNT ? 0u : tp_ptr[p];
    while (g) {
        const int i = __ffs(g) - 1;
        g &= g - 1;
        const uint32_t su = slot_of[v ^ (1u << i)];
        if (su == kNoSlot) continue;
        if (!COUNT) tp[b + c] = (su << kEntShift) | (2u * (uint32_t)i + (((v >> i) & 1u) ^ 1u));
        c++;
    }
    if (COUNT) cnt[p] = c;
}

// per group: in-group predecessor entries
__global__ void k_pl_gtail(int G, const uint32_t* __restrict__ info, const uint32_t* __restrict__ ig_ptr,
                           uint32_t* __restrict__ gtail) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const uint32_t* in = info + (size_t)g * 8;
    const uint32_t b = in[0], e = in[0] + in[1] + in[2];
    gtail[g] = ig_ptr[e] - ig_ptr[b];
}

// exclusive scan of n + 1 counts (the last one 0) into out[0 .. n], on the stream
int scan_excl(DevBuf<uint8_t>& tmp, const uint32_t* in, uint32_t* out, uint32_t n1, cudaStream_t s) {
    size_t bytes = 0;
    ESL_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, (int64_t)n1, s));
    if (tmp.n < bytes) ESL_TRY(tmp.alloc(bytes));
    ESL_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), bytes, in, out, (int64_t)n1, s));
    return ESL_OK;
}
int scan_incl(DevBuf<uint8_t>& tmp, const uint32_t* in, uint32_t* out, uint32_t n, cudaStream_t s) {
    size_t bytes = 0;
    ESL_CUDA(cub::DeviceScan::InclusiveSum(nullptr, bytes, in, out, (int64_t)n, s));
    if (tmp.n < bytes) ESL_TRY(tmp.alloc(bytes));
    ESL_CUDA(cub::DeviceScan::InclusiveSum(tmp.get(), bytes, in, out, (int64_t)n, s));
    return ESL_OK;
}

inline unsigned nblk(uint64_t n) { return (unsigned)std::max<uint64_t>(1, (n + 255) / 256); }

int build_plan_device(esl_ctx* ctx, const esl_net* net, SweepPlan*& out) {
    out = nullptr;
    cudaStream_t s = ctx->stream;
    const auto t_start = std::chrono::steady_clock::now();
    const size_t N = (size_t)net->N;
    const int n_sccs = net->n_sccs, T = net->T, TS = net->term_states;
    const int NT = n_sccs - T;
    const uint32_t M = (uint32_t)(N - (size_t)TS);
    std::unique_ptr<SweepPlan> P(new SweepPlan());
    P->TS = TS;
    P->M = M;
    DevBuf<uint8_t> tmp;
    DevBuf<uint32_t> slot_of;
    ESL_TRY(slot_of.alloc(N));
    ESL_CUDA(cudaMemsetAsync(slot_of.get(), 0xFF, N * 4, s));
    const int32_t* order = net->order.get();
    const int32_t* offsets = net->offsets.get();
    std::vector<uint32_t> h_info, h_tail;
    uint32_t G = 0, tot[3] = {0, 0, 0};
    if (M > 0) {
        DevBuf<uint32_t> gflag, gid, ssize, gfirst, info, pos_head, sccpos, ev, E, slot_grp, cnt_in, cnt_out,
            gtail;
        ESL_TRY(gflag.alloc(NT));
        ESL_TRY(gid.alloc(NT));
        ESL_TRY(ssize.alloc(NT));
        ESL_TRY(gfirst.alloc(NT + 1));
        ESL_TRY(info.alloc((size_t)NT * 8));
        ESL_TRY(pos_head.alloc(M));
        ESL_TRY(sccpos.alloc(M));
        ESL_TRY(ev.alloc((size_t)M + 1));
        ESL_TRY(E.alloc((size_t)M + 1));
        ESL_TRY(slot_grp.alloc(M));
        ESL_TRY(cnt_in.alloc((size_t)M + 1));
        ESL_TRY(cnt_out.alloc((size_t)M + 1));
        ESL_CUDA(cudaMemsetAsync(pos_head.get(), 0, (size_t)M * 4, s));
        ESL_COUNT_LAUNCH();
        k_pl_sccs<<<nblk(NT), 256, 0, s>>>(T, NT, TS, offsets, net->levels.get(), gflag.get(), ssize.get(),
                                           pos_head.get());
        ESL_TRY(scan_incl(tmp, gflag.get(), gid.get(), (uint32_t)NT, s));
        ESL_COUNT_LAUNCH();
        k_pl_gfirst<<<nblk(NT), 256, 0, s>>>(NT, gflag.get(), gid.get(), gfirst.get());
        ESL_COUNT_LAUNCH();
        k_pl_even<<<nblk((uint64_t)M + 1), 256, 0, s>>>(M, TS, order, ev.get());
        ESL_TRY(scan_excl(tmp, ev.get(), E.get(), M + 1, s));
        ESL_TRY(scan_incl(tmp, pos_head.get(), sccpos.get(), M, s));
        ESL_COUNT_LAUNCH();
        k_pl_groups<<<nblk((uint64_t)NT * 32), 256, 0, s>>>(T, TS, offsets, gid.get(), NT, gfirst.get(), ssize.get(),
                                                            E.get(), info.get());
        ESL_CUDA(cudaGetLastError());
        ESL_TRY(P->rows.alloc(M));
        ESL_COUNT_LAUNCH();
        k_pl_slots<<<nblk(M), 256, 0, s>>>(M, TS, order, net->F.get(), E.get(), sccpos.get(), gid.get(), info.get(),
                                           P->rows.get(), slot_of.get(), slot_grp.get());
        ESL_COUNT_LAUNCH();
        k_pl_preds<true><<<nblk(M), 256, 0, s>>>(M, P->rows.get(), net->G.get(), slot_of.get(), slot_grp.get(),
                                                 info.get(), cnt_in.get(), cnt_out.get(), nullptr, nullptr, nullptr,
                                                 nullptr, nullptr);
        ESL_CUDA(cudaMemsetAsync(cnt_in.get() + M, 0, 4, s));
        ESL_CUDA(cudaMemsetAsync(cnt_out.get() + M, 0, 4, s));
        ESL_TRY(P->ig_ptr.alloc((size_t)M + 1));
        ESL_TRY(P->og_ptr.alloc((size_t)M + 1));
        ESL_TRY(scan_excl(tmp, cnt_in.get(), P->ig_ptr.get(), M + 1, s));
        ESL_TRY(scan_excl(tmp, cnt_out.get(), P->og_ptr.get(), M + 1, s));
        ESL_CUDA(cudaGetLastError());
        // the group count and the group table
        ESL_CUDA(cudaMemcpyAsync(&G, gid.get() + NT - 1, 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        ESL_TRY(gtail.alloc(G));
        ESL_COUNT_LAUNCH();
        k_pl_gtail<<<nblk(G), 256, 0, s>>>((int)G, info.get(), P->ig_ptr.get(), gtail.get());
        ESL_CUDA(cudaGetLastError());
        h_info.resize((size_t)G * 8);
        h_tail.resize(G);
        ESL_CUDA(cudaMemcpyAsync(h_info.data(), info.get(), (size_t)G * 32, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(h_tail.data(), gtail.get(), (size_t)G * 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(&tot[0], P->ig_ptr.get() + M, 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(&tot[1], P->og_ptr.get() + M, 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        // the list of SCCs of >= 2 states
        uint32_t n2 = 0;
        for (uint32_t g = 0; g < G; g++) n2 += h_info[(size_t)g * 8 + 6];
        if (n2 > 0) {
            ESL_TRY(P->scc.alloc(n2));
            ESL_TRY(P->scc_key.alloc(n2));
            DevBuf<uint32_t> flag, sidx;
            ESL_TRY(flag.alloc((size_t)NT + 1));
            ESL_TRY(sidx.alloc((size_t)NT + 1));
            ESL_COUNT_LAUNCH();
            k_pl_scc2<<<nblk((uint64_t)NT + 1), 256, 0, s>>>(NT, ssize.get(), flag.get());
            ESL_TRY(scan_excl(tmp, flag.get(), sidx.get(), (uint32_t)NT + 1, s));
            ESL_COUNT_LAUNCH();
            k_pl_scc_list<<<nblk(NT), 256, 0, s>>>(NT, T, TS, offsets, gid.get(), ssize.get(), E.get(), info.get(),
                                                   sidx.get(), P->scc.get(), P->scc_key.get());
            ESL_CUDA(cudaGetLastError());
        }
        ESL_TRY(P->ig_ent.alloc(std::max<uint32_t>(tot[0], 1)));
        ESL_TRY(P->og_ent.alloc(std::max<uint32_t>(tot[1], 1)));
        ESL_TRY(P->desc.alloc(M));
        ESL_COUNT_LAUNCH();
        k_pl_preds<false><<<nblk(M), 256, 0, s>>>(M, P->rows.get(), net->G.get(), slot_of.get(), slot_grp.get(),
                                                  info.get(), nullptr, nullptr, P->ig_ptr.get(), P->og_ptr.get(),
                                                  P->ig_ent.get(), P->og_ent.get(), P->desc.get());
        ESL_CUDA(cudaGetLastError());
    } else {
        ESL_TRY(P->rows.alloc(1));
        ESL_TRY(P->desc.alloc(1));
        ESL_TRY(P->ig_ptr.alloc(1));
        ESL_TRY(P->og_ptr.alloc(1));
        ESL_TRY(P->ig_ent.alloc(1));
        ESL_TRY(P->og_ent.alloc(1));
        ESL_CUDA(cudaMemsetAsync(P->ig_ptr.get(), 0, 4, s));
        ESL_CUDA(cudaMemsetAsync(P->og_ptr.get(), 0, 4, s));
    }
    // transient predecessors of the terminal positions
    {
        DevBuf<uint32_t> cnt;
        ESL_TRY(cnt.alloc((size_t)TS + 1));
        ESL_TRY(P->tp_ptr.alloc((size_t)TS + 1));
        ESL_CUDA(cudaMemsetAsync(cnt.get(), 0, ((size_t)TS + 1) * 4, s));
        if (TS > 0) {
            ESL_COUNT_LAUNCH();
            k_pl_tpreds<true><<<nblk(TS), 256, 0, s>>>(TS, order, net->G.get(), slot_of.get(), cnt.get(), nullptr,
                                                       nullptr);
        }
        ESL_TRY(scan_excl(tmp, cnt.get(), P->tp_ptr.get(), (uint32_t)TS + 1, s));
        ESL_CUDA(cudaMemcpyAsync(&tot[2], P->tp_ptr.get() + TS, 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        ESL_TRY(P->tp_ent.alloc(std::max<uint32_t>(tot[2], 1)));
        if (TS > 0) {
            ESL_COUNT_LAUNCH();
            k_pl_tpreds<false><<<nblk(TS), 256, 0, s>>>(TS, order, net->G.get(), slot_of.get(), nullptr,
                                                        P->tp_ptr.get(), P->tp_ent.get());
        }
        ESL_CUDA(cudaGetLastError());
    }
    // the group table on the host
    uint32_t s0 = 0;
    for (uint32_t g = 0; g < G; g++) {
        const uint32_t* in = &h_info[(size_t)g * 8];
        SwGroup gr{};
        gr.beg = in[0];
        gr.ne = in[1];
        gr.no = in[2];
        gr.kind = (int)in[3];
        gr.max_scc = (int)in[4];
        gr.term = -1;
        gr.nin = h_tail[g];
        gr.s0 = s0;
        gr.ns = in[6];
        s0 += gr.ns;
        P->max_rows = std::max(P->max_rows, gr.ne + gr.no);
        P->max_even = std::max(P->max_even, gr.ne);
        P->max_odd = std::max(P->max_odd, gr.no);
        P->groups.push_back(gr);
    }
    ESL_CUDA(cudaStreamSynchronize(s));
    // the terminal plan, for networks with terminal SCCs above kDenseTerminalMax states
    if (net->max_terminal > kDenseTerminalMax) {
        std::vector<int32_t> h_order(TS), h_off(T + 1);
        std::vector<uint32_t> hF(N), hG(N);
        ESL_CUDA(cudaMemcpyAsync(h_order.data(), order, (size_t)TS * 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(h_off.data(), offsets, (size_t)(T + 1) * 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(hF.data(), net->F.get(), N * 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(hG.data(), net->G.get(), N * 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        ESL_TRY(build_terminal_plan(h_order, h_off, T, hF, hG, s, P->term));
    }
    if (debug_on())
        fprintf(stderr, "[esl-sweep] plan: %zu groups, %u slots, %.1f ms on the device\n", P->groups.size(), P->M,
                std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count());
    out = P.release();
    return ESL_OK;
}

// Most rows of one parity of an SCC
__host__ __device__ inline uint32_t scc_rows(const uint4& c) { return c.y > c.w ? c.y : c.w; }

// Slices of SCC j (see SweepPlan::sl): source[slice] = (first slot, rows | 64 and the cluster
// rank << 7 for an SCC split over a cluster | 512 for a narrow one, first slot of the other
// parity, its rows)
__global__ void k_pl_slices(uint32_t count, const uint4* __restrict__ scc, const uint2* __restrict__ scc_sl,
                            uint4* __restrict__ source) {
    const uint32_t j = blockIdx.x;
    if (j >= count) return;
    const uint4 c = scc[j];
    const uint2 f = scc_sl[j];
    if (f.x == kNoSlot) return;  // not solved by a CTA or a cluster
    const bool split = max(c.y, c.w) > (uint32_t)kSccMaxRows;
    const uint32_t narrow = scc_narrow(c.y, c.w) ? 512u : 0u;
    for (uint32_t r = threadIdx.x * 32; r < c.y; r += blockDim.x * 32)
        source[f.x + r / 32] =
            make_uint4(c.x + r, min(32u, c.y - r) | (split ? 64u | r / kSccMaxRows << 7 : 0u) | narrow, c.z, c.w);
    for (uint32_t r = threadIdx.x * 32; r < c.w; r += blockDim.x * 32)
        source[f.y + r / 32] =
            make_uint4(c.z + r, min(32u, c.w - r) | (split ? 64u | r / kSccMaxRows << 7 : 0u) | narrow, c.x, c.y);
}

// One warp per slice.  FILL false: its lines (four entries a line, the most of a row) in
// size[w], or for a narrow SCC its places in ell in size[slices + w] (the other one 0); true:
// the lines, from the exclusive sums of these.
template <bool FILL>
__global__ void k_pl_ell(uint32_t slices, const uint4* __restrict__ source, const uint32_t* __restrict__ ig_ptr,
                         const uint32_t* __restrict__ ig_ent, uint32_t* __restrict__ size,
                         const uint32_t* __restrict__ off, uint2* __restrict__ sl, uint4* __restrict__ ell) {
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= slices) return;
    const uint4 src = source[w];
    const bool narrow = src.y & 512u;
    const uint32_t rows = src.y & 63u, width = narrow ? rows : 32u;
    const bool row = lane < rows;
    const uint32_t p = row ? ig_ptr[src.x + lane] : 0u;
    const uint32_t cnt = row ? ig_ptr[src.x + lane + 1] - p : 0u;
    const uint32_t lines = (__reduce_max_sync(0xFFFFFFFFu, cnt) + 3) / 4;
    if (!FILL) {
        if (lane == 0) {
            size[w] = narrow ? 0u : lines;
            size[slices + w] = narrow ? lines * width : 0u;
        }
        return;
    }
    // (the narrow slices' sums go on from the lines of the others: off[slices])
    const uint32_t first = narrow ? off[slices] * 31 + off[slices + w] : off[w];
    uint4* out = ell + (narrow ? (size_t)first : (size_t)first * 32);
    if (lane == 0) sl[w] = make_uint2(lines, first);
    if (lane >= width) return;
    const bool split = src.y & 64u;  // (see kSccCluster)
    const uint32_t none = split ? (src.y >> 7 & 3u) << 13 | (uint32_t)kSccMaxRows : src.w;
    for (uint32_t j = 0; j < lines; j++) {
        uint32_t e[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            e[u] = none << 9;
            if (4 * j + u < cnt) {
                const uint32_t x = ig_ent[p + 4 * j + u], r = ent_slot(x) - src.z;
                e[u] = (split ? (r / kSccMaxRows) << 13 | r % kSccMaxRows : r) << 9 | (uint32_t)ent_rate(x) << 3;
            }
        }
        out[(size_t)j * width + lane] = make_uint4(e[0], e[1], e[2], e[3]);
    }
}

// slices of `rows` rows of one parity of an SCC (0: neither a CTA nor a cluster solves it)
__host__ __device__ inline uint32_t scc_slices(const uint4& c, uint32_t rows) {
    return scc_rows(c) > kSccClusterRows ? 0u : (rows + 31) / 32;
}

// The sorted list: SCC i = in[place[i]].  head[i]: it begins a shape of its group; slices[i]:
// its slices (both with one more, zero, entry for the scans)
__global__ void k_pl_scc_sorted(uint32_t count, const uint4* __restrict__ in, const uint64_t* __restrict__ key,
                                const int32_t* __restrict__ place, uint4* __restrict__ out, uint32_t* __restrict__ head,
                                uint32_t* __restrict__ slices) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > count) return;
    if (i == count) {
        head[i] = slices[i] = 0;
        return;
    }
    const uint4 c = in[place[i]], b = in[place[i ? i - 1 : 0]];
    out[i] = c;
    head[i] = (i == 0 || key[i] >> 38 != key[i - 1] >> 38 || c.y != b.y || c.w != b.w) ? 1u : 0u;
    slices[i] = scc_slices(c, c.y) + scc_slices(c, c.w);
}
// scc_sl, and of every shape's first SCC (its place, even rows, odd rows, group)
__global__ void k_pl_scc_shapes(uint32_t count, const uint4* __restrict__ scc, const uint64_t* __restrict__ key,
                                const uint32_t* __restrict__ head, const uint32_t* __restrict__ shape,
                                const uint32_t* __restrict__ slice, uint2* __restrict__ scc_sl,
                                uint4* __restrict__ shapes) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const uint4 c = scc[i];
    const bool kept = scc_rows(c) <= kSccClusterRows;
    scc_sl[i] = kept ? make_uint2(slice[i], slice[i] + scc_slices(c, c.y)) : make_uint2(kNoSlot, kNoSlot);
    if (head[i]) shapes[shape[i]] = make_uint4(i, c.y, c.w, (uint32_t)(key[i] >> 38));
}

// Sorts the SCC list (scc_sort_key), lists its shapes and lays out the predecessor lines of the
// SCCs that a CTA or a cluster solves.  Any SCC of at most kSccMaxRows rows of either parity
// fits a CTA's shared memory at one system.  A short list is sorted on the host (`list`, or
// read back where that is null), a long one on the device: a plan with 2,047, 8,191 and 32,767
// SCCs takes 380, 530 and 1,120 us with the host's sort, 420, 515 and 555 with the device's.
static_assert((2 * (kSccMaxRows + 1) + 2 * 26 + 6 * (kSccThreadsBig / 32) + 5 * kSccMaxRows) * 8 <= (int)kSccMaxSmem - 256,
              "k_sw_scc's arrays");
constexpr uint32_t kSccHostSort = 4096;
int finish_scc_list(esl_ctx* ctx, SweepPlan* P, const std::vector<uint4>* list) {
    cudaStream_t s = ctx->stream;
    uint32_t count = 0, slices = 0;
    for (const SwGroup& g : P->groups) count += g.ns;
    DevBuf<uint8_t> tmp;
    std::vector<uint4> shapes;  // (first SCC, even rows, odd rows, group)
    if (count > 0) ESL_TRY(P->scc_sl.alloc(count));
    if (count > 0 && (list || count <= kSccHostSort)) {
        std::vector<uint4> h(count);
        if (list) {
            h = *list;
            ESL_TRY(P->scc.alloc(count));
        } else {
            ESL_CUDA(cudaMemcpyAsync(h.data(), P->scc.get(), (size_t)count * sizeof(uint4), cudaMemcpyDeviceToHost, s));
            ESL_CUDA(cudaStreamSynchronize(s));
        }
        std::vector<uint2> first(count, make_uint2(kNoSlot, kNoSlot));
        for (uint32_t gi = 0; gi < P->groups.size(); gi++) {
            const SwGroup& g = P->groups[gi];
            std::stable_sort(h.begin() + g.s0, h.begin() + g.s0 + g.ns, [](const uint4& x, const uint4& y) {
                return scc_sort_key(0, x.y, x.w) < scc_sort_key(0, y.y, y.w);
            });
            for (uint32_t j = g.s0; j < g.s0 + g.ns; j++) {
                const uint4& c = h[j];
                if (j == g.s0 || c.y != h[j - 1].y || c.w != h[j - 1].w) shapes.push_back(make_uint4(j, c.y, c.w, gi));
                if (scc_rows(c) > kSccClusterRows) continue;
                first[j].x = slices;
                first[j].y = slices + scc_slices(c, c.y);
                slices = first[j].y + scc_slices(c, c.w);
            }
        }
        ESL_CUDA(cudaMemcpyAsync(P->scc.get(), h.data(), (size_t)count * sizeof(uint4), cudaMemcpyHostToDevice, s));
        ESL_CUDA(cudaMemcpyAsync(P->scc_sl.get(), first.data(), (size_t)count * sizeof(uint2), cudaMemcpyHostToDevice, s));
    } else if (count > 0) {
        DevBuf<uint4> sorted, d_shapes;
        DevBuf<uint64_t> key;
        DevBuf<int32_t> place0, place;
        DevBuf<uint32_t> head, shape, nsl, slice;
        ESL_TRY(sorted.alloc(count));
        ESL_TRY(key.alloc(count));
        ESL_TRY(place0.alloc(count));
        ESL_TRY(place.alloc(count));
        ESL_COUNT_LAUNCH();
        k_sw_iota<<<nblk(count), 256, 0, s>>>((int)count, place0.get());
        ESL_TRY(sort_pairs(P->scc_key.get(), key.get(), place0.get(), place.get(), count, tmp, s));
        for (DevBuf<uint32_t>* b : {&head, &shape, &nsl, &slice}) ESL_TRY(b->alloc((size_t)count + 1));
        ESL_COUNT_LAUNCH();
        k_pl_scc_sorted<<<nblk((uint64_t)count + 1), 256, 0, s>>>(count, P->scc.get(), key.get(), place.get(), sorted.get(),
                                                                  head.get(), nsl.get());
        ESL_TRY(scan_excl(tmp, head.get(), shape.get(), count + 1, s));
        ESL_TRY(scan_excl(tmp, nsl.get(), slice.get(), count + 1, s));
        uint32_t n_shapes = 0;
        ESL_CUDA(cudaMemcpyAsync(&n_shapes, shape.get() + count, 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(&slices, slice.get() + count, 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        ESL_TRY(d_shapes.alloc(n_shapes));
        ESL_COUNT_LAUNCH();
        k_pl_scc_shapes<<<nblk(count), 256, 0, s>>>(count, sorted.get(), key.get(), head.get(), shape.get(), slice.get(),
                                                    P->scc_sl.get(), d_shapes.get());
        ESL_CUDA(cudaGetLastError());
        shapes.resize(n_shapes);
        ESL_CUDA(cudaMemcpyAsync(shapes.data(), d_shapes.get(), (size_t)n_shapes * sizeof(uint4), cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        std::swap(P->scc.p, sorted.p);
        std::swap(P->scc.n, sorted.n);
    }
    P->scc_key.release();
    for (SwGroup& g : P->groups) g.singles = g.ne + g.no;
    for (size_t j = 0; j < shapes.size(); j++) {
        const uint4& x = shapes[j];
        SwGroup& g = P->groups[x.w];
        const uint32_t next = j + 1 < shapes.size() ? shapes[j + 1].x : count, many = next - x.x, rows = std::max(x.y, x.z);
        if (g.nsh++ == 0) {
            g.sh0 = (uint32_t)P->shapes.size();
            g.l0 = (uint32_t)P->large.size();
            g.most = rows;
        }
        P->shapes.push_back({x.y, x.z, many});
        g.singles -= (x.y + x.z) * many;
        if (rows > kSccClusterRows) {
            g.nlarge += many;
            P->large.resize(P->large.size() + many);
            ESL_CUDA(cudaMemcpyAsync(P->large.data() + P->large.size() - many, P->scc.get() + x.x,
                                     (size_t)many * sizeof(uint4), cudaMemcpyDeviceToHost, s));
            ESL_CUDA(cudaStreamSynchronize(s));
        }
    }
    for (SwGroup& g : P->groups) {
        g.resident = g.nlarge == 0;
        g.split = g.most > (uint32_t)kSccMaxRows;
    }
    // (the uploads above read vectors of this function)
    if (slices == 0) {
        ESL_CUDA(cudaStreamSynchronize(s));
        return ESL_OK;
    }
    DevBuf<uint4> source;
    DevBuf<uint32_t> size, off;
    ESL_TRY(source.alloc(slices));
    ESL_TRY(size.alloc(2 * (size_t)slices + 1));
    ESL_TRY(off.alloc(2 * (size_t)slices + 1));
    ESL_TRY(P->sl.alloc(slices));
    uint32_t total[2] = {0, 0};  // lines of 32 rows, and these and the places of narrow ones
    ESL_COUNT_LAUNCH();
    k_pl_slices<<<count, 32, 0, s>>>(count, P->scc.get(), P->scc_sl.get(), source.get());
    ESL_CUDA(cudaMemsetAsync(size.get() + 2 * (size_t)slices, 0, 4, s));
    ESL_COUNT_LAUNCH();
    k_pl_ell<false><<<nblk((uint64_t)slices * 32), 256, 0, s>>>(slices, source.get(), P->ig_ptr.get(), P->ig_ent.get(),
                                                                size.get(), nullptr, nullptr, nullptr);
    ESL_TRY(scan_excl(tmp, size.get(), off.get(), 2 * slices + 1, s));
    ESL_CUDA(cudaMemcpyAsync(&total[0], off.get() + slices, 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaMemcpyAsync(&total[1], off.get() + 2 * (size_t)slices, 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaStreamSynchronize(s));
    ESL_TRY(P->ell.alloc((size_t)total[0] * 31 + total[1]));
    ESL_COUNT_LAUNCH();
    k_pl_ell<true><<<nblk((uint64_t)slices * 32), 256, 0, s>>>(slices, source.get(), P->ig_ptr.get(), P->ig_ent.get(),
                                                               size.get(), off.get(), P->sl.get(), P->ell.get());
    ESL_CUDA(cudaGetLastError());
    ESL_CUDA(cudaStreamSynchronize(s));
    return ESL_OK;
}

// the SCC list of a plan whose groups are one SCC each
std::vector<uint4> one_scc_per_group(const SweepPlan* P) {
    std::vector<uint4> list;
    for (const SwGroup& g : P->groups) list.push_back(make_uint4(g.beg, g.ne, g.beg + g.ne, g.no));
    return list;
}

int build_plan(esl_ctx* ctx, const esl_net* net, SweepPlan*& out) {
    // one builder at a time, so that threads solving the same network share one plan
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (net->sweep) {
        out = static_cast<SweepPlan*>(net->sweep);
        return ESL_OK;
    }
    SweepPlan* P = nullptr;
    ESL_TRY(build_plan_device(ctx, net, P));
    int rc = finish_scc_list(ctx, P, nullptr);
    if (rc == ESL_OK && P->term) {
        const std::vector<uint4> list = one_scc_per_group(P->term);
        rc = finish_scc_list(ctx, P->term, &list);
    }
    if (rc != ESL_OK) {
        delete P;
        return rc;
    }
    esl_net* mnet = const_cast<esl_net*>(net);
    mnet->sweep = P;
    mnet->sweep_free = free_plan_sweep;
    out = P;
    return ESL_OK;
}

// The transient part of a small network as one group, even-parity states first: what the
// whole-system form (ESL_METHOD_FP64) and the absorption matrix solve.  back: the transposed
// system, whose rows gather from their successors at the row's own rates.
int build_whole_plan(esl_ctx* ctx, const esl_net* net, bool back, SweepPlan*& out) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    esl_net* mnet = const_cast<esl_net*>(net);
    void*& kept = mnet->whole[back];
    if (kept) {
        out = static_cast<SweepPlan*>(kept);
        return ESL_OK;
    }
    cudaStream_t s = ctx->stream;
    const size_t N = (size_t)net->N;
    const int TS = net->term_states;
    std::vector<int32_t> order(N), term_of(N);
    std::vector<uint32_t> F(N), G(N);
    ESL_CUDA(cudaMemcpyAsync(order.data(), net->order.get(), N * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaMemcpyAsync(term_of.data(), net->term_of.get(), N * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaMemcpyAsync(F.data(), net->F.get(), N * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaMemcpyAsync(G.data(), net->G.get(), N * 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaStreamSynchronize(s));
    std::unique_ptr<SweepPlan> P(new SweepPlan());
    const uint32_t M = (uint32_t)(N - (size_t)TS);
    P->M = M;
    P->TS = back ? 0 : TS;
    SwGroup g{};
    g.kind = 2;
    g.term = -1;
    g.max_scc = (int)M;
    std::vector<uint2> rows;
    std::vector<uint32_t> slot_of(N, kNoSlot), rev;
    for (int par = 0; par < 2; par++)
        for (uint32_t v = 0; v < N; v++)
            if (term_of[v] < 0 && (__builtin_popcount(v) & 1) == par) {
                slot_of[v] = (uint32_t)rows.size();
                rows.push_back(make_uint2(v, F[v]));
                (par ? g.no : g.ne)++;
            }
    g.ns = 1;
    P->max_rows = M;
    P->max_even = g.ne;
    P->max_odd = g.no;
    std::vector<uint32_t> ig_ptr(M + 1, 0), og_ptr(M + 1, 0), ig, tp_ptr{0}, tp;
    std::vector<uint4> desc(M);
    auto entries = [&](uint32_t v, std::vector<uint32_t>& e) {
        for (uint32_t m = back ? F[v] : G[v]; m; m &= m - 1) {
            const uint32_t i = (uint32_t)__builtin_ctz(m), su = slot_of[v ^ (1u << i)];
            if (su == kNoSlot) continue;
            // the rate of the edge's source: the neighbour's, or (back) the row's own
            const uint32_t b = ((v >> i) & 1u) ^ (back ? 0u : 1u);
            e.push_back((su << kEntShift) | (2u * i + b));
        }
    };
    for (uint32_t sl = 0; sl < M; sl++) {
        const uint32_t v = rows[sl].x;
        entries(v, ig);
        ig_ptr[sl + 1] = (uint32_t)ig.size();
        desc[sl] = make_uint4(v, F[v], ig_ptr[sl], ig_ptr[sl + 1] - ig_ptr[sl]);
        if (back) rev.push_back(G[v]);
    }
    g.nin = ig.size();
    for (int p = 0; p < P->TS; p++) {
        entries((uint32_t)order[p], tp);
        tp_ptr.push_back((uint32_t)tp.size());
    }
    P->groups.push_back(g);
    int rc = ESL_OK;
    auto up = [&](auto& d, const auto& h) {
        if (rc != ESL_OK) return;
        rc = d.alloc(std::max<size_t>(h.size(), 1));
        if (rc == ESL_OK && !h.empty() &&
            cudaMemcpyAsync(d.get(), h.data(), h.size() * sizeof(h[0]), cudaMemcpyHostToDevice, s) != cudaSuccess)
            rc = fail(ESL_ERR_CUDA, "plan upload failed");
    };
    up(P->rows, rows);
    up(P->desc, desc);
    up(P->ig_ptr, ig_ptr);
    up(P->ig_ent, ig);
    up(P->og_ptr, og_ptr);
    up(P->og_ent, std::vector<uint32_t>{});
    up(P->tp_ptr, tp_ptr);
    up(P->tp_ent, tp);
    if (back) up(P->rev, rev);
    if (rc == ESL_OK && cudaStreamSynchronize(s) != cudaSuccess) rc = fail(ESL_ERR_CUDA, "plan upload failed");
    const std::vector<uint4> list = one_scc_per_group(P.get());
    if (rc == ESL_OK) rc = finish_scc_list(ctx, P.get(), &list);
    if (rc != ESL_OK) return rc;
    mnet->sweep_free = free_plan_sweep;
    out = P.get();
    kept = P.release();
    return ESL_OK;
}

// L[t][v] of the backward plan's solution (rows: Z[slot][t]) and of the terminal states
__global__ void k_sw_scatter_L(uint32_t M, int Kp, size_t N, const uint2* __restrict__ rows, const double* __restrict__ Z,
                               const int32_t* __restrict__ term_of, double* __restrict__ L) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int t = blockIdx.y;
    if (i < N && term_of[i] >= 0) L[(size_t)t * N + i] = term_of[i] == t ? 1.0 : 0.0;
    if (i < M) L[(size_t)t * N + rows[i].x] = Z[i * Kp + t];
}
// b[t][v] = rate of v's edges into terminal SCC t, for transient v (0 elsewhere)
__global__ void k_sw_back_rhs(int n, size_t N, const uint32_t* __restrict__ F, const int32_t* __restrict__ term_of,
                              const double* __restrict__ rates, double* __restrict__ b) {
    const size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int t = blockIdx.y;
    if (v >= N) return;
    double sum = 0.0;
    if (term_of[v] < 0)
        for (uint32_t f = F[v]; f; f &= f - 1) {
            const int i = __ffs(f) - 1;
            if (term_of[v ^ ((size_t)1 << i)] == t) sum += rates[2 * i + ((v >> i) & 1u)];
        }
    b[(size_t)t * N + v] = sum;
}

// systems per CTA tile: a divisor of Kp, at most 128, and rates of the tile within 36 KB
// (with the reduction arrays the kernels stay inside the default 48 KB of shared memory).
// With `rows` > 0 the tile is also narrowed (down to 32) until one tile's slice of a
// vector over `rows` rows fits in the slice budget, so that the neighbour gathers of a
// Krylov iteration hit L2.  The budget is a tuning parameter (ESL_SWEEP_TILE_MB,
// default 48).
size_t tile_bytes() {
    static const size_t b = [] {
        const char* e = getenv("ESL_SWEEP_TILE_MB");
        const long mb = e ? atol(e) : 0;
        return (size_t)(mb > 0 ? mb : 48) << 20;
    }();
    return b;
}

// Relative residual target of an FP32 inner solve of the grid-wide groups, a tuning
// parameter (ESL_MIXED_INNER_REL, default 1e-5).
double mixed_inner_rel() {
    static const double r = [] {
        const char* e = getenv("ESL_MIXED_INNER_REL");
        const double v = e ? atof(e) : 0.0;
        return (v > 0.0 && v < 1.0) ? v : 1e-5;
    }();
    return r;
}

int tile_for(int Kp, int n, size_t elem, uint32_t rows = 0, size_t budget = 0) {
    if (budget == 0) budget = tile_bytes();
    int kt = 128;
    while (kt > 32 && (Kp % kt != 0 || (size_t)2 * n * kt * elem > 36 * 1024 ||
                       (size_t)rows * kt * elem > budget))
        kt >>= 1;
    return kt;
}

// Grid of a row kernel: blockIdx.y is the system tile, blockIdx.x strides over rows.
// Each tile gets up to 8 CTAs per SM, so a large group fills the GPU with one tile at a
// time (CTAs are dispatched x-fastest) and its working set stays that tile's slice.
dim3 row_grid(uint32_t rows, int Kp, int KT, int sm_count, int S = 1) {
    const int RB = kSwT / (KT / S);
    const unsigned ty = (unsigned)(Kp / KT);
    uint64_t want = ((uint64_t)rows + RB - 1) / RB;
    const uint64_t cap = std::max<uint64_t>(1, (uint64_t)sm_count * 8);
    if (want > cap) want = cap;
    if (want == 0) want = 1;
    return dim3((unsigned)want, ty);
}

// Launches k_sw_scc over group g without its first `skip` SCCs: its SCCs of more than kSccThreads rows, then the others
// with its singleton rows (see plan_scc_launch).
// Fewer systems: kSccGrid, which uses more of the chip for one SCC but solves the group's SCCs as
// one block.  A lone SCC of 16,384 (two CTAs) and 32,768 states (four), in ms, grid and clusters:
// 4 systems 1.26 / 1.65 and 1.36 / 1.77, 8: 1.30 / 1.65 and 1.43 / 1.78, 10: 1.50 / 1.68 and
// 2.15 / 1.82, 32: 2.42 / 1.86 and 3.25 / 1.90.
constexpr int kSccClusterMin = 8;
constexpr size_t kSccDynSmem = kSccMaxSmem - 256;  // beside the static arrays of kSccCluster and kSccGrid
// overlap: the launch may start, up to its first read of the sweep's vectors, before the
// previous one ends (not for the sweep's first: the rates are being written).
int launch_scc(esl_ctx* ctx, const SweepPlan* P, const SwGroup& g, uint32_t skip, bool defl, bool overlap, SccArgs ga) {
    const int K = ga.a.K, n = ga.a.n;
    ga.scc = P->scc.get() + g.s0;
    ga.scc_sl = P->scc_sl.get() + g.s0;
    ga.sl = P->sl.get();
    ga.ell = P->ell.get();
    const SccShape *sh = P->shapes.data() + g.sh0, *sh_end = sh + g.nsh;
    auto rows = [](const SccShape& x) { return std::max(x.even, x.odd); };
    uint32_t j = 0;  // SCCs before shape sh
    for (; j < skip; sh++) j += sh->count;
    // SCCs split over clusters: one launch per cluster size
    while (sh < sh_end && rows(*sh) > (uint32_t)kSccMaxRows) {
        auto size_of = [&](const SccShape& x) { return (rows(x) + kSccMaxRows - 1) / kSccMaxRows; };
        const uint32_t size = size_of(*sh);
        uint32_t j1 = j;
        for (; sh < sh_end && size_of(*sh) == size; sh++) j1 += sh->count;
        if ((uint64_t)(j1 - j) * K * size > 0x7FFFFFFFull) return fail(ESL_ERR_TOO_LARGE, "too many systems for one call");
        ga.nb = 1;
        ga.b[0] = SccBucket{0, (j1 - j) * (uint32_t)K, j, 0, 0, 10, 1};
        cudaLaunchAttribute attr[2]{};
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = size;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((j1 - j) * (uint32_t)K * size);
        cfg.blockDim = dim3(kSccThreadsBig);
        cfg.dynamicSmemBytes = scc_smem_doubles(true, false, n, kSccMaxRows, kSccMaxRows, 0, kSccThreadsBig) * 8;
        cfg.stream = ctx->stream;
        cfg.attrs = attr;
        cfg.numAttrs = overlap ? 2 : 1;
        auto kern = defl ? k_sw_scc<kSccCluster, true> : k_sw_scc<kSccCluster, false>;
        ESL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSccDynSmem));
        ESL_COUNT_LAUNCH();
        ESL_CUDA(cudaLaunchKernelEx(&cfg, kern, ga));
        overlap = true;
        j = j1;
    }
    for (int part = 0; part < 2; part++) {
        const bool big = part == 0;
        const SccShape* sh0 = sh;
        const uint32_t j0 = j;
        for (; sh < sh_end && (!big || rows(*sh) > (uint32_t)kSccThreads); sh++) j += sh->count;
        SccLaunch L;
        if (!plan_scc_launch(sh0, (size_t)(sh - sh0), j0, big, defl, K, n, ga.max_iters, ctx->sm_count, L))
            return fail(ESL_ERR_TOO_LARGE, "too many systems for one call");
        std::copy(L.b, L.b + L.nb, ga.b);
        ga.nb = L.nb;
        ga.ctas = L.ctas;
        int threads = L.threads;
        uint32_t singles = 0;  // CTAs for the singleton rows
        if (!big && !defl && g.singles > 0) {
            threads = std::max(threads, 128);
            const uint64_t pairs = (uint64_t)(g.ne + g.no) * (uint64_t)K;
            singles = (uint32_t)std::max<uint64_t>(
                1, std::min<uint64_t>((pairs + threads - 1) / threads, (uint64_t)ctx->sm_count * 8));
        }
        if (L.ctas + singles == 0) continue;
        auto go = [&](auto kern) -> int {
            // the same limit from every thread: contexts set it concurrently
            if (L.smem > 48 * 1024)
                ESL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSccMaxSmem));
            ESL_COUNT_LAUNCH();
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr.val.programmaticStreamSerializationAllowed = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(L.ctas + singles);
            cfg.blockDim = dim3(threads);
            cfg.dynamicSmemBytes = L.smem;
            cfg.stream = ctx->stream;
            cfg.attrs = &attr;
            cfg.numAttrs = overlap ? 1 : 0;
            ESL_CUDA(cudaLaunchKernelEx(&cfg, kern, ga));
            overlap = true;
            return ESL_OK;
        };
        if (defl) ESL_TRY(big ? go(k_sw_scc<kSccBig, true>) : go(k_sw_scc<kSccSmall, true>));
        else ESL_TRY(big ? go(k_sw_scc<kSccBig, false>) : go(k_sw_scc<kSccSmall, false>));
    }
    return ESL_OK;
}

// Launches k_sw_scc<kSccGrid> over group g: all of its rows, all systems (at most 32).
int launch_scc_grid(esl_ctx* ctx, const SwGroup& g, bool defl, SccArgs ga) {
    int lks = 0;
    while ((1 << lks) < ga.a.K) lks++;
    ga.nb = 1;
    ga.b[0] = SccBucket{0, 1, 0, 0, (uint8_t)lks, 10, 1};
    // one CTA per SM: its registers are all taken, and a launch that cannot be resident fails
    const uint64_t pairs = (uint64_t)std::max(g.ne, g.no) << lks;
    const unsigned grid = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((uint64_t)ctx->sm_count, (pairs + kSccThreadsBig - 1) / kSccThreadsBig));
    const size_t smem = ((size_t)(2 * ga.a.n + 6 * (kSccThreadsBig / 32)) << lks) * 8;
    const void* kern = defl ? (const void*)k_sw_scc<kSccGrid, true> : (const void*)k_sw_scc<kSccGrid, false>;
    if (smem > 48 * 1024)
        ESL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSccDynSmem));
    ESL_CUDA(cudaMemsetAsync(ga.bar, 0, sizeof(unsigned), ctx->stream));
    void* args[] = {&ga};
    ESL_COUNT_LAUNCH();
    ESL_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(kSccThreadsBig), args, smem, ctx->stream));
    return ESL_OK;
}

// the graphs (one per poll slot) of a Krylov solve, released on scope exit
struct GraphPair {
    cudaGraph_t graph[kSwPollDepth] = {};
    cudaGraphExec_t exec[kSwPollDepth] = {};
    GraphPair() = default;
    GraphPair(const GraphPair&) = delete;
    GraphPair& operator=(const GraphPair&) = delete;
    void reset() {
        for (int p = 0; p < kSwPollDepth; p++) {
            if (exec[p]) cudaGraphExecDestroy(exec[p]);
            if (graph[p]) cudaGraphDestroy(graph[p]);
            exec[p] = nullptr;
            graph[p] = nullptr;
        }
    }
    ~GraphPair() { reset(); }
};

bool debug_on() {
    static const bool on = getenv("ESL_DEBUG") != nullptr;
    return on;
}

// Compaction of running systems in the grid-wide groups (ESL_SWEEP_COMPACT=0 turns it
// off); groups under kCompactMinRows rows are launch-bound and keep their grid.
constexpr uint32_t kCompactMinRows = 4096;
// Operator kernels of the 32-system tiles of FP64 grid groups: the paired-row kernels,
// or one system per lane with ESL_SWEEP_OP=reg
bool paired_on() {
    static const bool on = [] {
        const char* e = getenv("ESL_SWEEP_OP");
        return !(e && !strcmp(e, "reg"));
    }();
    return on;
}

bool compact_on() {
    static const bool on = [] {
        const char* e = getenv("ESL_SWEEP_COMPACT");
        return !(e && e[0] == '0');
    }();
    return on;
}

// FNV-1a 64 over n 32-bit words of a device array
int dev_checksum(const void* d, size_t words, cudaStream_t s, uint64_t& h) {
    std::vector<uint32_t> v(words);
    if (words) {
        ESL_CUDA(cudaMemcpyAsync(v.data(), d, words * 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
    }
    h = 1469598103934665603ull;
    for (uint32_t w : v) {
        h ^= w;
        h *= 1099511628211ull;
    }
    return ESL_OK;
}

int plan_checksums(esl_ctx* ctx, const SweepPlan& P, uint64_t (&h)[12]) {
    cudaStream_t s = ctx->stream;
    uint32_t ig = 0, og = 0, tp = 0, count = 0;
    for (const SwGroup& g : P.groups) count += g.ns;
    if (P.M) {
        ESL_CUDA(cudaMemcpyAsync(&ig, P.ig_ptr.get() + P.M, 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(&og, P.og_ptr.get() + P.M, 4, cudaMemcpyDeviceToHost, s));
    }
    ESL_CUDA(cudaMemcpyAsync(&tp, P.tp_ptr.get() + P.TS, 4, cudaMemcpyDeviceToHost, s));
    ESL_CUDA(cudaStreamSynchronize(s));
    ESL_TRY(dev_checksum(P.rows.get(), (size_t)P.M * 2, s, h[0]));
    ESL_TRY(dev_checksum(P.desc.get(), (size_t)P.M * 4, s, h[1]));
    ESL_TRY(dev_checksum(P.ig_ptr.get(), P.M ? (size_t)P.M + 1 : 0, s, h[2]));
    ESL_TRY(dev_checksum(P.ig_ent.get(), ig, s, h[3]));
    ESL_TRY(dev_checksum(P.og_ptr.get(), P.M ? (size_t)P.M + 1 : 0, s, h[4]));
    ESL_TRY(dev_checksum(P.og_ent.get(), og, s, h[5]));
    ESL_TRY(dev_checksum(P.tp_ptr.get(), (size_t)P.TS + 1, s, h[6]));
    ESL_TRY(dev_checksum(P.tp_ent.get(), tp, s, h[7]));
    ESL_TRY(dev_checksum(P.scc.get(), (size_t)count * 4, s, h[8]));
    uint64_t first_slices = 0;
    ESL_TRY(dev_checksum(P.scc_sl.get(), (size_t)count * 2, s, first_slices));
    ESL_TRY(dev_checksum(P.sl.get(), P.sl.n * 2, s, h[9]));
    ESL_TRY(dev_checksum(P.ell.get(), P.ell.n * 4, s, h[10]));
    uint64_t g = 1469598103934665603ull;
    auto mix = [&](uint64_t x) {
        g ^= x;
        g *= 1099511628211ull;
    };
    for (const SwGroup& gr : P.groups) {
        mix(gr.beg);
        mix(gr.ne);
        mix(gr.no);
        mix((uint64_t)gr.kind);
        mix((uint64_t)gr.max_scc);
        mix(gr.nin);
        for (uint32_t x : {gr.s0, gr.ns, gr.sh0, gr.nsh, gr.l0, gr.nlarge, gr.most, gr.singles}) mix(x);
        mix(gr.resident);
        mix(gr.split);
    }
    for (const SccShape& x : P.shapes)
        for (uint32_t y : {x.even, x.odd, x.count}) mix(y);
    for (const uint4& c : P.large)
        for (uint32_t y : {c.x, c.y, c.z, c.w}) mix(y);
    mix(first_slices);
    mix(P.max_rows);
    mix(P.max_even);
    mix(P.max_odd);
    h[11] = g;
    return ESL_OK;
}

}  // namespace

int plan_checksums_for(esl_ctx* ctx, const esl_net* net, int host, uint64_t* out, int cap) {
    if (!sweep_supported(net)) return fail(ESL_ERR_TOO_LARGE, "level sweep supports at most 26 nodes");
    SweepPlan* P = nullptr;
    ESL_TRY(host ? build_plan_host(ctx, net, P) : build_plan_device(ctx, net, P));
    std::unique_ptr<SweepPlan> keep(P);
    if (!host) ESL_TRY(finish_scc_list(ctx, P, nullptr));
    uint64_t h[12];
    ESL_TRY(plan_checksums(ctx, *P, h));
    for (int i = 0; i < cap && i < 12; i++) out[i] = h[i];
    return ESL_OK;
}

void free_sweep_workspace(void* w) { delete static_cast<Workspace*>(w); }

int sweep_prepare(esl_ctx* ctx, const esl_net* net) {
    if (!sweep_supported(net)) return ESL_OK;
    SweepPlan* P = nullptr;
    return build_plan(ctx, net, P);
}

int sweep_targets(esl_ctx* ctx, const esl_net* net, std::vector<uint32_t>& states) {
    if (!sweep_supported(net)) return fail(ESL_ERR_TOO_LARGE, "level sweep supports at most 26 nodes");
    SweepPlan* P = nullptr;
    ESL_TRY(build_plan(ctx, net, P));
    std::vector<uint2> rows(P->M);
    if (P->M > 0) {
        ESL_CUDA(cudaMemcpyAsync(rows.data(), P->rows.get(), (size_t)P->M * sizeof(uint2), cudaMemcpyDeviceToHost,
                                 ctx->stream));
        ESL_CUDA(cudaStreamSynchronize(ctx->stream));
    }
    states.clear();
    for (const SwGroup& g : P->groups)
        if (g.kind == 2)
            for (uint32_t r = g.beg + g.ne; r < g.beg + g.ne + g.no; r++) states.push_back(rows[r].x);
    return ESL_OK;
}

// slots are packed into 26 bits of a predecessor entry
bool sweep_supported(const esl_net* net) { return net->n >= 1 && net->n <= 26; }

namespace {

// The group loop of the level sweep over plan P.  Transient mode (term == false): the
// groups of the transient states, y[k * T + t] += mass into terminal SCC t.  Terminal
// mode: the deflated groups of the big terminal SCCs (P = the terminal plan, nrhs = 1,
// x0 unused), their normalised kernels into y = Rb[k][position], FP64 throughout.
int sweep_run(esl_ctx* ctx, const esl_net* net, SweepPlan* P, bool term, int K, int nrhs, const double* rates,
              const double* x0, size_t x0_ld, const esl_solve_opts& o, double* y, SweepStats& st) {
    if (!ctx->sweep_work) ctx->sweep_work = new Workspace();
    Workspace& ws = *static_cast<Workspace*>(ctx->sweep_work);
    cudaStream_t s = ctx->stream;
    const int n = net->n, T = net->T;
    const int Kp = (K + 31) & ~31;
    const bool mixed = !term && o.method == ESL_METHOD_MIXED;
    const bool defl = term;
    int st_ = ESL_OK;
    double* Z = (double*)ws.get(W_Z, (size_t)std::max<uint32_t>(P->M, 1) * Kp * 8, &st_);
    double* rateT = (double*)ws.get(W_RATET, (size_t)2 * n * Kp * 8, &st_);
    double* scal = (double*)ws.get(W_SCAL, (size_t)C_NSCAL * Kp * 8, &st_);
    int* iscal = (int*)ws.get(W_ISCAL, (size_t)I_NISCAL * Kp * 4, &st_);
    int* d_cnt = (int*)ws.get(W_CNT, 64, &st_);
    // results of the SCC-resident groups: per system max |r|^2/|b|^2 and failure flag, per
    // group the most iterations and refinement steps
    const size_t loc_bytes = (size_t)Kp * 12 + P->groups.size() * 8;
    unsigned long long* loc_ratio = (unsigned long long*)ws.get(W_LOC, loc_bytes, &st_);
    if (st_ != ESL_OK) return st_;
    int* loc_fail = reinterpret_cast<int*>(loc_ratio + Kp);
    int* loc_iters = loc_fail + Kp;
    ESL_CUDA(cudaMemsetAsync(loc_ratio, 0, loc_bytes, s));
    ESL_CUDA(cudaMemsetAsync(d_cnt + 8, 0, 8, s));
    SwScalPtr sc;
    for (int j = 0; j < C_NSCAL; j++) sc.c[j] = scal + (size_t)j * Kp;
    for (int j = 0; j < I_NISCAL; j++) sc.i[j] = iscal + (size_t)j * Kp;
    ESL_COUNT_LAUNCH();
    k_sw_rate_table<<<dim3((Kp + 127) / 128, 2 * n), 128, 0, s>>>(n, K, Kp, nrhs, rates, rateT);
    ESL_CUDA(cudaGetLastError());

    const int KT64 = tile_for(Kp, n, 8);
    const size_t sm64 = (size_t)2 * n * KT64 * 8;
    SwArgs a{};
    a.n = n;
    a.K = K;
    a.Kp = Kp;
    a.nrhs = nrhs;
    a.rateT = rateT;
    a.rows = P->rows.get();
    a.desc = P->desc.get();
    a.ig_ptr = P->ig_ptr.get();
    a.ig_ent = P->ig_ent.get();
    int* h_cnt = reinterpret_cast<int*>(ctx->h_flag);  // pinned, at least 8 ints

    const double tol = o.tol > 0 ? o.tol : 1e-10;
    const int max_iters = o.max_iters > 0 ? o.max_iters : 600;
    const int max_refine = o.max_refine > 0 ? o.max_refine : 6;
    std::vector<int> h_flags;
    std::vector<char> failed(K, 0);
    int total_iters = 0;

    // arguments of k_sw_scc for group g (the row range is a's); resident: not kSccGrid
    auto scc_args = [&](const SwGroup& g, bool resident, SccArgs& ga) -> int {
        ga.a = a;
        ga.og_ptr = P->og_ptr.get();
        ga.og_ent = P->og_ent.get();
        ga.x0 = x0;
        ga.x0_ld = x0_ld;
        ga.warm = term ? nullptr : o.d_warm;
        ga.warm_ld = (size_t)net->N;
        ga.rev = P->rev.get();
        ga.Z = Z;
        const int slots[kOwnCount] = {W_R0, W_D, W_DS64, W_QO, W_BS, W_PH, W_W64, W_R, W_V, W_SH, W_TT, W_IQE};
        const bool big = g.most > (uint32_t)kSccThreads;
        for (int j = 0; j < (resident ? (big ? kOwnBS + 1 : 0) : kOwnCount); j++)
            ga.own[j] = (double*)ws.get(slots[j], (size_t)scc_own_rows(j, P->max_even, P->max_odd) * Kp * 8, &st_);
        if (!resident) {
            ga.bar = reinterpret_cast<unsigned*>(d_cnt) + 8;
            const bool no_end = barrier_timeout_test();
            ga.polls = no_end ? kBarrierTestPolls : kBarrierPolls;
            ga.missing = no_end ? 1 : 0;
            ga.part = (double*)ws.get(W_PART, (size_t)2 * ctx->sm_count * 3 * 32 * 8, &st_);
        }
        if (st_ != ESL_OK) return st_;
        ga.tol2 = tol * tol;
        ga.accept2 = kSwAcceptRel * kSwAcceptRel;
        ga.max_iters = max_iters;
        ga.max_outer = g.kind == 2 ? max_refine : max_refine + 3;
        ga.stall = g.kind == 2 ? kSwStall64 : kSwStall;
        ga.ratio = loc_ratio;
        ga.fail = loc_fail;
        ga.iters = loc_iters + (&g - P->groups.data());
        ga.refines = ga.iters + P->groups.size();
        if (term) {
            ga.pos = P->pos.get();
            ga.Rb = y;
            ga.TS = net->term_states;
        }
        return ESL_OK;
    };
    uint32_t largest = 0;  // states of the largest SCC
    for (const SccShape& x : P->shapes) largest = std::max(largest, x.even + x.odd);
    // debug timing: wall time of a group with the stream drained on both sides
    std::chrono::steady_clock::time_point g_t0;
    auto g_ms = [&]() {
        return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - g_t0).count();
    };
    // Grid-wide Krylov solve of one SCC of a group by the row kernels.
    auto solve_rows = [&](const SwGroup& g) -> int {
        const uint32_t rows = g.ne + g.no;
        a.beg = g.beg;
        a.ob = g.ob;
        a.ne = g.ne;
        a.no = g.no;
        a.flags = nullptr;
        a.KT = KT64;
        a.Qo = a.IQe = nullptr;
        a.gam = nullptr;
        a.inv_s = 1.0 / (double)std::max<uint32_t>(rows, 1);
        double* Bv = (double*)ws.get(W_BV, (size_t)P->max_rows * Kp * 8, &st_);
        if (st_ != ESL_OK) return st_;
        ESL_COUNT_LAUNCH();
        if (term)
            k_sw_defl_rhs<<<row_grid(rows, Kp, KT64, ctx->sm_count), kSwT, sm64, s>>>(a, Bv);
        else
            k_sw_rhs<false><<<row_grid(rows, Kp, KT64, ctx->sm_count), kSwT, sm64, s>>>(
                a, P->og_ptr.get(), P->og_ent.get(), x0, x0_ld, Z, Bv);
        ESL_CUDA(cudaGetLastError());
        st.krylov_groups++;
        const size_t vo = (size_t)std::max<uint32_t>(P->max_odd, 1) * Kp, ve = (size_t)std::max<uint32_t>(P->max_even, 1) * Kp;
        double* bS = (double*)ws.get(W_BS, vo * 8, &st_);
        double* R64 = (double*)ws.get(W_R64, vo * 8, &st_);
        double* dS64 = (double*)ws.get(W_DS64, vo * 8, &st_);
        float* dS32 = mixed ? (float*)ws.get(W_DS32, vo * 4, &st_) : nullptr;
        double* W64 = (double*)ws.get(W_W64, ve * 8, &st_);
        // 8 bytes per entry: a mixed solve may continue with FP64 inner steps in these buffers
        const size_t es = 8;
        void* WT = mixed ? ws.get(W_WT, ve * es, &st_) : (void*)W64;
        void* vR = ws.get(W_R, vo * es, &st_);
        void* vR0 = ws.get(W_R0, vo * es, &st_);
        void* vPH = ws.get(W_PH, vo * es, &st_);
        void* vV = ws.get(W_V, vo * es, &st_);
        void* vSH = ws.get(W_SH, vo * es, &st_);
        void* vTT = ws.get(W_TT, vo * es, &st_);
        void* vD = ws.get(W_D, vo * es, &st_);
        if (st_ != ESL_OK) return st_;
        double* X64 = Z + (size_t)g.ob * Kp;  // the odd rows, in place
        // tiles narrow enough that one tile's slice of a gathered vector stays in L2
        // the network's autotuned slice budget, or the default
        const int tmb = net->tune_tile_mb > 0 ? net->tune_tile_mb : ctx->tune_tile_mb;
        const size_t budget = tmb > 0 ? (size_t)tmb << 20 : 0;
        // FP64, not deflated: groups whose 64-system slice exceeds 1 MB (above 2,048 rows)
        // run 32-system tiles, where the paired-row operator kernels apply (measured 4-5%
        // faster per step on the n=20 bench network than 64- and 128-system tiles in
        // L2-sized slices)
        const size_t budget64 =
            paired_on() && !defl ? std::min(budget ? budget : tile_bytes(), (size_t)1 << 20) : budget;
        const int gKT64 = tile_for(Kp, n, 8, std::max(g.ne, g.no), budget64),
                  gKT32 = tile_for(Kp, n, 4, std::max(g.ne, g.no), budget);
        const size_t gsm64 = (size_t)2 * n * gKT64 * 8, gsm32 = (size_t)2 * n * gKT32 * 4;
        a.KT = gKT64;
        const dim3 ge = row_grid(g.ne, Kp, gKT64, ctx->sm_count), go = row_grid(g.no, Kp, gKT64, ctx->sm_count);
        ESL_CUDA(cudaMemsetAsync(scal, 0, (size_t)C_NSCAL * Kp * 8, s));
        ESL_CUDA(cudaMemsetAsync(iscal, 0, (size_t)I_NISCAL * Kp * 4, s));
        ESL_COUNT_LAUNCH();
        k_sw_diag<<<go, kSwT, gsm64, s>>>(a, dS64, dS32);
        // out-rate sums of the rows, read by the FP64 operator kernels of this group
        double* Qo = (double*)ws.get(W_QO, vo * 8, &st_);
        double* IQe = (double*)ws.get(W_IQE, ve * 8, &st_);
        if (st_ != ESL_OK) return st_;
        ESL_COUNT_LAUNCH();
        k_sw_qrows<<<row_grid(g.ne + g.no, Kp, gKT64, ctx->sm_count), kSwT, gsm64, s>>>(a, Qo, IQe);
        a.Qo = Qo;
        a.IQe = IQe;
        // reduced rhs bS = b_odd + A_oe (b_even / q_e)
        ESL_COUNT_LAUNCH();
        k_sw_elim<1, double, double, double><<<ge, kSwT, gsm64, s>>>(a, Bv, (const double*)nullptr, W64);
        ESL_COUNT_LAUNCH();
        k_sw_apply<1, 0, double><<<go, kSwT, gsm64, s>>>(a, nullptr, W64, Bv + (size_t)g.ne * Kp, nullptr, bS,
                                                     sc.c[C_BB], nullptr, nullptr, nullptr);
        ESL_COUNT_LAUNCH();
        const double* warm = term ? nullptr : o.d_warm;
        k_sw_init<<<go, kSwT, 0, s>>>(a, warm, (size_t)net->N, bS, dS64, X64);
        ESL_CUDA(cudaGetLastError());
        // An NVTX range names the row-kernel solve of the network's largest transient SCC (of
        // each, where several are that large; of none, where k_sw_scc solves it), so that a
        // profiler can select its launches (`ncu --nvtx --nvtx-include
        // "esl_largest_level_group/"`); without a profiler attached it costs nothing.
        struct NvtxRange {
            bool on;
            explicit NvtxRange(bool b) : on(b) {
                if (on) nvtxRangePushA("esl_largest_level_group");
            }
            ~NvtxRange() {
                if (on) nvtxRangePop();
            }
        } nvtx_range(!term && rows == largest);
        auto true_residual = [&]() -> int {
            a.flags = nullptr;
            a.KT = gKT64;
            ESL_CUDA(cudaMemsetAsync(sc.c[C_RR64], 0, (size_t)Kp * 8, s));
            if (defl) {
                // R64 = bS - (S X + gamma(X) u)
                ESL_CUDA(cudaMemsetAsync(sc.c[C_GAM0], 0, (size_t)Kp * 8, s));
                SwArgs ad = a;
                ad.gam = sc.c[C_GAM0];
                ESL_COUNT_LAUNCH();
                k_sw_elim<1, double, double, double, true><<<ge, kSwT, gsm64, s>>>(ad, nullptr, X64, W64);
                ESL_COUNT_LAUNCH();
                k_sw_apply<1, 1, double, true><<<go, kSwT, gsm64, s>>>(ad, X64, W64, bS, nullptr, R64, sc.c[C_D0],
                                                                        nullptr, nullptr, nullptr);
                ESL_COUNT_LAUNCH();
                k_sw_defl_fin<1><<<go, kSwT, 0, s>>>(ad, R64, nullptr, nullptr, nullptr, sc.c[C_GAM0], sc.c[C_RR64],
                                                    nullptr, nullptr);
                ESL_CUDA(cudaGetLastError());
                return ESL_OK;
            }
            ESL_COUNT_LAUNCH();
            k_sw_elim<1, double, double, double><<<ge, kSwT, gsm64, s>>>(a, nullptr, X64, W64);
            ESL_COUNT_LAUNCH();
            k_sw_apply<1, 1, double><<<go, kSwT, gsm64, s>>>(a, X64, W64, bS, nullptr, R64, sc.c[C_RR64], nullptr, nullptr, nullptr);
            ESL_CUDA(cudaGetLastError());
            return ESL_OK;
        };
        if (warm) {
            // least-squares scale of the warm start per system (C_R0V, C_TS as scratch)
            ESL_CUDA(cudaMemsetAsync(sc.c[C_R0V], 0, (size_t)Kp * 8, s));
            ESL_CUDA(cudaMemsetAsync(sc.c[C_TS], 0, (size_t)Kp * 8, s));
            ESL_COUNT_LAUNCH();
            k_sw_elim<1, double, double, double><<<ge, kSwT, gsm64, s>>>(a, nullptr, X64, W64);
            ESL_COUNT_LAUNCH();
            k_sw_apply<1, 4, double><<<go, kSwT, gsm64, s>>>(a, X64, W64, bS, nullptr, nullptr, sc.c[C_R0V],
                                                              sc.c[C_TS], nullptr, nullptr);
            ESL_COUNT_LAUNCH();
            k_sw_warm_scale<<<go, kSwT, 0, s>>>(a, sc.c[C_R0V], sc.c[C_TS], X64);
            ESL_CUDA(cudaGetLastError());
        }
        ESL_TRY(true_residual());
        bool inner64 = !mixed;
        int group_iters = 0;
        for (int outer = 0;; outer++) {
            const double inner_rel = inner64 ? 1e-13 : mixed_inner_rel();
            ESL_COUNT_LAUNCH();
            k_sw_outer<<<1, 1024, 0, s>>>(K, sc, tol * tol, inner_rel * inner_rel, kSwAcceptRel * kSwAcceptRel,
                                          outer, max_refine, d_cnt);
            ESL_CUDA(cudaGetLastError());
            ESL_CUDA(cudaMemcpyAsync(h_cnt, d_cnt, 4, cudaMemcpyDeviceToHost, s));
            ESL_CUDA(cudaStreamSynchronize(s));
            if (h_cnt[0] == 0) break;
            a.flags = sc.i[I_FLAGS];
            a.KT = inner64 ? gKT64 : gKT32;
            const size_t smT = inner64 ? gsm64 : gsm32;
            dim3 gei = row_grid(g.ne, Kp, a.KT, ctx->sm_count), goi = row_grid(g.no, Kp, a.KT, ctx->sm_count);
            // two systems per thread in the gather kernels when the tile is wide enough
            // (not in deflated groups)
            const bool s2 = !defl && a.KT >= 64 && (net->tune_s2 >= 0 ? net->tune_s2 != 0 : ctx->tune_s2 != 0);
            dim3 gei2 = row_grid(g.ne, Kp, a.KT, ctx->sm_count, 2), goi2 = row_grid(g.no, Kp, a.KT, ctx->sm_count, 2);
            // paired-row kernels on the 32-system tiles of FP64 inner solves (grids gei2 /
            // goi2: 16 rows per CTA step)
            const bool paired = inner64 && !defl && paired_on() && a.KT == 32 && a.Qo && a.IQe;
            // gathered-vector element offsets (row * Kp) fit in 32 bits
            const bool o32 = (uint64_t)std::max(g.ne, g.no) * (uint64_t)Kp < (1ull << 31);
            auto run_inner = [&](auto tag) -> int {
                using TT = decltype(tag);
                TT* R = (TT*)vR;
                TT* R0 = (TT*)vR0;
                TT* PH = (TT*)vPH;
                TT* V = (TT*)vV;
                TT* SH = (TT*)vSH;
                TT* Tt = (TT*)vTT;
                TT* D = (TT*)vD;
                TT* WW = (TT*)(sizeof(TT) == 8 ? (void*)W64 : WT);
                const TT* dS = (const TT*)(sizeof(TT) == 8 ? (void*)dS64 : (void*)dS32);
                // measurement hook: the launches of the first poll window, when every
                // started system still runs.  Algorithmic bytes per running system: the
                // operator moves every vector it touches once (the gathered vector too),
                // leaving out the per-row out-rate streams that a kernel could recompute;
                // the row structure (12 B per row, 4 B per predecessor entry) is shared.
                const double nrun = h_cnt[0];
                const double row_bytes = 12.0 * (g.ne + g.no) + 4.0 * (double)g.nin;
                const double op2_bytes = nrun * sizeof(TT) * (2.0 * g.ne + 4.0 * g.no) + row_bytes;
                const double op6_bytes = nrun * sizeof(TT) * (2.0 * g.ne + 5.0 * g.no) + row_bytes;
                const double s_bytes = nrun * sizeof(TT) * 4.0 * g.no, xrp_bytes = nrun * sizeof(TT) * 10.0 * g.no;
                ESL_COUNT_LAUNCH();
                k_sw_start<TT><<<goi, kSwT, 0, s>>>(a, sc.c[C_SCALE], R64, dS, R, R0, D, PH, V);
                // kSwPoll iterations; `par` picks the running-count slot of this poll window
                auto launch_chunk = [&](int par, bool record) -> int {
                    esl_ctx* pc = record ? ctx : nullptr;
                    for (int j = 0; j < kSwPoll; j++) {
                    if (defl) {
                        // v = A p and t = A s of the deflated operator (FP64 only)
                        if constexpr (sizeof(TT) == 8) {
                        SwArgs ad = a;
                        ad.gam = sc.c[C_GAM1];
                        ESL_COUNT_LAUNCH();
                        k_sw_elim<1, TT, TT, TT, true><<<gei, kSwT, smT, s>>>(ad, nullptr, PH, WW);
                        ESL_COUNT_LAUNCH();
                        k_sw_apply<1, 2, TT, true><<<goi, kSwT, smT, s>>>(ad, PH, WW, nullptr, R0, V, sc.c[C_D0],
                                                                         nullptr, nullptr, nullptr);
                        ESL_COUNT_LAUNCH();
                        k_sw_defl_fin<2><<<goi, kSwT, 0, s>>>(ad, (double*)V, nullptr, (const double*)R0, nullptr,
                                                             sc.c[C_GAM1], sc.c[C_R0V], nullptr, nullptr);
                        ESL_COUNT_LAUNCH();
                        k_sw_s<TT><<<goi, kSwT, 0, s>>>(a, sc, R, V, dS, SH);
                        ad.gam = sc.c[C_GAM2];
                        ESL_COUNT_LAUNCH();
                        k_sw_elim<1, TT, TT, TT, true><<<gei, kSwT, smT, s>>>(ad, nullptr, SH, WW);
                        ESL_COUNT_LAUNCH();
                        k_sw_apply<1, 6, TT, true><<<goi, kSwT, smT, s>>>(ad, SH, WW, nullptr, dS, Tt, sc.c[C_D0],
                                                                         sc.c[C_D1], R0, sc.c[C_D2]);
                        ESL_COUNT_LAUNCH();
                        k_sw_defl_fin<6><<<goi, kSwT, 0, s>>>(ad, (double*)Tt, (const double*)SH, (const double*)dS,
                                                             (const double*)R0, sc.c[C_GAM2], sc.c[C_TS],
                                                             sc.c[C_TT], sc.c[C_R0T]);
                        ESL_COUNT_LAUNCH();
                        k_sw_xrp<TT><<<goi, kSwT, 0, s>>>(a, sc, PH, SH, dS, Tt, R0, V, D, R);
                        ESL_COUNT_LAUNCH();
                        k_sw_scal<<<1, 1024, 0, s>>>(a.K, sc, max_iters, sizeof(TT) == 8 ? kSwStall64 : kSwStall,
                                                     d_cnt + 1 + par);
                        }
                        continue;
                    }
                    if constexpr (sizeof(TT) == 8) {
                        if (paired) {
                            // the paired-row kernels' rate table has a zero row appended
                            const size_t smP = smT + 32 * 8;
                            {
                                ProfScope ps(pc, "schur_operator", op2_bytes);
                                ESL_COUNT_LAUNCH();
                                if (o32) k_sw_elim_pr<true><<<gei2, kSwT, smP, s>>>(a, PH, WW);
                                else k_sw_elim_pr<false><<<gei2, kSwT, smP, s>>>(a, PH, WW);
                                ESL_COUNT_LAUNCH();
                                if (o32)
                                    k_sw_apply_pr<2, true><<<goi2, kSwT, smP, s>>>(a, PH, WW, R0, V, sc.c[C_R0V], nullptr,
                                                                                  nullptr, nullptr);
                                else
                                    k_sw_apply_pr<2, false><<<goi2, kSwT, smP, s>>>(a, PH, WW, R0, V, sc.c[C_R0V], nullptr,
                                                                                   nullptr, nullptr);
                            }
                            {
                                ProfScope ps(pc, "bicgstab_update", s_bytes);
                                ESL_COUNT_LAUNCH();
                                k_sw_s2<<<goi2, kSwT, 0, s>>>(a, sc, R, V, dS, SH);
                            }
                            {
                                ProfScope ps(pc, "schur_operator", op6_bytes);
                                ESL_COUNT_LAUNCH();
                                if (o32) k_sw_elim_pr<true><<<gei2, kSwT, smP, s>>>(a, SH, WW);
                                else k_sw_elim_pr<false><<<gei2, kSwT, smP, s>>>(a, SH, WW);
                                ESL_COUNT_LAUNCH();
                                if (o32)
                                    k_sw_apply_pr<6, true><<<goi2, kSwT, smP, s>>>(a, SH, WW, dS, Tt, sc.c[C_TS], sc.c[C_TT],
                                                                                  R0, sc.c[C_R0T]);
                                else
                                    k_sw_apply_pr<6, false><<<goi2, kSwT, smP, s>>>(a, SH, WW, dS, Tt, sc.c[C_TS],
                                                                                   sc.c[C_TT], R0, sc.c[C_R0T]);
                            }
                            {
                                ProfScope ps(pc, "bicgstab_update", xrp_bytes);
                                ESL_COUNT_LAUNCH();
                                k_sw_xrp2<<<goi2, kSwT, 0, s>>>(a, sc, PH, SH, dS, Tt, R0, V, D, R);
                            }
                            ESL_COUNT_LAUNCH();
                            k_sw_scal<<<1, 1024, 0, s>>>(a.K, sc, max_iters, kSwStall64, d_cnt + 1 + par);
                            continue;
                        }
                    }
                    {
                        ProfScope ps(pc, "schur_operator", op2_bytes);
                        ESL_COUNT_LAUNCH();
                        if (s2)
                            k_sw_elim<2, TT, TT, TT><<<gei2, kSwT, smT, s>>>(a, nullptr, PH, WW);
                        else
                            k_sw_elim<1, TT, TT, TT><<<gei, kSwT, smT, s>>>(a, nullptr, PH, WW);
                        ESL_COUNT_LAUNCH();
                        if (s2)
                            k_sw_apply<2, 2, TT><<<goi2, kSwT, smT, s>>>(a, PH, WW, nullptr, R0, V, sc.c[C_R0V], nullptr, nullptr, nullptr);
                        else
                            k_sw_apply<1, 2, TT><<<goi, kSwT, smT, s>>>(a, PH, WW, nullptr, R0, V, sc.c[C_R0V], nullptr, nullptr, nullptr);
                    }
                    {
                        ProfScope ps(pc, "bicgstab_update", s_bytes);
                        ESL_COUNT_LAUNCH();
                        if constexpr (sizeof(TT) == 8)
                            k_sw_s2<<<goi2, kSwT, 0, s>>>(a, sc, R, V, dS, SH);
                        else
                            k_sw_s<TT><<<goi, kSwT, 0, s>>>(a, sc, R, V, dS, SH);
                    }
                    {
                        ProfScope ps(pc, "schur_operator", op6_bytes);
                        ESL_COUNT_LAUNCH();
                        if (s2)
                            k_sw_elim<2, TT, TT, TT><<<gei2, kSwT, smT, s>>>(a, nullptr, SH, WW);
                        else
                            k_sw_elim<1, TT, TT, TT><<<gei, kSwT, smT, s>>>(a, nullptr, SH, WW);
                        ESL_COUNT_LAUNCH();
                        if (s2)
                            k_sw_apply<2, 6, TT><<<goi2, kSwT, smT, s>>>(a, SH, WW, nullptr, dS, Tt, sc.c[C_TS],
                                                                          sc.c[C_TT], R0, sc.c[C_R0T]);
                        else
                            k_sw_apply<1, 6, TT><<<goi, kSwT, smT, s>>>(a, SH, WW, nullptr, dS, Tt, sc.c[C_TS],
                                                                          sc.c[C_TT], R0, sc.c[C_R0T]);
                    }
                    {
                        ProfScope ps(pc, "bicgstab_update", xrp_bytes);
                        ESL_COUNT_LAUNCH();
                        if constexpr (sizeof(TT) == 8)
                            k_sw_xrp2<<<goi2, kSwT, 0, s>>>(a, sc, PH, SH, dS, Tt, R0, V, D, R);
                        else
                            k_sw_xrp<TT><<<goi, kSwT, 0, s>>>(a, sc, PH, SH, dS, Tt, R0, V, D, R);
                    }
                    ESL_COUNT_LAUNCH();
                    k_sw_scal<<<1, 1024, 0, s>>>(a.K, sc, max_iters, sizeof(TT) == 8 ? kSwStall64 : kSwStall,
                                                 d_cnt + 1 + par);
                    }
                    ESL_CUDA(cudaGetLastError());
                    return ESL_OK;
                };
                // compaction state: Kc leading columns hold the systems that may still run
                const bool can_compact = compact_on() && Kp <= kCompactMaxKp && (g.ne + g.no) >= kCompactMinRows;
                int Kc = Kp;
                bool compacted = false;
                int *cperm = nullptr, *p2 = nullptr;
                PermList pl{};
                int npl = 0;
                auto add_perm = [&](const void* p, uint32_t nrows, int es) {
                    if (p && nrows) pl.a[npl++] = PermArr{const_cast<void*>(p), nrows, es};
                };
                const dim3 gei0 = gei, goi0 = goi, gei20 = gei2, goi20 = goi2;
                const unsigned perm_blocks = (unsigned)std::max<uint64_t>(
                    1, std::min<uint64_t>(((uint64_t)std::max(g.ne, g.no) + kPermWarps - 1) / kPermWarps,
                                          (uint64_t)ctx->sm_count * 8));
                // After the first poll window the launches of a window are replayed from a
                // CUDA graph (one per slot parity): the small level groups are bound by the
                // host's launch rate, not by the GPU.
                GraphPair gp;
                bool capturable = s != cudaStreamLegacy && s != nullptr && s != cudaStreamPerThread;
                cudaGraph_t* graph = gp.graph;
                cudaGraphExec_t* gexec = gp.exec;
                int it = 0, chunk = 0;
                for (; it < max_iters; it += kSwPoll, chunk++) {
                    const int par = chunk % kSwPollDepth;  // the window's running-count slot
                    if (chunk == 0 || !capturable) {
                        ESL_TRY(launch_chunk(par, ctx->prof && chunk == 0));
                    } else if (!gexec[par]) {
                        if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
                            // the legacy default stream cannot be captured: launch directly
                            capturable = false;
                            ESL_TRY(launch_chunk(par, false));
                            goto poll;
                        }
                        int rc = launch_chunk(par, false);
                        if (cudaStreamEndCapture(s, &graph[par]) != cudaSuccess && rc == ESL_OK)
                            rc = fail(ESL_ERR_CUDA, "stream capture failed");
                        if (rc == ESL_OK && cudaGraphInstantiate(&gexec[par], graph[par], 0) != cudaSuccess)
                            rc = fail(ESL_ERR_CUDA, "graph instantiation failed");
                        if (rc == ESL_OK && cudaGraphLaunch(gexec[par], s) != cudaSuccess)
                            rc = fail(ESL_ERR_CUDA, "graph launch failed");
                        if (rc != ESL_OK) return rc;
                    } else {
                        count_launches((defl ? 9 : 7) * kSwPoll);
                        if (cudaGraphLaunch(gexec[par], s) != cudaSuccess)
                            return fail(ESL_ERR_CUDA, "graph launch failed");
                    }
                poll:
                    ESL_CUDA(cudaMemcpyAsync(h_cnt + 1 + par, d_cnt + 1 + par, 4, cudaMemcpyDeviceToHost, s));
                    ESL_CUDA(cudaEventRecord(ctx->poll_ev[par], s));
                    if (chunk >= kSwPollDepth - 1) {
                        const int old_slot = (chunk - (kSwPollDepth - 1)) % kSwPollDepth;
                        ESL_CUDA(cudaEventSynchronize(ctx->poll_ev[old_slot]));
                        const int nr = h_cnt[1 + old_slot];
                        if (nr == 0) {
                            it += kSwPoll;
                            break;
                        }
                        // The count is that of a window before the ones in flight, an upper
                        // bound of the systems still running when the compaction (queued
                        // behind them) runs.
                        const int tiles_now = Kc / a.KT, tiles_new = (nr + a.KT - 1) / a.KT;
                        if (can_compact && tiles_now - tiles_new >= 2) {
                            if (!compacted) {
                                cperm = (int*)ws.get(W_PERM, (size_t)Kp * 8, &st_);
                                if (st_ != ESL_OK) return st_;
                                p2 = cperm + Kp;
                                ESL_COUNT_LAUNCH();
                                k_sw_iota<<<(Kp + 255) / 256, 256, 0, s>>>(Kp, cperm);
                                add_perm(R, g.no, sizeof(TT));
                                add_perm(R0, g.no, sizeof(TT));
                                add_perm(PH, g.no, sizeof(TT));
                                add_perm(V, g.no, sizeof(TT));
                                add_perm(SH, g.no, sizeof(TT));
                                add_perm(Tt, g.no, sizeof(TT));
                                add_perm(D, g.no, sizeof(TT));
                                add_perm(dS64, g.no, 8);
                                add_perm(dS32, g.no, 4);
                                add_perm(a.Qo, g.no, 8);
                                add_perm(a.IQe, g.ne, 8);
                                add_perm(a.rateT, 2 * n, 8);
                                add_perm(scal, C_NSCAL, 8);
                                add_perm(iscal, I_NISCAL, 4);
                                compacted = true;
                            }
                            ESL_COUNT_LAUNCH();
                            k_sw_perm_build<<<1, 1024, 0, s>>>(Kc, sc.i[I_FLAGS], cperm, p2);
                            ESL_COUNT_LAUNCH();
                            k_sw_row_perm<<<dim3(perm_blocks, npl), kPermWarps * 32, (size_t)kPermWarps * Kc * 8, s>>>(
                                pl, Kp, Kc, p2, 0);
                            ESL_CUDA(cudaGetLastError());
                            Kc = tiles_new * a.KT;
                            a.K = Kc;
                            gei = row_grid(g.ne, Kc, a.KT, ctx->sm_count);
                            goi = row_grid(g.no, Kc, a.KT, ctx->sm_count);
                            gei2 = row_grid(g.ne, Kc, a.KT, ctx->sm_count, 2);
                            goi2 = row_grid(g.no, Kc, a.KT, ctx->sm_count, 2);
                            gp.reset();  // the poll-window graphs hold the old grid
                            st.compactions++;
                        }
                    }
                }
                if (compacted) {
                    // every array back to the original system order
                    ESL_COUNT_LAUNCH();
                    k_sw_row_perm<<<dim3(perm_blocks, npl), kPermWarps * 32, (size_t)kPermWarps * Kp * 8, s>>>(
                        pl, Kp, Kp, cperm, 1);
                    ESL_CUDA(cudaGetLastError());
                    a.K = K;
                    gei = gei0;
                    goi = goi0;
                    gei2 = gei20;
                    goi2 = goi20;
                }
                group_iters += it;
                ESL_COUNT_LAUNCH();
                k_sw_commit<TT><<<goi, kSwT, 0, s>>>(a, sc.c[C_SCALE], D, X64);
                ESL_CUDA(cudaGetLastError());
                return ESL_OK;
            };
            const int iters_before = group_iters;
            if (inner64) {
                ESL_TRY(run_inner(double{}));
            } else {
                ESL_TRY(run_inner(float{}));
            }
            if (debug_on() && g.ne + g.no > 20000)
                fprintf(stderr, "[esl-sweep]   round %d: %d systems, %d iterations (%s), %.3f ms\n", outer, h_cnt[0],
                        group_iters - iters_before, inner64 ? "fp64" : "fp32", g_ms());
            ESL_TRY(true_residual());
            // an FP32 step that no longer halves the residual: continue in FP64
            if (!inner64 && outer >= 2) inner64 = true;
        }
        // even rows of the group from the odd solution, straight into Z
        a.flags = nullptr;
        a.KT = gKT64;
        ESL_COUNT_LAUNCH();
        k_sw_elim<1, double, double, double><<<ge, kSwT, gsm64, s>>>(a, Bv, X64, Z + (size_t)g.beg * Kp);
        ESL_CUDA(cudaGetLastError());
        if (term) {
            // the SCC's kernel at its positions in the reordering, normalised per system
            double* sums = sc.c[C_D1];
            ESL_CUDA(cudaMemsetAsync(sums, 0, (size_t)Kp * 8, s));
            ESL_COUNT_LAUNCH();
            k_sw_term_out<<<row_grid(rows, Kp, gKT64, ctx->sm_count), kSwT, 0, s>>>(a, P->pos.get(), Z, net->term_states,
                                                                                   y, sums);
            ESL_COUNT_LAUNCH();
            k_sw_term_norm<<<dim3((rows + 255) / 256, K), 256, 0, s>>>(K, net->term_states, g.pos0, rows, sums, y);
            ESL_CUDA(cudaGetLastError());
        }
        h_flags.resize(K);
        std::vector<double> h_rr(K), h_bb(K);
        ESL_CUDA(cudaMemcpyAsync(h_flags.data(), sc.i[I_FLAGS], (size_t)K * 4, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(h_rr.data(), sc.c[C_RR64], (size_t)K * 8, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(h_bb.data(), sc.c[C_BB], (size_t)K * 8, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        double worst = 0.0;
        for (int k = 0; k < K; k++) {
            if (h_flags[k] & SW_FAIL) failed[k] = 1;
            if (h_bb[k] > 0) worst = std::max(worst, std::sqrt(h_rr[k] / h_bb[k]));
        }
        st.relres = std::max(st.relres, worst);
        total_iters += group_iters;
        if (debug_on()) {
            fprintf(stderr, "[esl-sweep] group beg %u even %u odd %u max_scc %d: iters %d relres %.3e, %.3f ms\n",
                    g.beg, g.ne, g.no, g.max_scc, group_iters, worst, g_ms());
            if (g.ne + g.no > 20000) {
                // Krylov iterations per system over all refinement rounds
                std::vector<int> its(K);
                ESL_CUDA(cudaMemcpy(its.data(), sc.i[I_TOTAL], (size_t)K * 4, cudaMemcpyDeviceToHost));
                std::sort(its.begin(), its.end());
                fprintf(stderr, "[esl-sweep]   iterations per system: min %d p50 %d p90 %d p99 %d max %d\n",
                        its.front(), its[K / 2], its[(K * 9) / 10], its[(K * 99) / 100], its.back());
            }
        }
        return ESL_OK;
    };
    bool first_launch = true;
    for (const SwGroup& g : P->groups) {
        if (debug_on()) {
            ESL_CUDA(cudaStreamSynchronize(s));
            g_t0 = std::chrono::steady_clock::now();
        }
        a.beg = g.beg;
        a.ob = g.beg + g.ne;
        a.Qo = a.IQe = nullptr;
        a.ne = g.ne;
        a.no = g.no;
        a.flags = nullptr;
        a.KT = KT64;
        const uint32_t rows = g.ne + g.no;
        a.gam = nullptr;
        a.inv_s = 1.0 / (double)std::max<uint32_t>(rows, 1);
        // singleton SCCs only: a row kernel, or the singleton CTAs of k_sw_scc, whose lanes
        // hold rows when there are fewer than 32 systems
        if (g.kind == 0 && K >= 32) {
            ESL_COUNT_LAUNCH();
            k_sw_rhs<true><<<row_grid(rows, Kp, KT64, ctx->sm_count), kSwT, sm64, s>>>(
                a, P->og_ptr.get(), P->og_ent.get(), x0, x0_ld, Z, nullptr);
            ESL_CUDA(cudaGetLastError());
            continue;
        }
        // (kSccGrid: where the rule lies, see there)
        const bool resident = g.resident && (!g.split || K >= kSccClusterMin);
        if (resident || K <= 32) {
            SccArgs ga{};
            ESL_TRY(scc_args(g, resident, ga));
            st.local_groups++;
            const bool overlap = !first_launch;
            first_launch = false;
            if (resident) ESL_TRY(launch_scc(ctx, P, g, 0, term, overlap, ga));
            else ESL_TRY(launch_scc_grid(ctx, g, term, ga));
            if (debug_on()) {
                ESL_CUDA(cudaStreamSynchronize(s));
                fprintf(stderr, "[esl-sweep] local group beg %u even %u odd %u max_scc %d sccs %u singles %u, %.3f ms\n",
                        g.beg, g.ne, g.no, g.max_scc, g.ns, g.singles, g_ms());
            }
            continue;
        }
        // ---- grid-wide Krylov ----
        // The SCCs of a group share no edge: those beyond a cluster are solved one by one,
        // each with its own coefficients and end, the others and the singletons by k_sw_scc.
        // As one block the group's iterations served the union of the SCCs' spectra on all of
        // its rows (316,541 rows in SCCs of 126,976, 63,488, 63,488, 30,688, 30,688 and fewer
        // states, 512 systems: 420 -> 312 ms).
        std::vector<SwGroup> pieces;
        for (uint32_t j = g.l0; j < g.l0 + g.nlarge; j++) {
            const uint4& c = P->large[j];
            SwGroup q = g;
            q.beg = c.x;
            q.ne = c.y;
            q.ob = c.z;
            q.no = c.w;
            // (the share of the rows, for the measurement hook)
            q.nin = (uint64_t)((double)g.nin * (c.y + c.w) / std::max<uint32_t>(g.ne + g.no, 1));
            pieces.push_back(q);
        }
        if (pieces.size() < g.ns || (!term && g.singles > 0)) {
            SccArgs ga{};
            const bool overlap = !first_launch;
            first_launch = false;
            ESL_TRY(scc_args(g, true, ga));
            st.local_groups++;
            ESL_TRY(launch_scc(ctx, P, g, (uint32_t)pieces.size(), term, overlap, ga));
        }
        for (const SwGroup& q : pieces) ESL_TRY(solve_rows(q));
    }
    // masses into the terminal SCCs
    a.flags = nullptr;
    a.KT = KT64;
    a.gam = nullptr;
    if (!term && P->TS > 0) {
        ESL_COUNT_LAUNCH();
        k_sw_term<<<row_grid((uint32_t)P->TS, Kp, KT64, ctx->sm_count), kSwT, sm64, s>>>(
            a, P->TS, net->order.get(), net->term_of.get(), P->tp_ptr.get(), P->tp_ent.get(), x0, x0_ld, Z, T, y);
        ESL_CUDA(cudaGetLastError());
    }
    // expected occupation by state (the learned warm start's training label)
    if (!term && o.d_occupation && P->M > 0) {
        ESL_COUNT_LAUNCH();
        k_sw_occupation<<<dim3((P->M + 31) / 32, Kp / 32), 256, 0, s>>>(P->M, K, Kp, (size_t)net->N, P->rows.get(), Z,
                                                                        o.d_occupation);
        ESL_CUDA(cudaGetLastError());
    }
    // results of the SCC-resident groups
    if (st.local_groups > 0) {
        std::vector<unsigned char> h_loc(loc_bytes);
        int h_bar[2] = {0, 0};
        ESL_CUDA(cudaMemcpyAsync(h_loc.data(), loc_ratio, loc_bytes, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaMemcpyAsync(h_bar, d_cnt + 8, 8, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        if (h_bar[1]) return fail(ESL_ERR_TIMEOUT, "a grid barrier of the level sweep did not complete in time");
        std::vector<int> h_its(P->groups.size());
        std::memcpy(h_its.data(), h_loc.data() + (size_t)Kp * 12, h_its.size() * 4);
        for (size_t j = 0; j < P->groups.size(); j++) {
            int steps;
            std::memcpy(&steps, h_loc.data() + (size_t)Kp * 12 + (P->groups.size() + j) * 4, 4);
            st.refinements = std::max(st.refinements, steps);
        }
        for (int k = 0; k < K; k++) {
            double ratio;
            int bad;
            std::memcpy(&ratio, h_loc.data() + (size_t)k * 8, 8);
            std::memcpy(&bad, h_loc.data() + (size_t)Kp * 8 + (size_t)k * 4, 4);
            st.relres = std::max(st.relres, std::sqrt(ratio));
            if (bad) failed[k] = 1;
            else st.relres_kept = std::max(st.relres_kept, std::sqrt(ratio));
        }
        // groups of larger SCCs add their iterations, groups of small ones run beside them
        int small = 0;
        for (size_t j = 0; j < h_its.size(); j++) {
            if (P->groups[j].kind == 2)
                total_iters += h_its[j];
            else
                small = std::max(small, h_its[j]);
        }
        total_iters += small;
    }
    st.iters = total_iters;
    st.failed.clear();
    for (int k = 0; k < K; k++)
        if (failed[k]) st.failed.push_back(k);
    if (!st.failed.empty()) {
        char msg[160];
        snprintf(msg, sizeof msg, "level sweep%s: %zu of %d systems above the acceptance residual",
                 term ? " (terminal kernels)" : "", st.failed.size(), K);
        return fail(ESL_ERR_NOT_CONVERGED, msg);
    }
    return ESL_OK;
}

}  // namespace

int sweep_forward(esl_ctx* ctx, const esl_net* net, int K, int nrhs, const double* rates, const double* x0,
                  size_t x0_ld, const esl_solve_opts& o, double* y, SweepStats& st) {
    if (!sweep_supported(net)) return fail(ESL_ERR_TOO_LARGE, "level sweep supports at most 26 nodes");
    SweepPlan* P = nullptr;
    ESL_TRY(build_plan(ctx, net, P));
    return sweep_run(ctx, net, P, false, K, nrhs, rates, x0, x0_ld, o, y, st);
}

// The whole-system form is solved as one resident block while CTA-sized (8,192 transient
// states of a network of at most 13 nodes): its Krylov solve, seven launches per iteration
// however few the states, took 1.2 ms where the block takes 0.3 (n=11, one system).
bool whole_supported(const esl_net* net) {
    return net->n <= 13 && net->N - net->term_states >= 4 && (int64_t)net->term_states < net->N;
}

int sweep_whole(esl_ctx* ctx, const esl_net* net, int K, int nrhs, const double* rates, const double* x0, size_t x0_ld,
                const esl_solve_opts& o, double* y, SweepStats& st) {
    SweepPlan* P = nullptr;
    ESL_TRY(build_whole_plan(ctx, net, false, P));
    if (!P->groups[0].resident || !P->max_even || !P->max_odd)
        return fail(ESL_ERR_NOT_CONVERGED, "the transient part is not one block");
    return sweep_run(ctx, net, P, false, K, nrhs, rates, x0, x0_ld, o, y, st);
}

int sweep_absorption(esl_ctx* ctx, const esl_net* net, const double* rates, const esl_solve_opts& o, double* d_L,
                     SweepStats& st) {
    SweepPlan* P = nullptr;
    ESL_TRY(build_whole_plan(ctx, net, true, P));
    if (!P->groups[0].resident || !P->max_even || !P->max_odd)
        return fail(ESL_ERR_NOT_CONVERGED, "the transient part is not one block");
    const size_t N = (size_t)net->N;
    const int T = net->T, Kp = (T + 31) & ~31;
    if (!ctx->sweep_work) ctx->sweep_work = new Workspace();
    Workspace& ws = *static_cast<Workspace*>(ctx->sweep_work);
    int st_ = ESL_OK;
    double* b = (double*)ws.get(W_BV, (size_t)T * N * 8, &st_);
    if (st_ != ESL_OK) return st_;
    cudaStream_t s = ctx->stream;
    const dim3 grid((unsigned)((N + 255) / 256), T);
    ESL_COUNT_LAUNCH();
    k_sw_back_rhs<<<grid, 256, 0, s>>>(net->n, N, net->F.get(), net->term_of.get(), rates, b);
    ESL_CUDA(cudaGetLastError());
    ESL_TRY(sweep_run(ctx, net, P, false, T, T, rates, b, N, o, nullptr, st));
    const double* Z = (const double*)ws.get(W_Z, (size_t)P->M * Kp * 8, &st_);
    ESL_COUNT_LAUNCH();
    k_sw_scatter_L<<<grid, 256, 0, s>>>(P->M, Kp, N, P->rows.get(), Z, net->term_of.get(), d_L);
    ESL_CUDA(cudaGetLastError());
    return ESL_OK;
}

int sweep_terminal(esl_ctx* ctx, const esl_net* net, int B, const double* rates, const esl_solve_opts& o, double* Rb,
                   SweepStats& st) {
    if (!sweep_supported(net)) return fail(ESL_ERR_TOO_LARGE, "level sweep supports at most 26 nodes");
    SweepPlan* P = nullptr;
    ESL_TRY(build_plan(ctx, net, P));
    if (!P->term) return ESL_OK;
    // terminal kernels can be badly conditioned and cost little next to the transient
    // part: a tighter tolerance and larger budgets than the transient solve's
    esl_solve_opts to = o;
    to.method = ESL_METHOD_DIRECT;
    to.d_warm = nullptr;
    to.d_occupation = nullptr;
    to.tol = std::min(o.tol > 0 ? o.tol : 1e-10, 1e-12);
    to.max_iters = std::max(o.max_iters, 3000);
    to.max_refine = std::max(o.max_refine, 8);
    return sweep_run(ctx, net, P->term, true, B, 1, rates, nullptr, 0, to, Rb, st);
}

}  // namespace esl
