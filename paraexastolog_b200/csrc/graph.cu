// SCC decomposition, terminal SCCs, levels and the vertex reordering, all on the
// device and all driven by the per-state flip masks (no adjacency arrays).
//
// Replaces transition_graph::reorganize_vertices (cuda/src/transition_graph.cu:123-202),
// its SCC solver (cuda/src/sga/two_phase.cu:12-145) and the level labelling
// (cuda/src/kernels/transition_graph.cu:3-27).
//
// Graph: edge s -> s ^ (1<<i) iff bit i of F[s]; edge s ^ (1<<i) -> s iff bit i of G[s].
// SCCs: iterated trim (a state with no live successor or no live predecessor is a
// singleton SCC), then rounds of forward max-priority propagation followed by a backward
// reach within each colour from its root (the state whose colour is its own priority,
// i.e. the largest of its SCC); every round removes at least one SCC per colour.  Labels
// are made canonical afterwards: the label of an SCC is its smallest state, the same
// label the reference gives singletons.
// Levels: level 1 = SCC without out-edges to other SCCs (terminal); otherwise
// 1 + max level of its successor SCCs (the reference's labelling fixpoint).
// Order: terminal SCCs by label ascending, then the others by decreasing level and,
// within a level, decreasing label -- the order the reference's stable sort by
// level and reversal produce (cuda/src/transition_graph.cu:151-184) -- with the
// states of an SCC ascending.
// Every fixpoint loop runs under an iteration budget and fails with ESL_ERR_TIMEOUT.
#include <chrono>
#include <cstdio>
#include <cstdlib>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>

#include "esl_internal.h"

namespace esl {
namespace {

constexpr int kThreads = 256;

inline unsigned blocks_for(uint64_t N) { return (unsigned)((N + kThreads - 1) / kThreads); }

// ---- SCCs, canonical labels and levels in one cooperative launch ---------------------------
// Every fixpoint of the decomposition is monotone, so its states may be relaxed in any
// order and read any mixture of old and new neighbour values: threads run several passes
// over their states between two grid barriers, and the barriers only decide termination
// (a phase in which no state changed).  With a launch per pass and a host read of the flag
// per few passes, launches and reads took most of the time: the n=20 network 27.4 ms (1,587
// launches, 474 reads) against 7.8 ms here, the n=13 one 4.1 against 1.0 ms.  A pass over
// 2^20 states (17 us) is bound by the L2 traffic of the neighbour reads (whole-warp walks of
// the union of flips and four states in flight measured the same), a pass over few states
// by round trips to L2, a level per pass at worst (the n=20 network has 143 levels; the state
// that raises a level raises its own copy in the same pass: 8.9 -> 7.8 ms).
//
// A CTA owns the 32-state chunks c with c % grid == its index, which spreads live states
// evenly, and keeps the list of its live states.  Colours are pseudo-random priorities
// (a bijection of the state index): with the index itself as colour the same network took
// 28 rounds whose live sets shrink 2.5 times slower.
constexpr int kSccT = 1024;
constexpr uint32_t kReached = 0x80000000u;

struct GraphState {        // device, zeroed before the launch
    unsigned arrived;      // grid barrier: arrivals so far
    int status;            // 0, or 1: a budget ran out, 2: a barrier wait ran out
    unsigned changed[3];   // by phase % 3
    unsigned live[3];      // by round % 3
    unsigned rounds, phases;
};

struct GraphArgs {
    int n;
    uint32_t N;
    const uint32_t *F, *G;
    int32_t* lab;
    uint32_t* color;   // 0: dead; priority + 1, kReached once it reaches its colour's root
    int32_t* canon;
    int32_t* level;
    uint32_t* list;    // grid x cap
    uint32_t cap;      // states per CTA
    uint64_t* keys;
    int32_t* vals;
    int64_t budget;    // phases per fixpoint
    unsigned polls;    // bound of a barrier wait
    unsigned missing;  // arrivals that never come (0, or 1 when the bounded wait is tested)
    GraphState* st;
};

// Bijection of [0, 2^n): odd multiplications and xor-shifts
__device__ __forceinline__ uint32_t priority_of(uint32_t v, int n) {
    const uint32_t m = (1u << n) - 1u;
    const int h = max(n >> 1, 1);
    v = (v * 0x9E3779B1u) & m;
    v ^= v >> h;
    v = (v * 0x85EBCA6Bu) & m;
    v ^= v >> (h + 1);
    return (v * 0xC2B2AE35u) & m;
}

// Grid barrier with a bounded wait; false once the launch has failed anywhere.  One thread
// reads the status for its CTA: threads that read it themselves could see it change between
// their reads, and part of a CTA would leave while the rest waits for it.
__device__ bool grid_barrier(const GraphArgs& g, unsigned& target) {
    __shared__ bool s_ok;
    GraphState* st = g.st;
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&st->arrived, 1u);
        unsigned polls = 0;
        // (the difference, not the order: the arrivals may wrap around)
        while ((int)(*(volatile unsigned*)&st->arrived - target) < 0 && *(volatile int*)&st->status != 2)
            if (++polls > g.polls) atomicExch(&st->status, 2);
        __threadfence();
        s_ok = *(volatile int*)&st->status == 0;
    }
    __syncthreads();
    return s_ok;
}

// Calls fn on the values of arr at the neighbours of v in mask, eight at a time (0 past the
// last), until it returns true.  A pass over few states is a chain of L2 round trips:
// eight loads in flight make it one or two of them.
template <class Fn>
__device__ __forceinline__ void for_neighbours(uint32_t v, uint32_t mask, const uint32_t* arr, Fn fn) {
    while (mask) {
        uint32_t x[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t bit = mask & (0u - mask);
            x[j] = bit ? __ldcg(arr + (v ^ bit)) : 0u;
            mask ^= bit;
        }
        if (fn(x)) return;
    }
}

__global__ void __launch_bounds__(kSccT, 1) k_scc(const GraphArgs g) {
    const uint32_t tid = threadIdx.x, cta = blockIdx.x, ctas = gridDim.x;
    GraphState* st = g.st;
    uint32_t* list = g.list + (size_t)cta * g.cap;
    __shared__ unsigned s_warp[kSccT / 32 + 1];
    unsigned target = g.missing, phase = 0;
    // state i of this CTA
    auto state_at = [&](uint32_t i) { return ((i >> 5) * ctas + cta) * 32u + (i & 31u); };
    const uint32_t chunks = (g.N + 31) / 32;
    const uint32_t own = (chunks / ctas + (cta < chunks % ctas ? 1u : 0u)) * 32u;
    // keeps the states of the list with a nonzero colour; returns their count
    auto compact = [&](uint32_t count, bool init) {
        uint32_t kept = 0;
        for (uint32_t i0 = 0; i0 < count; i0 += kSccT) {
            const uint32_t i = i0 + tid;
            uint32_t v = 0;
            bool keep = false;
            if (i < count) {
                v = init ? state_at(i) : list[i];
                keep = v < g.N && (init || __ldcg(g.color + v) != 0u);
            }
            const unsigned m = __ballot_sync(0xFFFFFFFFu, keep);
            if ((tid & 31) == 0) s_warp[tid >> 5] = __popc(m);
            __syncthreads();
            if (tid < 32) {
                unsigned x = s_warp[tid], y = x;
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned z = __shfl_up_sync(0xFFFFFFFFu, y, o);
                    if ((int)tid >= o) y += z;
                }
                s_warp[tid] = y - x;
                if (tid == 31) s_warp[32] = y;
            }
            __syncthreads();
            if (keep) list[kept + s_warp[tid >> 5] + __popc(m & ((1u << (tid & 31)) - 1u))] = v;
            kept += s_warp[32];
            __syncthreads();
        }
        return kept;
    };
    // Runs pass(place) over the CTA's first `count` list places until a whole phase changes
    // nothing: `passes` sweeps per phase while the states are few (a sweep is then shorter
    // than a barrier).  `seeded`: this thread changed states that the passes read since the
    // last barrier, which the first phase may not see everywhere, so that it does not count.
    // A phase gets at least as far as one sweep that reads only what the phase before it left;
    // the budget is in such sweeps.  False: failed.
    auto fixpoint = [&](uint32_t count, unsigned passes, bool after_seeds, bool seeded, int64_t budget, auto pass) -> bool {
        bool ch = seeded;
        for (int64_t used = after_seeds ? 0 : 1;; ch = false, used++) {
            for (unsigned k = 0; k < passes; k++)
                for (uint32_t i = tid; i < count; i += kSccT) ch |= pass(i);
            if (cta == 0 && tid == 0) st->changed[(phase + 1) % 3] = 0;
            if (__syncthreads_or(ch) && tid == 0) st->changed[phase % 3] = 1;
            if (!grid_barrier(g, target)) return false;
            const unsigned any = *(volatile unsigned*)&st->changed[phase % 3];
            phase++;
            if (!any) return true;
            if (used >= budget) {
                if (tid == 0) atomicCAS(&st->status, 0, 1);
                // every CTA sees the same flag and budget: all leave here
                return false;
            }
        }
    };
    uint32_t count = compact(own, true);
    for (uint32_t i = tid; i < count; i += kSccT) {
        const uint32_t v = list[i];
        g.color[v] = 1u;  // live
        g.canon[v] = 0x7FFFFFFF;
        g.level[v] = 1;
    }
    if (!grid_barrier(g, target)) return;
    uint32_t live = g.N;
    unsigned round = 0;
    bool seeded = false;
    // a state without a live successor or without a live predecessor is its own SCC
    auto trim = [&](uint32_t i) {
        const uint32_t v = list[i];
        if (__ldcg(g.color + v) == 0u) return false;
        bool out = false, in = false;
        auto alive = [](bool& hit) {
            return [&hit](const uint32_t (&x)[8]) {
                hit = (x[0] | x[1] | x[2] | x[3] | x[4] | x[5] | x[6] | x[7]) != 0u;
                return hit;
            };
        };
        for_neighbours(v, g.F[v], g.color, alive(out));
        if (out) for_neighbours(v, g.G[v], g.color, alive(in));
        if (in) return false;
        g.lab[v] = (int32_t)priority_of(v, g.n);
        __stcg(g.color + v, 0u);
        return true;
    };
    for (;; round++) {
        const unsigned passes = live > 2u * kSccT * ctas ? 1u : 4u;
        if (!fixpoint(count, passes, round > 0, seeded, g.budget, trim)) return;
        count = compact(count, false);
        if (cta == 0 && tid == 0) st->live[(round + 1) % 3] = 0;
        if (tid == 0 && count) atomicAdd(&st->live[round % 3], count);
        for (uint32_t i = tid; i < count; i += kSccT) __stcg(g.color + list[i], priority_of(list[i], g.n) + 1u);
        if (!grid_barrier(g, target)) return;
        live = *(volatile unsigned*)&st->live[round % 3];
        if (live == 0) break;
        // largest priority among the live ancestors
        if (!fixpoint(count, passes, false, false, g.budget, [&](uint32_t i) {
                const uint32_t v = list[i], c = __ldcg(g.color + v);
                uint32_t m = c;
                for_neighbours(v, g.G[v], g.color, [&](const uint32_t (&x)[8]) {
#pragma unroll
                    for (int j = 0; j < 8; j++) m = max(m, x[j]);
                    return false;
                });
                if (m > c) __stcg(g.color + v, m);
                return m > c;
            }))
            return;
        // backward from each colour's root (the state of that priority) within the colour
        seeded = false;
        for (uint32_t i = tid; i < count; i += kSccT) {
            const uint32_t v = list[i], c = priority_of(v, g.n) + 1u;
            if (__ldcg(g.color + v) == c) {
                __stcg(g.color + v, c | kReached);
                seeded = true;
            }
        }
        if (!fixpoint(count, passes, true, seeded, g.budget, [&](uint32_t i) {
                const uint32_t v = list[i], c = __ldcg(g.color + v);
                if (c & kReached) return false;
                bool hit = false;
                for_neighbours(v, g.F[v], g.color, [&](const uint32_t (&x)[8]) {
#pragma unroll
                    for (int j = 0; j < 8; j++) hit |= x[j] == (c | kReached);
                    return hit;
                });
                if (hit) __stcg(g.color + v, c | kReached);
                return hit;
            }))
            return;
        seeded = false;
        for (uint32_t i = tid; i < count; i += kSccT) {
            const uint32_t v = list[i], c = __ldcg(g.color + v);
            if (c & kReached) {
                g.lab[v] = (int32_t)((c & ~kReached) - 1u);
                __stcg(g.color + v, 0u);
                seeded = true;
            }
        }
    }
    if (cta == 0 && tid == 0) {
        st->rounds = round;
        st->phases = phase;
    }
    // canonical labels: smallest state of each SCC
    for (uint32_t i = tid; i < own; i += kSccT) {
        const uint32_t v = state_at(i);
        if (v < g.N) atomicMin(&g.canon[g.lab[v]], (int32_t)v);
    }
    if (!grid_barrier(g, target)) return;
    for (uint32_t i = tid; i < own; i += kSccT) {
        const uint32_t v = state_at(i);
        if (v < g.N) g.lab[v] = __ldcg(g.canon + g.lab[v]);
    }
    if (!grid_barrier(g, target)) return;
    // levels, stored at the SCC's label: 1 + the largest level among successor SCCs.  The
    // list takes each state's flips that leave its SCC, the colours a copy of its SCC's
    // level, which neighbours read without going through the label.  The state that raises its
    // SCC's level raises its own copy with it, the SCC's other states theirs a pass later: a
    // level costs one pass behind singletons and two behind larger SCCs, hence twice the budget.
    for (uint32_t i = tid; i < own; i += kSccT) {
        const uint32_t v = state_at(i);
        uint32_t x = 0;
        if (v < g.N) {
            const int32_t c = g.lab[v];
            for (uint32_t f = g.F[v]; f; f &= f - 1) {
                const uint32_t bit = f & (0u - f);
                if (__ldcg(g.lab + (v ^ bit)) != c) x |= bit;
            }
            __stcg(g.color + v, 1u);
        }
        list[i] = x;
    }
    if (!grid_barrier(g, target)) return;
    if (!fixpoint(own, g.N > 2u * kSccT * ctas ? 1u : 4u, false, false, 2 * g.budget, [&](uint32_t i) {
            const uint32_t v = state_at(i);
            if (v >= g.N) return false;
            const int32_t c = g.lab[v];
            const uint32_t l = (uint32_t)__ldcg(g.level + c);
            bool ch = false;
            if (l > __ldcg(g.color + v)) {
                __stcg(g.color + v, l);
                ch = true;
            }
            uint32_t best = 0;
            for_neighbours(v, list[i], g.color, [&](const uint32_t (&x)[8]) {
#pragma unroll
                for (int j = 0; j < 8; j++) best = max(best, x[j]);
                return false;
            });
            if (best >= l && best > 0) {
                atomicMax(&g.level[c], (int32_t)best + 1);
                __stcg(g.color + v, best + 1);
                ch = true;
            }
            return ch;
        }))
        return;
    // sort key: terminal -> label; other -> (1, MAXLVL - level, MAXLBL - label)
    for (uint32_t i = tid; i < own; i += kSccT) {
        const uint32_t v = state_at(i);
        if (v >= g.N) continue;
        const int32_t c = g.lab[v], l = __ldcg(g.level + c);
        g.keys[v] = l == 1 ? (uint64_t)c
                           : (1ull << 62) | ((uint64_t)(0x3FFFFFFF - l) << 31) | (uint64_t)(0x7FFFFFFF - c);
        g.vals[v] = (int32_t)v;
    }
}

__global__ void k_heads(uint64_t N, const uint64_t* __restrict__ keys, int32_t* __restrict__ pos_out,
                        uint8_t* __restrict__ head) {
    uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= N) return;
    head[p] = (p == 0 || keys[p] != keys[p - 1]) ? 1 : 0;
    pos_out[p] = (int32_t)p;
}

__global__ void k_scc_levels(int n_sccs, const int32_t* __restrict__ offsets, const int32_t* __restrict__ order,
                             const int32_t* __restrict__ lab, const int32_t* __restrict__ level_by_label,
                             int32_t* __restrict__ level_at) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_sccs) return;
    level_at[k] = level_by_label[lab[order[offsets[k]]]];
}

__global__ void k_term_of(uint64_t N, int T, int term_states, const int32_t* __restrict__ offsets,
                          const int32_t* __restrict__ order, int32_t* __restrict__ term_of) {
    uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= N) return;
    if ((int64_t)p >= term_states) {
        term_of[order[p]] = -1;
        return;
    }
    int lo = 0, hi = T;  // offsets[lo] <= p < offsets[hi]
    while (hi - lo > 1) {
        int mid = (lo + hi) / 2;
        if (offsets[mid] <= (int32_t)p) lo = mid; else hi = mid;
    }
    term_of[order[p]] = lo;
}

// same-class masks: a neighbour counts only if both states are transient or both in
// the same terminal SCC
__global__ void k_domain_masks(int n, uint64_t N, const uint32_t* __restrict__ F, const uint32_t* __restrict__ G,
                               const int32_t* __restrict__ term_of, uint32_t* __restrict__ Fd,
                               uint32_t* __restrict__ Gd) {
    uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= N) return;
    int32_t c = term_of[v];
    uint32_t f = F[v], g = G[v], fd = 0, gd = 0;
    for (int i = 0; i < n; i++) {
        uint32_t b = 1u << i;
        if ((f | g) & b) {
            bool same = term_of[v ^ (1ull << i)] == c;
            if (same && (f & b)) fd |= b;
            if (same && (g & b)) gd |= b;
        }
    }
    Fd[v] = fd;
    Gd[v] = gd;
}

}  // namespace

int sort_pairs(const uint64_t* keys, uint64_t* keys_out, const int32_t* vals, int32_t* vals_out, size_t count,
               DevBuf<uint8_t>& tmp, cudaStream_t s) {
    size_t bytes = 0;
    ESL_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, keys, keys_out, vals, vals_out, (int64_t)count, 0, 64, s));
    if (tmp.n < bytes) ESL_TRY(tmp.alloc(bytes));
    ESL_CUDA(cub::DeviceRadixSort::SortPairs(tmp.get(), bytes, keys, keys_out, vals, vals_out, (int64_t)count, 0, 64, s));
    return ESL_OK;
}

bool barrier_timeout_test() {
    const char* e = getenv("ESL_BARRIER_TIMEOUT_TEST");
    return e && e[0] == '1';
}

int build_graph(esl_ctx* ctx, esl_net* net) {
    const uint64_t N = (uint64_t)net->N;
    const int n = net->n;
    cudaStream_t s = ctx->stream;
    const unsigned nb = blocks_for(N);
    const uint32_t* F = net->F.get();
    const uint32_t* G = net->G.get();
    const bool dbg = getenv("ESL_DEBUG") != nullptr;
    const auto t0 = std::chrono::steady_clock::now();
    auto ms_since = [&]() {
        return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    };
    ESL_TRY(net->labels.alloc(N));
    int32_t* lab = net->labels.get();
    DevBuf<int32_t> level;
    DevBuf<uint64_t> keys;
    DevBuf<int32_t> vals;
    ESL_TRY(level.alloc(N));
    ESL_TRY(keys.alloc(N));
    ESL_TRY(vals.alloc(N));
    {
        DevBuf<uint32_t> color, list;
        DevBuf<int32_t> canon;
        DevBuf<GraphState> state;
        ESL_TRY(color.alloc(N));
        ESL_TRY(canon.alloc(N));
        ESL_TRY(state.alloc(1));
        GraphArgs ga{};
        // one state per thread while that leaves SMs free: fewer CTAs, shorter barriers
        const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)ctx->sm_count, (N + kSccT - 1) / kSccT);
        ga.n = n;
        ga.N = (uint32_t)N;
        ga.F = F;
        ga.G = G;
        ga.lab = lab;
        ga.color = color.get();
        ga.canon = canon.get();
        ga.level = level.get();
        ga.cap = (uint32_t)(((N + 31) / 32 + grid - 1) / grid * 32);
        ESL_TRY(list.alloc((size_t)ga.cap * grid));
        ga.list = list.get();
        ga.keys = keys.get();
        ga.vals = vals.get();
        // a sweep can only fail to progress once per state (or the context's budget)
        ga.budget = ctx->graph_sweeps > 0 ? ctx->graph_sweeps : (int64_t)N + 64;
        ga.st = state.get();
        const bool no_end = barrier_timeout_test();
        ga.polls = no_end ? kBarrierTestPolls : kBarrierPolls;
        ga.missing = no_end ? 1 : 0;
        ESL_CUDA(cudaMemsetAsync(state.get(), 0, sizeof(GraphState), s));
        GraphState h{};
        {
            // nominal algorithmic bytes (measurement hook): masks, label, colour and level
            // of every state once
            ProfScope ps(ctx, "graph_sweep", 24.0 * (double)N);
            void* args[] = {&ga};
            ESL_COUNT_LAUNCH();
            ESL_CUDA(cudaLaunchCooperativeKernel((const void*)k_scc, dim3(grid), dim3(kSccT), args, 0, s));
        }
        ESL_CUDA(cudaMemcpyAsync(&h, state.get(), sizeof h, cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        if (h.status == 1) return fail(ESL_ERR_TIMEOUT, "fixpoint budget exceeded in the SCC decomposition or the levels");
        if (h.status) return fail(ESL_ERR_TIMEOUT, "a grid barrier of the SCC decomposition did not complete in time");
        if (dbg)
            fprintf(stderr, "[esl-graph] SCCs and levels: %u rounds, %u phases, %.1f ms\n", h.rounds, h.phases, ms_since());
    }

    // ordering by a stable radix sort of (class, level, label) keys
    {
        DevBuf<uint64_t> keys_out;
        DevBuf<int32_t> pos;
        DevBuf<uint8_t> head;
        ESL_TRY(keys_out.alloc(N));
        ESL_TRY(net->order.alloc(N));
        DevBuf<uint8_t> tmp;
        ESL_TRY(sort_pairs(keys.get(), keys_out.get(), vals.get(), net->order.get(), N, tmp, s));
        // SCC heads
        ESL_TRY(pos.alloc(N));
        ESL_TRY(head.alloc(N));
        ESL_COUNT_LAUNCH();
        k_heads<<<nb, kThreads, 0, s>>>(N, keys_out.get(), pos.get(), head.get());
        ESL_CUDA(cudaGetLastError());
        DevBuf<int32_t> offs;
        DevBuf<int64_t> d_count;
        ESL_TRY(offs.alloc(N + 1));
        ESL_TRY(d_count.alloc(1));
        size_t sel_bytes = 0;
        ESL_CUDA(cub::DeviceSelect::Flagged(nullptr, sel_bytes, pos.get(), head.get(), offs.get(), d_count.get(),
                                            (int64_t)N, s));
        DevBuf<uint8_t> tmp2;
        ESL_TRY(tmp2.alloc(sel_bytes));
        ESL_CUDA(cub::DeviceSelect::Flagged(tmp2.get(), sel_bytes, pos.get(), head.get(), offs.get(), d_count.get(),
                                            (int64_t)N, s));
        int64_t n_sccs = 0;
        ESL_CUDA(cudaMemcpyAsync(&n_sccs, d_count.get(), sizeof(int64_t), cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        net->n_sccs = (int)n_sccs;
        ESL_TRY(net->offsets.alloc(n_sccs + 1));
        ESL_CUDA(cudaMemcpyAsync(net->offsets.get(), offs.get(), n_sccs * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
        int32_t Nend = (int32_t)N;
        ESL_CUDA(cudaMemcpyAsync(net->offsets.get() + n_sccs, &Nend, sizeof(int32_t), cudaMemcpyHostToDevice, s));
        ESL_TRY(net->levels.alloc(n_sccs));
        ESL_COUNT_LAUNCH();
        k_scc_levels<<<(unsigned)((n_sccs + kThreads - 1) / kThreads), kThreads, 0, s>>>(
            (int)n_sccs, net->offsets.get(), net->order.get(), lab, level.get(), net->levels.get());
        ESL_CUDA(cudaGetLastError());
        // terminal count: leading SCCs with level 1
        std::vector<int32_t> h_lv(n_sccs);
        ESL_CUDA(cudaMemcpyAsync(h_lv.data(), net->levels.get(), n_sccs * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        int T = 0;
        while (T < n_sccs && h_lv[T] == 1) T++;
        net->T = T;
        net->h_offsets.resize(T + 1);
        ESL_CUDA(cudaMemcpyAsync(net->h_offsets.data(), net->offsets.get(), (T + 1) * sizeof(int32_t),
                                 cudaMemcpyDeviceToHost, s));
        ESL_CUDA(cudaStreamSynchronize(s));
        net->term_states = net->h_offsets[T];
        net->max_terminal = 0;
        for (int t = 0; t < T; t++)
            net->max_terminal = std::max(net->max_terminal, net->h_offsets[t + 1] - net->h_offsets[t]);
    }
    ESL_TRY(net->term_of.alloc(N));
    ESL_COUNT_LAUNCH();
    k_term_of<<<nb, kThreads, 0, s>>>(N, net->T, net->term_states, net->offsets.get(), net->order.get(),
                                      net->term_of.get());
    ESL_CUDA(cudaGetLastError());
    ESL_TRY(net->Fdom.alloc(N));
    ESL_TRY(net->Gdom.alloc(N));
    ESL_COUNT_LAUNCH();
    k_domain_masks<<<nb, kThreads, 0, s>>>(n, N, F, G, net->term_of.get(), net->Fdom.get(), net->Gdom.get());
    ESL_CUDA(cudaGetLastError());
    ESL_CUDA(cudaStreamSynchronize(s));
    if (dbg) fprintf(stderr, "[esl-graph] done: %.1f ms\n", ms_since());
    return ESL_OK;
}

}  // namespace esl
