// Host rules of the SCC-resident solver (k_sw_scc in sweep.cu): sizes and launch shapes,
// without CUDA types, so that they can be checked on a machine without a GPU.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define ESL_HD __host__ __device__
#else
#define ESL_HD
#endif

namespace esl {

constexpr int kSccMaxRows = 4096;  // most odd (or even) rows of an SCC solved by one CTA
// threads of a CTA with one row per thread (128 registers each), and with several
constexpr int kSccThreads = 512, kSccThreadsBig = 1024;
constexpr int kSccBuckets = 16;    // most (KS, team size) pairs of a launch
constexpr size_t kSccMaxSmem = 227 * 1024;
// (row, system) pairs of a small SCC's team at most: n=12 x 64 rate sets, one n=22 solve and
// n=17 x 185 systems 1.22, 36.6 and 12.9 ms; 128: 1.22, 36.2, 12.8; 512: 1.26, 37.5, 12.9
constexpr int kSccPairs = 256;
// Shared memory of an elimination (it takes fewer systems above that: 24 KB 1.217 ms at n=12 x 64,
// 12 KB 1.232, 48 KB 1.218), and of the teams of a CTA (two CTAs per SM; 55 and 220 KB are within
// 1% of it in the cases above)
constexpr size_t kSccDenseSmem = 24 * 1024, kSccTeamSmem = 110 * 1024;

// SCCs of at most kSccDense odd rows are solved by elimination: a Krylov iteration is a
// chain of FP64 reductions, about 4 us however small the SCC, an elimination step one
// barrier and a division (n=12 x 64 rate sets 1.93 -> 1.5 ms; at 32 rows the steps cost as
// much as the iterations, n=22 67 -> 61 ms).  A budget of fewer iterations than rows is too
// small for it.
constexpr int kSccDense = 16;
ESL_HD inline bool scc_dense(int so, int max_iters) { return so <= kSccDense && so <= max_iters; }
ESL_HD inline int scc_dense_ld(int so) { return (so + 1) | 1; }

// shared-memory doubles of a work item (see the carving in k_sw_scc)
ESL_HD inline size_t scc_smem_doubles(bool big, bool dense, int n, int se, int so, int lks, int nact) {
    const size_t m = (size_t)(se > so ? se : so), KS = (size_t)1 << lks;
    return (m + 1 + se + 1 + 2 * n + 6 * (size_t)(nact >> 5) + (big ? 4 * (size_t)so + se : 0) +
            (dense ? (size_t)so * scc_dense_ld(so) + 2 : 0)) *
           KS;
}

// Group-sized vectors that k_sw_scc keeps in memory, in the order of SccArgs::own.  The
// first five are per odd row (kSccBig); kSccGrid uses all of them.
enum SccOwn { kOwnR0, kOwnD, kOwnDS, kOwnQ, kOwnBS, kOwnA, kOwnW, kOwnR, kOwnV, kOwnP, kOwnT, kOwnIQ, kOwnCount };

// Rows of vector j in a group of `even` and `odd` rows.  kOwnA holds odd rows while an
// operator is applied to it, and 1 / q of the even rows before that.
inline uint32_t scc_own_rows(int j, uint32_t even, uint32_t odd) {
    const uint32_t rows = j == kOwnW || j == kOwnIQ ? even : j == kOwnA ? std::max(even, odd) : odd;
    return std::max<uint32_t>(rows, 1);
}

// ---- the launch of the SCCs that fit a CTA -------------------------------------------------
// A work item is (SCC, KS = 1 << lks systems).  The SCCs of a launch, largest first, are cut
// into buckets of one KS and team size.
struct SccBucket {
    uint32_t cta0, items;  // first CTA, work items
    uint32_t scc0;         // first SCC of the group's list
    uint32_t stride;       // doubles of shared memory per team
    uint8_t lks, lteam;    // log2 KS, log2 threads of a team
    uint8_t teams;         // teams per CTA
};

// consecutive SCCs of the same numbers of rows
struct SccShape {
    uint32_t even, odd, count;
};

// SCCs whose lines of predecessor entries (SweepPlan::ell) hold their own rows only, not 32.
// Such a row has at most 2 lines (4 entries each), which the solver keeps in registers; a width
// that also varies in its loops cost 2% (n=12 x 64 rate sets 1.15 -> 1.17 ms).  At 32 always, the
// 524,287 SCCs of two states of one free node beside 19 that decay took 512 MB, 16 MB this way.
ESL_HD inline bool scc_narrow(uint32_t even, uint32_t odd) { return even <= 8 && odd <= 8; }

// Order of the SCC list: by group, then by decreasing max(even, odd), so that the launch of a
// group begins with its largest SCCs (it lasts as long as their CTAs, which must not start
// behind the small ones), then by the other parity, so that equal shapes follow one another
// (for larger SCCs at times interrupted by others, which costs a shape more).
ESL_HD inline uint64_t scc_sort_key(uint32_t group, uint32_t even, uint32_t odd) {
    const uint32_t most = even > odd ? even : odd, least = even > odd ? odd : even;
    return (uint64_t)group << 38 | (uint64_t)(0x3FFFFFFu - most) << 12 | (uint64_t)(least & 0x7FFu) << 1 | (odd > even ? 1u : 0u);
}

struct SccLaunch {
    SccBucket b[kSccBuckets];
    int nb = 0;
    uint32_t ctas = 0;
    int threads = 32;
    size_t smem = 0;  // bytes per CTA
};

// Plans the launch of `count` shapes that begin with SCC scc0 of the group, in order of
// decreasing max(even, odd): all of more than kSccThreads rows (big) or none.  false: too many
// work items.
// KS is the largest power of two that keeps (row, system) pairs of small SCCs within kSccPairs
// threads; large SCCs, one CTA per SM, take more systems while shared memory holds them and the
// SMs stay filled.  An SCC joins the bucket before it where that one's KS is larger and fits
// (the footprint of unequal parities is not monotone in the order), and all that is left joins
// the last bucket, at the smallest KS among them.
inline bool plan_scc_launch(const SccShape* shapes, size_t count, uint32_t scc0, bool big, bool defl, int K, int n,
                            int max_iters, int sm_count, SccLaunch& L) {
    L = SccLaunch();
    int lmax = 0;
    while (lmax < 5 && (1 << lmax) < K) lmax++;
    uint64_t total = 0;
    for (size_t j = 0; j < count; j++) total += shapes[j].count;
    const size_t limit = big ? kSccMaxSmem : kSccTeamSmem;
    auto rows = [&](const SccShape& s) { return (int)std::max(s.even, s.odd); };
    auto team = [&](const SccShape& s, int lks) {
        int t = big ? 10 : 5;
        while (!big && (1 << t) < (rows(s) << lks)) t++;
        return t;
    };
    auto is_dense = [&](const SccShape& s) { return !big && !defl && scc_dense((int)s.odd, max_iters); };
    auto doubles = [&](const SccShape& s, int lks, int lteam) {
        return scc_smem_doubles(big, is_dense(s), n, (int)s.even, (int)s.odd, lks, 1 << lteam);
    };
    auto fits = [&](const SccShape& s, int lks, size_t bytes) { return doubles(s, lks, team(s, lks)) * 8 <= bytes; };
    auto own_lks = [&](const SccShape& s) {
        int l = 0;
        if (big)
            while (l < lmax && fits(s, l + 1, kSccMaxSmem) &&
                   total * (uint64_t)((K + (2 << l) - 1) >> (l + 1)) >= (uint64_t)sm_count)
                l++;
        else
            while (l < lmax && (rows(s) << (l + 1)) <= kSccPairs && (!is_dense(s) || fits(s, l + 1, kSccDenseSmem))) l++;
        return l;
    };
    uint64_t all = 0;
    uint32_t scc = scc0;
    for (size_t j = 0; j < count; j++) {
        const SccShape& s = shapes[j];
        SccBucket* last = L.nb > 0 ? &L.b[L.nb - 1] : nullptr;
        int lks, lteam;
        if (L.nb == kSccBuckets) {
            lks = last->lks;
            lteam = last->lteam;
        } else {
            lks = own_lks(s);
            if (last && last->lks > lks && fits(s, last->lks, limit)) lks = last->lks;
            lteam = team(s, lks);
            if (!last || last->lks != lks || last->lteam != lteam) {
                if (L.nb + 1 == kSccBuckets) {
                    for (size_t i = j; i < count; i++) lks = std::min(lks, own_lks(shapes[i]));
                    for (size_t i = j; i < count; i++) lteam = std::max(i == j ? 0 : lteam, team(shapes[i], lks));
                }
                L.b[L.nb++] = SccBucket{0, 0, scc, 0, (uint8_t)lks, (uint8_t)lteam, 1};
                last = &L.b[L.nb - 1];
            }
        }
        all += (uint64_t)s.count * (uint64_t)((K + (1 << lks) - 1) >> lks);
        if (all > 0x3FFFFFFFull) return false;
        last->items += s.count * (uint32_t)((K + (1 << lks) - 1) >> lks);
        last->stride = std::max(last->stride, (uint32_t)doubles(s, lks, lteam));
        scc += s.count;
    }
    // Items share CTAs once there are more of them than SMs; a CTA then has the threads of the
    // largest team at least
    for (int j = 0; j < L.nb; j++) L.threads = std::max(L.threads, 1 << L.b[j].lteam);
    const bool share = !big && all > (uint64_t)sm_count;
    if (share) L.threads = std::max(L.threads, kSccPairs);
    for (int j = 0; j < L.nb; j++) {
        SccBucket& b = L.b[j];
        if (share)
            b.teams = (uint8_t)std::max<size_t>(
                1, std::min<size_t>({(size_t)(L.threads >> b.lteam), (size_t)16, kSccTeamSmem / ((size_t)b.stride * 8)}));
        b.cta0 = L.ctas;
        L.ctas += (b.items + b.teams - 1) / b.teams;
        L.smem = std::max(L.smem, (size_t)b.teams * b.stride * 8);
    }
    return true;
}

}  // namespace esl
