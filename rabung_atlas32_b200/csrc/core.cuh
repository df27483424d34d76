#pragma once
// core.cuh -- host planning and one census call of librabung_census.so, for
// one prime word width.  Included once by census.cu (p < 2^32, 32-bit words,
// handle cz_handle, records cz_profile) and once by census_wide.cu (CZ_WIDE:
// p < 2^33, 64-bit words, handle cz_handle64, records cz_profile64), so the
// two domains share every line of planning, routing, waves, re-runs and
// kernel launches.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"
#include "labels.cuh"
#include "dense.cuh"
#include "table.cuh"
#include "sparse.cuh"
#include "group.cuh"
#include "finalize.cuh"
#include "a4.cuh"
#include "../../include/rabung_census.h"

#if CZ_WIDE
#define CZ_HANDLE cz_handle64
#define CZ_RECORD cz_profile64
#else
#define CZ_HANDLE cz_handle
#define CZ_RECORD cz_profile
#endif

using namespace CZ_NS;

namespace {

constexpr u32 CHAIN_LIMIT = (1u << 20) + 8192u;   // table labels cover n < CHAIN_LIMIT
constexpr u32 B_MAX = (1u << 20);
constexpr u64 PW_LIMIT = CZ_WIDE ? (1ull << 33) : (1ull << 32);   // primes of this build lie below
constexpr u32 TABLE_DYN_SMEM = 190u * 1024u;        // dynamic part; static part ~34 KB

struct Buf {
    void *p = nullptr;
    size_t cap = 0;
};

bool cover_cert(u64 B, u64 D, u64 H, u64 p) {
    if (H * D > 2 * B) return false;
    const unsigned __int128 lhs = (unsigned __int128)4 * B * D - (unsigned __int128)H * D * D;
    return lhs > (unsigned __int128)4 * p;
}

// table radius for a prime: D = floor(2 sqrt(p/H) / n), B = floor((4p + H D^2)/(4D)) + 1
// (the reference's lower-branch choice, paper/GPU_METHOD_EN.tex "Choosing parameters";
// P/src/clipped_cover.hpp:14-21), certified in integers.
bool cover_B(u64 p, u32 Q, u32 ndiv, u32 &Bout) {
    const u64 H = Q - 1u;
    const double D0 = 2.0 * std::sqrt((double)p / (double)H);
    u64 D = (u64)(D0 / (double)ndiv);
    if (D < 1) D = 1;
    const u64 B = (4ull * p + H * D * D) / (4ull * D) + 1ull;
    if (B >= p || D >= p || B > B_MAX) return false;
    if (!cover_cert(B, D, H, p)) return false;
    Bout = (u32)B;
    return true;
}

// least D with the certificate for (p, B, Q)
bool cover_D(u64 p, u32 B, u32 Q, u32 &Dout) {
    const u64 H = Q - 1u;
    const long double disc = (long double)B * B - (long double)H * p;
    if (disc <= 0) return false;
    long double est = (2.0L * B - 2.0L * std::sqrt(disc)) / (long double)H;
    u64 D = est < 1 ? 1 : (u64)est;
    while (D > 1 && cover_cert(B, D - 1, H, p)) --D;
    while (!cover_cert(B, D, H, p)) {
        ++D;
        if (H * D > 2ull * B || D >= p || D > B_MAX) return false;
    }
    Dout = (u32)D;
    return true;
}

u32 popc(u32 x) { return (u32)__builtin_popcount(x); }

// one launch with its own error code: a launch failure is reported through the
// return value, and an error the caller left pending is neither read nor cleared
template <class... A>
bool launch(void (*k)(A...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    void *argv[] = {static_cast<void *>(&args)...};
    return cudaLaunchKernel(reinterpret_cast<const void *>(k), grid, block, argv, smem, st) == cudaSuccess;
}

}  // namespace

struct CZ_HANDLE {
    cz_config cfg{};
    int dev = 0;
    int sms = 148;
    cudaStream_t st = nullptr;
    cudaStream_t st2 = nullptr;         // A4 counts beside the filter
    cudaEvent_t fork = nullptr, join = nullptr;
    std::string err;
    u32 *d_small = nullptr;
    uint2 *d_chain = nullptr;
    u32 n_small = 0;
    // device memory of the current plan: descriptors and results in b_small (one
    // copy in, one copy out), tables in b_big; the others below are places in them
    Buf b_small, b_big;
    size_t up_bytes = 0, down_off = 0, down_bytes = 0;
    Buf b_in, b_count, b_a4out, b_sreq, b_sout;     // sieve, A4 and benchmark calls
    Buf b_primes, b_profs, b_state, b_planes, b_summ, b_chunk, b_summp, b_didx, b_sidx,
        b_slist, b_dlist, b_dpre, b_out, b_a4, b_counter,
        b_dlab, b_dlaboff, b_dlabp, b_groups, b_rgs, b_item0, b_jobs, b_lab, b_pw, b_gplanes, b_gplanes2;
    // host copies of the current plan
    std::vector<PrimeDesc> hp;
    std::vector<ProfDesc> hprof;
    std::vector<u32> h_chunk, h_summp, h_didx, h_sidx, h_slist, h_dlist;
    // the lists of a plan in the making: a refused one leaves those above whole
    struct Lists {
        std::vector<PrimeDesc> hp;
        std::vector<ProfDesc> hprof;
        std::vector<u32> chunk, summp, didx, dlist;
    } next;
    // dense scan: waves of primes whose label arrays fit the pool together
    struct DenseWave { u32 i0, i1, lchunk0, lchunks, chunk0, chunk1; };
    std::vector<u64> h_dlaboff;         // per dense-local prime (NO_LABELS: powers in the scan)
    std::vector<u32> h_dlabp;           // label chunks (prefix)
    std::vector<DenseWave> hwaves;
    std::vector<GroupDesc> hgroups;     // profiles filtered 32 per word (group.cuh)
    std::vector<RowGroup> hrgs;
    std::vector<u32> hitem0;
    std::vector<LabelJob> hjobs;
    u32 n = 0, nprof = 0, ndense = 0, nsparse = 0, nchunks = 0, nsl = 0, ndl = 0;
    u32 ntable = 0;                     // sparse primes with a profile outside the groups (table_kernel)
    bool tab_split = false;             // few of them: labels from the label matrix, several CTAs a prime
    u32 gmaxB = 0, gmaxq = 0, lab_smem = 0;
    u32 table_smem = 0, dense_smem = 0;
    u32 flags = 0;
    bool have_plan = false;
    CZ_HANDLE *sub = nullptr;           // re-runs of missed speculations, on their own plan and buffers
    bool sub_live = false;              // the last call re-ran profiles there (a replay repeats them)
    CZ_HANDLE *root = nullptr;          // a re-run handle's owner: its stream, events, pinned memory and tables are used
    cudaEvent_t ev[12]{};
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t gexec = nullptr;
    cz_stats last{};
    std::vector<OutRecord> hout;
    void *pin = nullptr;
    size_t pin_cap = 0;
};

namespace {

bool ck(CZ_HANDLE *h, cudaError_t e, const char *what) {
    if (e == cudaSuccess) return true;
    h->err = std::string(what) + ": " + cudaGetErrorString(e);
    return false;
}

bool ensure(CZ_HANDLE *h, Buf &b, size_t bytes) {
    if (bytes == 0) bytes = 16;
    if (b.cap >= bytes) return true;
    if (b.p) cudaFree(b.p);
    b.p = nullptr;
    b.cap = 0;
    cudaError_t e = cudaSuccess;
    for (size_t want : {bytes + bytes / 4, bytes}) {       // no slack where memory is short
        e = cudaMalloc(&b.p, want);
        if (e == cudaSuccess) { b.cap = want; return true; }
        cudaGetLastError();                                // or the next launch check reports it
        b.p = nullptr;
    }
    return ck(h, e, "cudaMalloc");
}

template <class T> T *P(Buf &b) { return reinterpret_cast<T *>(b.p); }

// primes below CHAIN_LIMIT and the prime-power chain: chain[n] = (index of
// q = spf(n) | e << 24, n / q^e) with q^e the full power of q in n, so a walk
// takes one step per distinct prime factor (at most 7 below 2^20), not one per
// factor.  Constants, made once per process (some 25 ms); each handle copies
// them to its device.
struct StaticTables {
    std::vector<u32> primes;
    std::vector<uint2> chain;
};
const StaticTables &static_tables() {
    static StaticTables t;
    static std::once_flag once;
    std::call_once(once, [] {
        std::vector<u32> spf(CHAIN_LIMIT, 0), index(CHAIN_LIMIT, 0);
        for (u32 i = 2; i < CHAIN_LIMIT; ++i) {
            if (spf[i]) continue;
            spf[i] = i;
            index[i] = (u32)t.primes.size();
            t.primes.push_back(i);
            if ((u64)i * i < CHAIN_LIMIT)
                for (u32 j = i * i; j < CHAIN_LIMIT; j += i)
                    if (!spf[j]) spf[j] = i;
        }
        t.chain.resize(CHAIN_LIMIT);
        t.chain[0] = make_uint2(0, 0);
        t.chain[1] = make_uint2(0, 1);
        for (u32 n = 2; n < CHAIN_LIMIT; ++n) {
            const u32 q = spf[n];
            u32 m = n, e = 0;
            while (m % q == 0) { m /= q; ++e; }
            t.chain[n] = make_uint2(index[q] | (e << 24), m);     // index < 2^17, e <= 20
        }
    });
    return t;
}

bool build_static_tables(CZ_HANDLE *h) {
    const StaticTables &t = static_tables();
    h->n_small = (u32)t.primes.size();
    if (!ck(h, cudaMalloc(&h->d_small, t.primes.size() * 4), "cudaMalloc small")) return false;
    if (!ck(h, cudaMalloc(&h->d_chain, t.chain.size() * sizeof(uint2)), "cudaMalloc chain")) return false;
    if (!ck(h, cudaMemcpy(h->d_small, t.primes.data(), t.primes.size() * 4, cudaMemcpyHostToDevice), "copy small")) return false;
    if (!ck(h, cudaMemcpy(h->d_chain, t.chain.data(), t.chain.size() * sizeof(uint2), cudaMemcpyHostToDevice), "copy chain")) return false;
    return true;
}

u32 q_for(const cz_config &c, u32 r) { return c.q_cap[r] ? c.q_cap[r] : 16u; }

// dense segment length in x (32 x steps), default DENSE_SEG
u32 dense_seg(const cz_config &c) {
    const u32 steps = c.dense_steps ? std::min(4096u, std::max(8u, c.dense_steps)) : (u32)DENSE_STEPS;
    return 32u * steps;
}

// chunks of the dense scan of p
u32 dense_chunks(pw_t p, u32 seg) {
    const u32 nh = (u32)((p - 1u) / 2u);                   // < 2^32 for p < 2^33
    const u32 nseg = (u32)(((u64)nh + seg - 1u) / seg);    // nh + seg wraps 32 bits near 2^33
    return (nseg + DENSE_WARPS - 1u) / DENSE_WARPS;
}

// 2: the anchor filter, with its table radius B; 1: the dense scan
u32 route_of(const cz_config &c, pw_t p, u32 mask, u32 mode, u32 &B) {
    if (mode != CZ_SPARSE && (mode != CZ_AUTO || p < c.sparse_min_p)) return 1u;
    u32 Qmax = 0;
    for (u32 r = 2; r <= 9; ++r)
        if (mask & (1u << (r - 2))) Qmax = std::max(Qmax, q_for(c, r));
    return p >= 4096u && Qmax + 1u < p && cover_B(p, Qmax, c.cover_n, B) ? 2u : 1u;
}

// speculative threshold: floor(log_r p - margin_r), a low quantile of M for
// random-looking colourings (M ~ log_r p); 0 disables
u32 qspec_for(const cz_config &c, double lg_p, u32 r, bool allow, u32 level) {
    if (!allow || !c.speculate) return 0u;
    const double lg = lg_p / std::log((double)r);
    const double m = c.spec_margin10[r] / 10.0;
    const double v = std::floor(lg - m) - level;
    return v < 3.0 ? 0u : (u32)v;
}

// Dense primes from DENSE_LABEL_MIN_P on keep the labels of the x coprime to
// 210 in memory (dense.cuh), in waves of at most DENSE_LABEL_WORDS 16-bit labels
// (one prime below 2^33 takes 0.98e9 of them at most).  Where the line lies: 400
// primes near 7e4 take 0.53 ms with the scan's own powers and 0.31 ms with kept
// labels, 400 near 2e4 the same either way (0.39 ms).  The pool stays inside what
// the planes leave of the budget; a prime whose labels alone exceed that takes a
// power for every x.
// Returns the pool's size in labels (limit 0: no labels).
constexpr u64 DENSE_LABEL_MIN_P = 1u << 16, DENSE_LABEL_WORDS = 1ull << 30;
u64 plan_dense_labels(CZ_HANDLE *h, u64 limit) {
    h->h_dlaboff.clear();
    h->h_dlabp.assign(1, 0u);
    h->hwaves.clear();
    if (!h->ndense) return 0;
    CZ_HANDLE::DenseWave w{0, 0, 0, 0, 0, 0};
    u64 used = 0, most = 0;
    auto close = [&](u32 i) {
        w.i1 = i;
        w.chunk1 = h->h_chunk[i];
        w.lchunks = h->h_dlabp[i] - w.lchunk0;
        h->hwaves.push_back(w);
        w = CZ_HANDLE::DenseWave{i, 0, h->h_dlabp[i], 0, h->h_chunk[i], 0};
        most = std::max(most, used);
        used = 0;
    };
    for (u32 i = 0; i < h->ndense; ++i) {
        const pw_t p = h->hp[h->h_didx[i]].p;
        u64 need = 0, off = NO_LABELS;
        u32 nch = 0;
        if (p >= DENSE_LABEL_MIN_P) {
            const u32 nl = labels_below((u32)((p - 1u) / 2u));
            need = ((u64)nl + DLABEL_HEAD + 7u) & ~7ull;
            if (need <= limit) {
                nch = (nl + DLABEL_CHUNK - 1u) / DLABEL_CHUNK;
                if (used && used + need > limit) close(i);
                off = used;
                used += need;
            }
        }
        h->h_dlaboff.push_back(off);
        h->h_dlabp.push_back(h->h_dlabp.back() + nch);
    }
    close(h->ndense);
    return most;
}

// host plan of one call
constexpr u32 CZ_NOSPEC = 1u << 16;      // internal: plan without speculative thresholds
constexpr u32 CZ_HOSTPLAN = 1u << 17;    // internal: host plan only, every sparse profile on its own planes (serving)

// Cost of a profile on its own planes, in groups of its order and size (a group
// costs the same whatever its members), and of a group besides its anchors, as
// so much more p.  Measured on 40 windows of 61 primes: groups of near primes
// of at least 1 / 4 / 8 / 12 members 42.4 / 41.7 / 45.8 / 53.4 ms, this cut with
// a cost of 1/8, 1/5, 1/3 41.2 / 36.7 / 36.7 ms; 37 primes near 7e8 with 1/8,
// 1/5, 1/3 2.32 / 2.21 / 1.99 ms on the device, 7 primes near 4.2e9 1.99 / 2.13 /
// 2.93 ms: the line lies between.
#ifndef CZ_GROUP_OWN_COST
#define CZ_GROUP_OWN_COST (1.0 / 4.0)
#endif
constexpr double OWN_COST = CZ_GROUP_OWN_COST, GROUP_FIXED = 2e7;

// compared planes and anchor stages of a group: least cost per visited anchor
// and position of the row.  A stage costs F loads; beta is the bits it is worth
// (-log2 of the chance that two colours agree in the compared planes); a step
// of 32 anchors x 32 members leaves 1024 2^(-beta (t-1)) survivors, each
// costing about seven loads' time in the queue and the screen.
double group_plan(u32 r, u32 q, u32 &F, u32 &t) {
    static const double beta2[10] = {0, 0, 1.0, 1.585, 2.0, 1.837, 1.848, 1.914, 2.0, 1.948};
    static const double beta3[10] = {0, 0, 0, 0, 0, 2.322, 2.585, 2.807, 3.0, 2.880};
    double bc = 0;
    F = t = 0;
    for (u32 f = r == 2 ? 1u : 2u; f <= (r == 2 ? 1u : r <= 4 ? 2u : 3u); ++f) {
        const double beta = f == 3 ? beta3[r] : beta2[r];
        const u32 lo = f == 1 ? G_TMIN1 : f == 2 ? G_TMIN2 : G_TMIN3, hi = f == 1 ? G_TMAX1 : f == 2 ? G_TMAX2 : G_TMAX3;
        for (u32 k = lo; k <= hi && k <= q; ++k) {
            const double c = (k * f + 1024.0 * std::exp2(-beta * (k - 1.0)) * 7.0) / (q - k + 1.0);
            if (!t || c < bc) { F = f; t = k; bc = c; }
        }
    }
    return bc;
}

// elliptic cover with table radius at most B (group.cuh): E and the least D
// with 3 E^2 D^2 >= 4 p^2, the largest row limit sqrt(E^2 + (H D / 2)^2) at most B
bool cover_ellipse(u64 p, u32 B, u32 q, u32 &E, u32 &D) {
    const long double H = q - 1.0L, k = 2.0L * p / std::sqrt(3.0L);
    auto ok = [&](u64 d) { return (unsigned __int128)3 * E * E * d * d >= (unsigned __int128)4 * p * p; };
    // E^2 + (H k / (2 E))^2 = (B - slack)^2, the larger root; D is rounded up,
    // which moves the largest limit by up to about H / 2
    for (u32 slack = 4; slack <= 4u + 2u * q && B > 16u + slack; slack += 4u) {
        const long double b2 = ((long double)B - slack) * ((long double)B - slack), disc = b2 * b2 - H * H * k * k;
        if (disc <= 0) return false;
        E = (u32)std::sqrt((b2 + std::sqrt(disc)) / 2.0L);
        u64 d = (u64)(k / E);
        while (d > 1 && ok(d - 1)) --d;
        while (!ok(d)) ++d;
        const u64 top = (u64)std::sqrt((long double)E * E + H * H * d * d / 4.0L) + 3u;
        if (top > B) continue;
        if (d >= p || E >= p || d > B_MAX || (q - 1u) * d > 2ull * B) return false;
        D = (u32)d;
        return true;
    }
    return false;
}

// the row whose limit is largest: E cos a + (H D / 2) sin a peaks at tan a = H D / (2 E)
u32 group_apex(const GroupDesc &G) {
    const double h = (G.q - 1.0) * G.D / 2.0;
    return (u32)(G.D * h / std::sqrt(h * h + (double)G.E * G.E));
}

// rows before the wide row groups of G
u32 group_narrow_rows(const GroupDesc &G) {
    return std::min(group_narrow_end(G.t, G.F), (G.D / G_ROWS + 1u) * G_ROWS);
}

// plane words of a profile on its own planes (a multiple of 8: vector loads and
// tile copies align)
u64 own_words(const PrimeDesc &P, const ProfDesc &D) {
    return ((u64)D.npp * (P.nwords + P.nwords2) + 7ull) & ~7ull;
}

// Where the groups would take more than the plane budget, those that take more
// than their members' own planes are dissolved: a full group takes less, one of
// four members up to five times as much (2 B words a plane against 3 B / 32 a
// member and stored plane), a whole call of scattered primes up to 1.9 times as
// measured.  The waves of a call are cut by own planes, so the rest fits.
void keep_groups_in_budget(CZ_HANDLE *h) {
    u64 rest = 0, total = 0;                     // words of the profiles outside groups, of everything
    std::vector<u64> took(h->hgroups.size()), own(h->hgroups.size(), 0);
    for (const ProfDesc &D : h->hprof)
        if (h->hp[D.prime].route == 2u) rest += own_words(h->hp[D.prime], D);
    for (size_t g = 0; g < took.size(); ++g) {
        GroupDesc G = h->hgroups[g];
        group_layout(G, group_narrow_rows(G));
        took[g] = (6ull * G.CL + G.nq) * G.np;
        for (u32 k = 0; k < G.n; ++k) {
            const ProfDesc &D = h->hprof[G.prof[k]];
            own[g] += own_words(h->hp[D.prime], D);
        }
        rest -= own[g];
        total += took[g];
    }
    if (4u * (total + rest) <= (u64)h->cfg.plane_budget_mb << 20) return;
    size_t kept = 0;
    for (size_t g = 0; g < took.size(); ++g)
        if (took[g] <= own[g]) h->hgroups[kept++] = h->hgroups[g];
    h->hgroups.resize(kept);
}

// row groups and items of one group; appended to rgs
u32 group_items(GroupDesc &G, std::vector<RowGroup> &rgs) {
    const u32 dn = group_narrow_rows(G);
    group_layout(G, dn);
    G.rg0 = (u32)rgs.size();
    u32 item = 0;
    const u32 apex = group_apex(G);                     // the limit rises up to this row, then falls
    const u32 wmax = group_wide_max(G.t, G.F);
    for (u32 d0 = 0; d0 <= G.D;) {
        RowGroup R{};
        R.item = item;
        R.d0 = d0;
        R.nrows = std::min(G_ROWS, G.D + 1u - d0);
        if (d0 < dn) R.nrows = std::min(R.nrows, dn - d0);
        const u32 d1 = d0 + R.nrows - 1u;
        const u32 top = apex >= d0 && apex <= d1
                            ? G.B
                            : row_limit(G.E, G.D, G.B, G.q, apex < d0 ? std::max(1u, d0) : d1, 8u);
        if (d0 < dn) {
            R.W = group_narrow_span(G.t, G.F, d1);
            item += top / 6u / R.W + 1u;
        } else {
            const u32 len = (d1 + 5u) / 6u;
            R.ncol = (len + wmax - 1u) / wmax;
            R.W = ((len + R.ncol - 1u) / R.ncol + 31u) & ~31u;
            const u32 c0 = (((G.t - 1u) * d0 + 1u) >> 1) / 6u, sp = G.s * d0 / 6u;
            const u32 bands = top / 6u >= c0 ? (top / 6u - c0) / sp + 1u : 0u;
            item += bands * R.ncol;
        }
        rgs.push_back(R);
        d0 += R.nrows;
    }
    G.nrg = (u32)rgs.size() - G.rg0;
    return item;
}

// row of prime i in the call's label matrix, at least nq labels long
u32 need_labels(CZ_HANDLE *h, u32 i, u32 nq) {
    PrimeDesc &P = h->hp[i];
    if (P.job == 0xFFFFFFFFu) { P.job = (u32)h->hjobs.size(); h->hjobs.push_back(LabelJob{i, 0u, 0ull}); }
    h->hjobs[P.job].nq = std::max(h->hjobs[P.job].nq, nq);
    return P.job;
}

// The sparse profiles of each order, in descending p, are cut into groups of up
// to 32 and profiles kept on their own planes, at least modelled cost: a group
// runs its largest prime's cover at its least threshold.  Cuts are considered
// at 32 members and where p falls by more than 1/16: a run of near primes is
// best filled up, and fewer cuts are less host work (1/8, 1/16 and 1/32 are the
// same within 1 % on 40 windows of 61 primes, 200 of 12, 4000 scattered primes
// and blocks).  Sets ProfDesc.grouped and the group's q as its members'
// speculative threshold.
void plan_groups(CZ_HANDLE *h, const std::vector<u32> &primes_below, u64 &gwords, u64 &gwords2, u64 &pwwords) {
    std::vector<u32> by[10];
    for (u32 g = 0; g < h->nprof; ++g) {
        const ProfDesc &D = h->hprof[g];
        if (h->hp[D.prime].route == 2u && std::min(D.qspec, D.Q) >= 3u) by[D.r].push_back(g);
    }
    // the members of a group that stays
    auto join = [h](GroupDesc &G) {
        for (u32 k = 0; k < G.n; ++k) {
            ProfDesc &D = h->hprof[G.prof[k]];
            const pw_t p = h->hp[D.prime].p;
            D.grouped = 1u;
            D.qspec = G.q;
            G.job[k] = need_labels(h, D.prime, G.nq);
            if ((u64)((p - 1u) >> 1) % G.r != 0u) G.sig |= 1u << k;
        }
    };
    // could the groups exceed the budget at all?  At most 4 planes of 2 B words,
    // guards and colours of the primes each, were every profile a group
    u64 maxB = 0;
    for (const PrimeDesc &P : h->hp) maxB = std::max<u64>(maxB, P.B);
    const bool tight = 16ull * h->nprof * (2u * std::max<u64>(maxB, 16384u) + maxB / 2u + 8192u) >
                       (u64)h->cfg.plane_budget_mb << 20;
    struct Cut { double cost; size_t from; u32 q; };
    for (u32 r = 9; r >= 2; --r) {                   // costliest orders first: the launch ends on cheap items
        auto &v = by[r];
        const size_t n = v.size();
        if (!n) continue;
        auto prime = [&](size_t k) { return h->hp[h->hprof[v[k]].prime].p; };
        auto thr = [&](size_t k) { return std::min(h->hprof[v[k]].qspec, h->hprof[v[k]].Q); };
        if (!std::is_sorted(v.begin(), v.end(), [h](u32 x, u32 y) {
                return h->hp[h->hprof[x].prime].p > h->hp[h->hprof[y].prime].p; }))
            std::stable_sort(v.begin(), v.end(), [h](u32 x, u32 y) {
                return h->hp[h->hprof[x].prime].p > h->hp[h->hprof[y].prime].p;
            });
        double per[256];                             // modelled cost per position by q; 0: not asked yet
        std::fill(per, per + 256, 0.0);
        auto unit = [&](u32 q) {
            u32 F, t;
            if (per[q] == 0.0) per[q] = group_plan(r, q, F, t);
            return per[q];
        };
        std::vector<Cut> best(n + 1, Cut{-1.0, 0, 0});
        best[0].cost = 0;
        for (size_t i = 0; i < n; ++i) {
            if (best[i].cost < 0) continue;
            const double pmax = (double)prime(i);
            double own = 0;
            u32 q = 255;
            for (size_t e = i + 1; e <= n && e <= i + 32; ++e) {
                const pw_t p = prime(e - 1);
                q = std::min(q, thr(e - 1));
                own += (double)p * unit(thr(e - 1)) * OWN_COST;
                if (e < n && e < i + 32 && prime(e) >= p - p / 16u) continue;
                const double group = (pmax + GROUP_FIXED) * unit(q);
                const double c = best[i].cost + std::min(own, group);
                if (best[e].cost < 0 || c < best[e].cost) best[e] = Cut{c, i, group <= own ? q : 0u};
            }
        }
        std::vector<size_t> ends;                    // ends of the groups, largest primes first
        for (size_t e = n; e > 0; e = best[e].from)
            if (best[e].q) ends.push_back(e);
        u32 B = 0, E = 0, Dd = 0, cq = 0, F = 0, t = 0;
        pw_t cover_p = 0;                            // the prime the current cover was made for
        for (size_t x = ends.size(); x-- > 0;) {
            const size_t e = ends[x], i = best[e].from;
            const u32 q = best[e].q;
            const pw_t pmax = prime(i), pmin = prime(e - 1);
            // a cover serves every smaller prime too: neighbouring groups share one,
            // and with it their row groups, while that costs less than 1/1024 (1/128
            // and 1/8192 are the same within 1 % on the same calls)
            u32 own = 0;
            for (size_t k = i; k < e; ++k) own = std::max(own, h->hp[h->hprof[v[k]].prime].B);
            if (q != cq || own > B || (u64)pmax + pmax / 1024u < (u64)cover_p) {
                cq = 0;
                B = own;
                group_plan(r, q, F, t);
                if (!t || !cover_ellipse(pmax, B, q, E, Dd)) continue;
                cq = q;
                cover_p = pmax;
            }
            if (B >= pmin || Dd >= pmin) continue;
            GroupDesc G{};
            G.r = r; G.np = planes_for(r); G.F = F;
            G.B = B; G.E = E; G.D = Dd; G.q = q; G.t = t; G.s = q - t + 1u;
            G.n = (u32)(e - i);
            G.nq = (u32)(std::upper_bound(primes_below.begin(), primes_below.end(), B) - primes_below.begin());
            for (size_t k = i; k < e; ++k) G.prof[k - i] = v[k];
            if (!tight) join(G);
            h->hgroups.push_back(G);
        }
    }
    if (tight) {
        keep_groups_in_budget(h);
        for (GroupDesc &G : h->hgroups) join(G);
    }
    u32 items = 0, own = 0;
    const GroupDesc *pv = nullptr;
    for (GroupDesc &G : h->hgroups) {
        G.item0 = items;
        h->hitem0.push_back(items);
        if (pv && pv->r == G.r && pv->B == G.B && pv->E == G.E && pv->D == G.D && pv->q == G.q) {
            G.I0 = pv->I0; G.CL = pv->CL; G.rg0 = pv->rg0; G.nrg = pv->nrg;
        } else {
            own = group_items(G, h->hrgs);
        }
        pv = &G;
        items += own;
        G.off = gwords;
        gwords += 6ull * G.CL * std::min(2u, G.np);  // CL is a multiple of 4: 16-byte aligned
        G.off2 = gwords2;
        gwords2 += 6ull * G.CL * (G.np > 2u ? G.np - 2u : 0u);
        G.pwoff = pwwords;
        pwwords += (u64)G.nq * G.np;
        h->gmaxB = std::max(h->gmaxB, G.B);
        h->gmaxq = std::max(h->gmaxq, G.nq);
    }
    h->hitem0.push_back(items);
}

// the host arrays of a plan that the device reads
struct Part { Buf *at; const void *from; size_t bytes; };
std::vector<Part> upload_parts(CZ_HANDLE *h) {
    auto part = [](Buf &b, const auto &v) { return Part{&b, v.data(), sizeof(v[0]) * v.size()}; };
    return {part(h->b_primes, h->hp), part(h->b_profs, h->hprof), part(h->b_chunk, h->h_chunk),
            part(h->b_summp, h->h_summp), part(h->b_didx, h->h_didx), part(h->b_sidx, h->h_sidx),
            part(h->b_dlaboff, h->h_dlaboff), part(h->b_dlabp, h->h_dlabp), part(h->b_groups, h->hgroups),
            part(h->b_rgs, h->hrgs), part(h->b_item0, h->hitem0), part(h->b_jobs, h->hjobs),
            part(h->b_slist, h->h_slist), part(h->b_dlist, h->h_dlist)};
}

// masks: the wanted orders of each prime (nullptr: every admissible one);
// level: speculative thresholds lowered by so much (re-runs)
int plan(CZ_HANDLE *h, const pw_t *primes, u32 n, u32 flags, const u32 *masks = nullptr, u32 level = 0) {
    const cz_config &c = h->cfg;
    const u32 mode = flags & CZ_AUTO;
    const u32 seg = dense_seg(c);
    // primes, orders and routes beside the resident plan: a request refused in
    // this loop leaves that plan whole, for a replay
    CZ_HANDLE::Lists &N = h->next;
    N.hp.assign(n, PrimeDesc{});
    N.hprof.clear();
    N.didx.clear(); N.dlist.clear(); N.summp.clear();
    N.chunk.assign(1, 0u);
    u64 plane_words = 0;
    u32 max_slots_t = 8, max_slots_d = 8, max_nq = 0, nsparse = 0;
    u64 summ_slots = 0;
    for (u32 i = 0; i < n; ++i) {
        const pw_t p = primes[i];
        if (p < 2u || (u64)p >= PW_LIMIT) { h->err = "prime out of domain: " + std::to_string(p); return CZ_EINVAL; }
        PrimeDesc &P = N.hp[i];
        P.p = p;
        P.mask = p > 2u ? mask_of(p) & (masks ? masks[i] : ~0u) : 0u;
        P.m = lcm_of_mask(P.mask);
        P.e = P.mask ? (p - 1u) / P.m : 0u;
        P.first_prof = (u32)N.hprof.size();
        P.nprof = popc(P.mask);
        P.job = 0xFFFFFFFFu;
        if (!P.nprof) continue;
        P.route = route_of(c, p, P.mask, mode, P.B);
        const bool sparse = P.route == 2u;
        if (sparse) {
            // view widths in words, multiples of 4: every view and every tile
            // copy of the filter starts on a 16-byte boundary
            P.K0 = (P.B + 31u) / 32u + 4u;
            P.nwords = (2u * P.K0 + 8u + 3u) & ~3u;
            P.K2 = (P.B + 63u) / 64u + 4u;
            P.nwords2 = (2u * P.K2 + 8u + 3u) & ~3u;
            ++nsparse;
            max_slots_t = std::max(max_slots_t, hash_slots(P.m));
        } else {
            if (mode == CZ_SPARSE) {
                h->err = "sparse path unsupported for p = " + std::to_string(p);
                return CZ_EINVAL;
            }
            const u32 nch = dense_chunks(p, seg);
            if ((u64)N.chunk.back() + nch > 0xFFFFFFFFull || summ_slots + (u64)nch * P.nprof > 0xFFFFFFFFull) {
                h->err = "dense scan too large for one call (chunk index beyond 32 bits)";
                return CZ_ELIMIT;
            }
            N.didx.push_back(i);
            N.summp.push_back((u32)summ_slots);
            summ_slots += (u64)nch * P.nprof;
            N.chunk.push_back(N.chunk.back() + nch);
            max_slots_d = std::max(max_slots_d, hash_slots(P.m));
        }
        const double lg_p = sparse ? std::log((double)p) : 0.0;
        for (u32 r = 2; r <= 9; ++r) {
            if (!(P.mask & (1u << (r - 2)))) continue;
            ProfDesc D{};
            D.prime = i;
            D.r = r;
            D.np = planes_for(r);
            D.npp = planes_stored(r);
            D.out_slot = (u32)N.hprof.size();
            if (sparse) {
                D.Q = q_for(c, r);
                D.qspec = qspec_for(c, lg_p, r, !(flags & CZ_NOSPEC), level);
                D.tpref = c.anchor_t[r] ? c.anchor_t[r] : anchor_pref(r, c.anchor_bits);
            } else {
                D.local = (u32)N.didx.size() - 1u;
                N.dlist.push_back((u32)N.hprof.size());
            }
            N.hprof.push_back(D);
        }
    }
    h->have_plan = false;
    h->hp.swap(N.hp);
    h->hprof.swap(N.hprof);
    h->h_didx.swap(N.didx); h->h_dlist.swap(N.dlist); h->h_summp.swap(N.summp); h->h_chunk.swap(N.chunk);
    h->h_sidx.clear(); h->h_slist.clear();
    h->hgroups.clear(); h->hrgs.clear(); h->hitem0.clear(); h->hjobs.clear();
    h->nsparse = nsparse; h->gmaxB = 0; h->gmaxq = 0;
    h->n = n;
    h->nprof = (u32)h->hprof.size();
    h->ndense = (u32)h->h_didx.size();
    h->nchunks = h->h_chunk.back();
    u64 gwords = 0, gwords2 = 0, pwwords = 0;
    // the grouped filter always screens (a switch in its kernel cost 1 % with
    // 64-bit words: 13.93 -> 14.06 ms for 96 primes); without the screen every
    // profile is filtered by itself
    if (h->nsparse && c.screen && !(flags & (CZ_NOSPEC | CZ_HOSTPLAN))) plan_groups(h, static_tables().primes, gwords, gwords2, pwwords);
    for (u32 g = 0; g < h->nprof; ++g) {
        ProfDesc &D = h->hprof[g];
        const PrimeDesc &P = h->hp[D.prime];
        if (P.route != 2u || D.grouped) continue;
        // with B from the largest cap a denominator bound exists for every order
        if (!cover_D(P.p, P.B, D.Q, D.D)) { h->err = "no cover for p = " + std::to_string(P.p); return CZ_EINVAL; }
        D.plane_off = plane_words;
        plane_words += own_words(P, D);
        if (h->h_sidx.empty() || h->h_sidx.back() != D.prime) h->h_sidx.push_back(D.prime);
        D.local = (u32)h->h_sidx.size() - 1u;
        h->h_slist.push_back(g);
    }
    h->ntable = (u32)h->h_sidx.size();
    // few primes: their labels are computed over the whole GPU (table.cuh)
    h->tab_split = h->ntable && 2u * h->ntable <= (u32)h->sms;
    if (h->tab_split)
        for (u32 i : h->h_sidx) {
            const u32 nmax = 32u * ((h->hp[i].B + 1u + 31u) / 32u + 1u);
            const std::vector<u32> &hs = static_tables().primes;
            need_labels(h, i, (u32)(std::lower_bound(hs.begin(), hs.end(), nmax) - hs.begin()));
        }
    // longest first: the persistent filter hands out profiles in list order,
    // so the costly ones (more stored planes, larger p) start first and the
    // launch ends on short profiles
    std::stable_sort(h->h_slist.begin(), h->h_slist.end(), [h](u32 x, u32 y) {
        const ProfDesc &a = h->hprof[x], &b = h->hprof[y];
        if (a.npp != b.npp) return a.npp > b.npp;
        return h->hp[a.prime].p > h->hp[b.prime].p;
    });
    h->nsl = (u32)h->h_slist.size();
    h->ndl = (u32)h->h_dlist.size();
    // primes below the largest table end, for the table kernel's shared memory
    u32 maxB = 0;
    for (u32 i : h->h_sidx) maxB = std::max(maxB, h->hp[i].B);
    if (h->ntable) {
        const u32 nmax = 32u * ((maxB + 1u + 31u) / 32u + 1u);
        const std::vector<u32> &hs = static_tables().primes;
        max_nq = (u32)(std::lower_bound(hs.begin(), hs.end(), nmax) - hs.begin());
    }
    h->lab_smem = max_slots_t * (u32)(sizeof(pw_t) + 2u) + 16u;
    const u64 budget = (u64)c.plane_budget_mb << 20, planes = 4ull * (plane_words + gwords + gwords2 + pwwords);
    u64 dlab = plan_dense_labels(h, std::min(DENSE_LABEL_WORDS, (budget - std::min(budget, planes)) / 2u));
    u64 labels = 0;
    for (LabelJob &J : h->hjobs) { J.off = labels; labels += (J.nq + 63u) & ~63u; }
    h->table_smem = max_slots_t * (u32)(sizeof(pw_t) + 2u) + 8u + max_nq * 2u + 16u;
    if (h->table_smem > TABLE_DYN_SMEM) {
        h->err = "table shared memory above the per-block limit";
        return CZ_EINVAL;
    }
    h->dense_smem = max_slots_d * (u32)(sizeof(pw_t) + 2u) + 16u;
    if (flags & CZ_HOSTPLAN) return CZ_OK;
    // device memory: uploaded descriptors, then the results (counters, records,
    // A4, states) that come back in one copy, in one buffer; tables in another
    size_t small = 0, big = 0;
    std::vector<std::pair<Buf *, size_t>> at_small, at_big;
    auto place = [](std::vector<std::pair<Buf *, size_t>> &v, size_t &end, Buf &b, size_t bytes) {
        v.push_back({&b, end});
        end += (bytes + 255) & ~size_t(255);
    };
    for (const Part &x : upload_parts(h)) place(at_small, small, *x.at, x.bytes);
    h->up_bytes = h->down_off = small;
    place(at_small, small, h->b_counter, 64);
    place(at_small, small, h->b_out, sizeof(OutRecord) * h->nprof);
    place(at_small, small, h->b_a4, 4ull * n);
    place(at_small, small, h->b_state, sizeof(ProfState) * h->nprof);
    h->down_bytes = small - h->down_off;
    place(at_small, small, h->b_dpre, 4ull * h->nprof);
    auto place_big = [&]() {
        at_big.clear();
        big = 0;
        place(at_big, big, h->b_planes, plane_words * 4ull);
        place(at_big, big, h->b_summ, sizeof(Summ) * summ_slots);
        place(at_big, big, h->b_dlab, 2ull * dlab);
        place(at_big, big, h->b_lab, 2ull * labels);
        place(at_big, big, h->b_pw, 4ull * pwwords);
        place(at_big, big, h->b_gplanes, 4ull * gwords);
        place(at_big, big, h->b_gplanes2, 4ull * gwords2);
        return ensure(h, h->b_big, big);
    };
    if (!ensure(h, h->b_small, small)) return CZ_ECUDA;
    if (!place_big()) {
        if (!dlab) return CZ_ECUDA;
        dlab = plan_dense_labels(h, 0);                   // the dense scan runs without them, as the device's memory is short
        if (!place_big()) return CZ_ECUDA;
        h->err.clear();
    }
    for (auto &x : at_small) x.first->p = static_cast<char *>(h->b_small.p) + x.second;
    for (auto &x : at_big) x.first->p = static_cast<char *>(h->b_big.p) + x.second;
    h->flags = flags;
    h->have_plan = true;
    return CZ_OK;
}

int upload(CZ_HANDLE *h, cz_stats *s) {
    CZ_HANDLE *o = h->root ? h->root : h;               // owner of the pinned memory
    const size_t total = std::max(h->up_bytes, h->down_bytes);
    if (o->pin_cap < total) {
        if (o->pin) cudaFreeHost(o->pin);
        o->pin = nullptr;
        o->pin_cap = 0;
        // at least a megabyte: a call's re-runs and most later calls fit
        const size_t want = std::max(total + total / 4, size_t(1) << 20);
        if (!ck(h, cudaHostAlloc(&o->pin, want, cudaHostAllocDefault), "cudaHostAlloc")) return CZ_ECUDA;
        o->pin_cap = want;
    }
    // the host plan, laid out as on the device, in one copy
    char *stage = static_cast<char *>(o->pin);
    const char *base = static_cast<const char *>(h->b_small.p);
    for (const Part &x : upload_parts(h))
        if (x.bytes) std::memcpy(stage + (static_cast<const char *>(x.at->p) - base), x.from, x.bytes);
    if (!ck(h, cudaMemcpyAsync(h->b_small.p, stage, h->up_bytes, cudaMemcpyHostToDevice, h->st), "h2d")) return CZ_ECUDA;
    if (s) s->h2d_bytes = h->up_bytes;
    return CZ_OK;
}

// rows per threshold epoch of a call with few profiles, at least EPOCH_MIN and
// EPOCH_PER_PROFILE a profile: the filter's items then fill the GPU (one prime
// near 2^32: 1024 rows 0.59 ms, 64 a profile 0.41; 3 primes near 4.2e9 with 128,
// 64, 32 a profile 0.90 / 0.86 / 0.84 ms)
constexpr u32 EPOCH_MIN = 32, EPOCH_PER_PROFILE = 32;

// enqueue the device work of the current plan on h->st; returns launches
int enqueue(CZ_HANDLE *h, bool timed, u32 &launches) {
    cudaStream_t st = h->st;
    launches = 0;
    auto rec = [&](int i) { if (timed) cudaEventRecord(h->ev[i], st); };
    rec(0);
    // work counters and the A4 error word, before anything that runs beside
    cudaMemsetAsync(h->b_counter.p, 0, 64, st);
    if (h->n) {
        setup_kernel<<<(h->n + SETUP_WARPS - 1) / SETUP_WARPS, SETUP_WARPS * 32, 0, st>>>(P<PrimeDesc>(h->b_primes), P<ProfDesc>(h->b_profs),
                                                         P<ProfState>(h->b_state), h->n);
        ++launches;
    }
    rec(1);
    // the A4 counts need the primes only and leave the GPU mostly idle (a long
    // chain of curve operations per prime): they run beside the tables and the
    // filter on a stream of their own, joined before the call's end
    const bool a4 = (h->flags & CZ_A4) && h->n;
    if (a4) {
        cudaEventRecord(h->fork, st);
        cudaStreamWaitEvent(h->st2, h->fork, 0);
        if (timed) cudaEventRecord(h->ev[7], h->st2);
        a4_kernel<<<(h->n + A4_WARPS - 1) / A4_WARPS, A4_WARPS * 32, 0, h->st2>>>(
            P<PrimeDesc>(h->b_primes), h->n, P<u32>(h->b_a4), P<u32>(h->b_counter) + 8);
        if (timed) cudaEventRecord(h->ev[8], h->st2);
        cudaEventRecord(h->join, h->st2);
        ++launches;
    }
    const u32 ngroups = (u32)h->hgroups.size(), njobs = (u32)h->hjobs.size();
    if (njobs) {
        LabelArgs la;
        la.primes = P<PrimeDesc>(h->b_primes);
        la.state = P<ProfState>(h->b_state);
        la.jobs = P<LabelJob>(h->b_jobs);
        la.nchunk = std::max(2u, std::min(96u, 8u * (u32)h->sms / njobs));
        la.lab = P<unsigned short>(h->b_lab);
        la.small_primes = h->d_small;
        plabel_kernel<<<njobs * la.nchunk, 256, h->lab_smem, st>>>(la);
        ++launches;
    }
    if (ngroups) {
        GTableArgs ga;
        ga.groups = P<GroupDesc>(h->b_groups);
        ga.ngroups = ngroups;
        ga.lab = P<unsigned short>(h->b_lab);
        ga.jobs = P<LabelJob>(h->b_jobs);
        ga.pw = P<u32>(h->b_pw);
        ga.planes = P<u32>(h->b_gplanes);
        ga.planes2 = P<u32>(h->b_gplanes2);
        ga.chain = h->d_chain;
        ga.small_primes = h->d_small;
        const u32 qblk = (h->gmaxq + 31u) / 32u;
        gpack_kernel<<<(ngroups * qblk + 7u) / 8u, 256, 0, st>>>(ga, qblk);
        gtable_low_kernel<<<ngroups, 512, 0, st>>>(ga);
        launches += 2;
        for (u32 lo = G_LOW; lo <= h->gmaxB; lo *= 2u) {
            const u32 nblk = (lo / 6u + 2u + 255u) / 256u;
            gtable_level_kernel<<<ngroups * nblk, 256, 0, st>>>(ga, lo, nblk);
            ++launches;
        }
    }
    if (h->ntable) {
        TableArgs ta;
        ta.primes = P<PrimeDesc>(h->b_primes);
        ta.profs = P<ProfDesc>(h->b_profs);
        ta.state = P<ProfState>(h->b_state);
        ta.planes = P<u32>(h->b_planes);
        ta.sparse_primes = P<u32>(h->b_sidx);
        ta.nsparse = h->ntable;
        ta.small_primes = h->d_small;
        ta.n_small = h->n_small;
        ta.chain = h->d_chain;
        ta.chain_limit = CHAIN_LIMIT;
        ta.lab = h->tab_split ? P<unsigned short>(h->b_lab) : nullptr;
        ta.jobs = P<LabelJob>(h->b_jobs);
        ta.nchunk = h->tab_split ? std::max(1u, std::min(64u, 2u * (u32)h->sms / h->ntable)) : 1u;
        const u32 grid = ta.lab ? h->ntable * ta.nchunk : std::min<u32>(h->ntable, (u32)h->sms);
        table_kernel<<<grid, TABLE_THREADS, ta.lab ? 0u : h->table_smem, st>>>(ta);
        ++launches;
    }
    rec(2);
    if (ngroups) {
        GFilterArgs fa;
        fa.primes = P<PrimeDesc>(h->b_primes);
        fa.profs = P<ProfDesc>(h->b_profs);
        fa.state = P<ProfState>(h->b_state);
        fa.groups = P<GroupDesc>(h->b_groups);
        fa.item0 = P<u32>(h->b_item0);
        fa.rgs = P<RowGroup>(h->b_rgs);
        fa.ngroups = ngroups;
        fa.nitems = h->hitem0.back();
        fa.planes = P<u32>(h->b_gplanes);
        fa.planes2 = P<u32>(h->b_gplanes2);
        fa.next = P<u32>(h->b_counter) + 4;
        const u32 most = h->cfg.sparse_blocks ? std::min(h->cfg.sparse_blocks, (u32)h->sms) : (u32)h->sms;
        gfilter_kernel<<<std::min(fa.nitems, most), (G_WARPS + 2) * 32, G_SMEM, st>>>(fa);
        ++launches;
    }
    if (h->nsl) {
        SparseArgs sa{};                       // serving fields stay null: one-call census
        sa.primes = P<PrimeDesc>(h->b_primes);
        sa.profs = P<ProfDesc>(h->b_profs);
        sa.state = P<ProfState>(h->b_state);
        sa.planes = P<u32>(h->b_planes);
        sa.prof_list = P<u32>(h->b_slist);
        sa.nlist = h->nsl;
        sa.next = P<u32>(h->b_counter);
        u32 grid = h->cfg.sparse_blocks ? h->cfg.sparse_blocks : (u32)CZ_SPARSE_MINB * (u32)h->sms;
        // a call with few profiles spreads each profile's rows over more CTAs
        // (up to 64), so small calls fill the GPU; large calls keep the tuned group
        sa.group = std::max(std::max(1u, h->cfg.cta_per_profile), std::min(64u, grid / std::max(1u, h->nsl)));
        sa.tune.screen = h->cfg.screen;
        // and cuts its rows into shorter epochs, so that there are items for them:
        // near 2^32 a profile has 8 epochs of 1024 rows and some 5 tiles each
        const u32 erows = h->cfg.epoch_rows ? h->cfg.epoch_rows : EPOCH_ROWS_DEFAULT;
        sa.epoch_rows = std::min(erows, std::max(EPOCH_MIN, EPOCH_PER_PROFILE * h->nsl));
        grid = std::min(grid, h->nsl * sa.group);
        sparse_kernel<<<grid, SPARSE_WARPS * 32, TILE_WORDS * 4u, st>>>(sa);
        ++launches;
    }
    rec(3);
    if (h->ndense) {
        DenseArgs da;
        da.primes = P<PrimeDesc>(h->b_primes);
        da.dense_idx = P<u32>(h->b_didx);
        da.profs = P<ProfDesc>(h->b_profs);
        da.chunk_prefix = P<u32>(h->b_chunk);
        da.summ_prefix = P<u32>(h->b_summp);
        da.nprimes = h->ndense;
        da.summ = P<Summ>(h->b_summ);
        da.state = P<ProfState>(h->b_state);
        da.seg = dense_seg(h->cfg);
        da.lab_off = P<u64>(h->b_dlaboff);
        da.lab = P<unsigned short>(h->b_dlab);
        for (const CZ_HANDLE::DenseWave &w : h->hwaves) {
            if (w.lchunks) {
                DLabelArgs dl;
                dl.primes = da.primes;
                dl.dense_idx = da.dense_idx;
                dl.chunk_prefix = P<u32>(h->b_dlabp);
                dl.i0 = w.i0;
                dl.i1 = w.i1;
                dl.chunk0 = w.lchunk0;
                dl.lab_off = da.lab_off;
                dl.lab = P<unsigned short>(h->b_dlab);
                dl.state = da.state;
                dlabel_kernel<<<w.lchunks, 256, h->dense_smem, st>>>(dl);
                ++launches;
            }
            da.chunk0 = w.chunk0;
            da.nchunks = w.chunk1;
            const u32 grid = std::min<u32>(w.chunk1 - w.chunk0, (u32)h->sms * 8u);
            dense_scan_kernel<<<grid, DENSE_WARPS * 32, h->dense_smem, st>>>(da);
            ++launches;
        }
        DenseMergeArgs ma;
        ma.primes = P<PrimeDesc>(h->b_primes);
        ma.profs = P<ProfDesc>(h->b_profs);
        ma.chunk_prefix = P<u32>(h->b_chunk);
        ma.summ_prefix = P<u32>(h->b_summp);
        ma.nprimes = h->ndense;
        ma.summ = P<Summ>(h->b_summ);
        ma.state = P<ProfState>(h->b_state);
        ma.prefix_out = P<u32>(h->b_dpre);
        dense_merge_kernel<<<(h->ndl + 7) / 8, 256, 0, st>>>(ma, P<u32>(h->b_dlist), h->ndl);
        ++launches;
    }
    rec(4);
    if (h->nprof) {
        finalize_kernel<<<(h->nprof + FINAL_WARPS - 1) / FINAL_WARPS, FINAL_WARPS * 32, 0, st>>>(
            P<PrimeDesc>(h->b_primes), P<ProfDesc>(h->b_profs), P<ProfState>(h->b_state), P<u32>(h->b_dpre),
            h->nprof, (h->flags & CZ_VERIFY) ? 1u : 0u, P<u32>(h->b_counter) + 4, ngroups ? h->hitem0.back() : 0u,
            P<OutRecord>(h->b_out));
        ++launches;
    }
    rec(5);
    if (a4) cudaStreamWaitEvent(st, h->join, 0);
    rec(6);
    return ck(h, cudaGetLastError(), "launch") ? CZ_OK : CZ_ECUDA;
}

void read_times(CZ_HANDLE *h, cz_stats *s) {
    float t[6] = {0};
    for (int i = 0; i < 5; ++i) cudaEventElapsedTime(&t[i], h->ev[i], h->ev[i + 1]);
    if ((h->flags & CZ_A4) && h->n) cudaEventElapsedTime(&t[5], h->ev[7], h->ev[8]);
    s->ms_setup = t[0]; s->ms_table = t[1]; s->ms_sparse = t[2]; s->ms_dense = t[3];
    s->ms_finalize = t[4]; s->ms_a4 = t[5];
    cudaEventElapsedTime(&s->ms_device, h->ev[0], h->ev[6]);
}

// status of every record: a speculative miss goes to *respec (profile index),
// another status that the dense scan can settle to *fallback (prime index),
// anything else refuses the call
int check_records(CZ_HANDLE *h, std::vector<u32> *fallback, std::vector<u32> *respec = nullptr) {
    for (u32 g = 0; g < h->nprof; ++g) {
        const OutRecord &o = h->hout[g];
        if (o.status) {
            const PrimeDesc &P = h->hp[h->hprof[g].prime];
            if (respec && P.route == 2u && o.status == ST_SPEC) {
                respec->push_back(g);
                continue;
            }
            if (fallback && P.route == 2u && !(o.status & (ST_ROOT | ST_LABEL | ST_VERIFY))) {
                if (fallback->empty() || fallback->back() != h->hprof[g].prime)
                    fallback->push_back(h->hprof[g].prime);
                continue;
            }
            char buf[160];
            snprintf(buf, sizeof buf, "refused: p=%llu r=%u status=0x%x", (unsigned long long)o.p, o.r, o.status);
            h->err = buf;
            return CZ_EREFUSED;
        }
    }
    return CZ_OK;
}

}  // namespace


namespace {

void handle_close(CZ_HANDLE *h) {
    if (!h) return;
    handle_close(h->sub);
    cudaSetDevice(h->dev);
    if (h->gexec) cudaGraphExecDestroy(h->gexec);
    if (h->graph) cudaGraphDestroy(h->graph);
    Buf *bufs[] = {&h->b_small, &h->b_big, &h->b_in, &h->b_count, &h->b_a4out, &h->b_sreq, &h->b_sout};
    for (Buf *b : bufs) if (b->p) cudaFree(b->p);
    if (!h->root) {
        if (h->pin) cudaFreeHost(h->pin);
        if (h->d_small) cudaFree(h->d_small);
        if (h->d_chain) cudaFree(h->d_chain);
        for (auto &e : h->ev) if (e) cudaEventDestroy(e);
        if (h->fork) cudaEventDestroy(h->fork);
        if (h->join) cudaEventDestroy(h->join);
        if (h->st2) cudaStreamDestroy(h->st2);
        if (h->st) cudaStreamDestroy(h->st);
    }
    delete h;
}

// a handle for a call's re-runs: its own plan and device memory, everything
// else its owner's (the two never run at the same time)
CZ_HANDLE *open_sub(CZ_HANDLE *o) {
    CZ_HANDLE *h = new CZ_HANDLE();
    h->cfg = o->cfg;
    h->dev = o->dev;
    h->sms = o->sms;
    h->st = o->st; h->st2 = o->st2; h->fork = o->fork; h->join = o->join;
    std::copy(o->ev, o->ev + 12, h->ev);
    h->d_small = o->d_small; h->d_chain = o->d_chain; h->n_small = o->n_small;
    h->root = o->root ? o->root : o;
    return h;
}

int handle_open(const cz_config *cfg, CZ_HANDLE **out) {
    if (!out) return CZ_EINVAL;
    *out = nullptr;
    CZ_HANDLE *h = new CZ_HANDLE();
    if (cfg) h->cfg = *cfg; else cz_default_config(&h->cfg);
    if (h->cfg.cover_n < 2 || h->cfg.cover_n > 8) { delete h; return CZ_EINVAL; }
    for (int r = 2; r <= 9; ++r)
        if (h->cfg.q_cap[r] && (h->cfg.q_cap[r] < 3 || h->cfg.q_cap[r] > 255)) { delete h; return CZ_EINVAL; }
    for (int r = 0; r < 10; ++r)
        if (h->cfg.anchor_t[r] && (h->cfg.anchor_t[r] < 2 || h->cfg.anchor_t[r] > 32)) { delete h; return CZ_EINVAL; }
    if (h->cfg.epoch_rows > (1u << 20)) { delete h; return CZ_EINVAL; }
    h->dev = h->cfg.device;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || h->dev < 0 || h->dev >= ndev) { delete h; return CZ_ECUDA; }
    cudaSetDevice(h->dev);
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, h->dev);
    h->sms = prop.multiProcessorCount;
    if (cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&h->st2, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&h->fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&h->join, cudaEventDisableTiming) != cudaSuccess) {
        handle_close(h);
        return CZ_ECUDA;
    }
    for (auto &e : h->ev) cudaEventCreate(&e);
    cudaFuncSetAttribute(table_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TABLE_DYN_SMEM);
    cudaFuncSetAttribute(dense_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    cudaFuncSetAttribute(dlabel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    // the filter stages its tiles in shared memory: the whole unified array
    // goes to shared memory, two CTAs of TILE_WORDS words each per SM
    cudaFuncSetAttribute(sparse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(TILE_WORDS * 4u));
    cudaFuncSetAttribute(sparse_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(gfilter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G_SMEM);
    cudaFuncSetAttribute(gfilter_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(plabel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    if (!build_static_tables(h)) { handle_close(h); return CZ_ECUDA; }
    *out = h;
    return CZ_OK;
}

// profiles of n primes: sum over primes of #{r in 2..9 : r | p - 1}
u32 count_profiles(const pw_t *primes, u32 n) {
    u32 c = 0;
    for (u32 i = 0; i < n; ++i)
        if (primes[i] > 2u) c += popc(mask_of(primes[i]));
    return c;
}

// plane-pool bytes one prime would take (0 for the dense route)
u64 plane_bytes(const cz_config &c, pw_t p, u32 flags) {
    if (p < 3u) return 0;
    const u32 mode = flags & CZ_AUTO;
    if (mode == CZ_DENSE || (mode == CZ_AUTO && p < c.sparse_min_p)) return 0;
    const u32 mask = mask_of(p);
    u32 Qmax = 0, units = 0;
    for (u32 r = 2; r <= 9; ++r)
        if (mask & (1u << (r - 2))) { Qmax = std::max(Qmax, q_for(c, r)); units += planes_stored(r); }
    u32 B = 0;
    if (Qmax + 1u >= p || !cover_B(p, Qmax, c.cover_n, B)) return 0;
    const u64 words = (2ull * ((B + 31u) / 32u + 4u) + 8ull) + (2ull * ((B + 63u) / 64u + 4u) + 8ull);
    return 4ull * words * units + 64ull * units;
}

int census_impl(CZ_HANDLE *h, const pw_t *primes, uint32_t n, uint32_t flags, CZ_RECORD *out,
                uint32_t out_cap, uint32_t *a4_out, cz_stats *stats, bool allow_fallback,
                const u32 *masks = nullptr, u32 level = 0);

// a batch whose plane pool would exceed the budget runs as consecutive waves
int census_waves(CZ_HANDLE *h, const pw_t *primes, uint32_t n, uint32_t flags, CZ_RECORD *out,
                        uint32_t out_cap, uint32_t *a4_out, cz_stats *stats) {
    const u64 budget = (u64)h->cfg.plane_budget_mb << 20;
    u64 acc = 0;
    u32 start = 0, prof_off = 0, waves = 0;
    cz_stats tot{};
    for (u32 i = 0; i <= n; ++i) {
        const u64 b = i < n ? plane_bytes(h->cfg, primes[i], flags) : 0;
        if (i == n || (acc + b > budget && i > start)) {
            const u32 m = i - start;
            const u32 np = count_profiles(primes + start, m);
            cz_stats s{};
            int rc = census_impl(h, primes + start, m, flags, out + prof_off, out_cap - prof_off,
                                 a4_out ? a4_out + start : nullptr, &s, true);
            if (rc) return rc;
            ++waves;
            tot.ms_setup += s.ms_setup; tot.ms_table += s.ms_table; tot.ms_sparse += s.ms_sparse;
            tot.ms_dense += s.ms_dense; tot.ms_a4 += s.ms_a4; tot.ms_finalize += s.ms_finalize;
            tot.ms_device += s.ms_device; tot.ms_h2d += s.ms_h2d; tot.ms_d2h += s.ms_d2h;
            tot.n_dense += s.n_dense; tot.n_sparse += s.n_sparse; tot.n_profiles += s.n_profiles;
            tot.n_fallback += s.n_fallback; tot.n_respec += s.n_respec; tot.ms_respec += s.ms_respec;
            tot.kernels += s.kernels; tot.words += s.words; tot.completions += s.completions;
            tot.tests += s.tests; tot.h2d_bytes += s.h2d_bytes; tot.d2h_bytes += s.d2h_bytes;
            tot.staged_bytes += s.staged_bytes;
            prof_off += np;
            start = i;
            acc = 0;
        }
        acc += b;
    }
    tot.n_primes = n;
    tot.waves = waves;
    h->have_plan = waves == 1 && h->have_plan;
    if (stats) *stats = tot;
    return CZ_OK;
}

int census_impl(CZ_HANDLE *h, const pw_t *primes, uint32_t n, uint32_t flags, CZ_RECORD *out,
                       uint32_t out_cap, uint32_t *a4_out, cz_stats *stats, bool allow_fallback,
                       const u32 *masks, u32 level) {
    if (!h) return CZ_EINVAL;
    cudaSetDevice(h->dev);
    h->err.clear();
    cz_stats s{};
    if (n == 0) { if (stats) *stats = s; return CZ_OK; }
    if (!primes || !out || ((flags & CZ_A4) && !a4_out)) { h->err = "null buffer"; return CZ_EINVAL; }
    if ((flags & CZ_AUTO) == 0) flags |= CZ_AUTO;
    int rc = plan(h, primes, n, flags, masks, level);
    if (rc) return rc;
    h->sub_live = false;
    if (out_cap < h->nprof) { h->have_plan = false; h->err = "output capacity below profile count"; return CZ_EINVAL; }
    if (h->gexec) { cudaGraphExecDestroy(h->gexec); h->gexec = nullptr; }
    if (h->graph) { cudaGraphDestroy(h->graph); h->graph = nullptr; }
    cudaEventRecord(h->ev[9], h->st);
    if ((rc = upload(h, &s))) return rc;
    cudaEventRecord(h->ev[10], h->st);
    u32 launches = 0;
    if ((rc = enqueue(h, true, launches))) return rc;
    // counters, records, A4 and states come back in one copy
    const char *pin = static_cast<const char *>((h->root ? h->root : h)->pin);
    const char *down = static_cast<const char *>(h->b_small.p) + h->down_off;
    if (!ck(h, cudaMemcpyAsync((void *)pin, down, h->down_bytes, cudaMemcpyDeviceToHost, h->st), "d2h")) return CZ_ECUDA;
    cudaEventRecord(h->ev[11], h->st);
    if (!ck(h, cudaStreamSynchronize(h->st), "census")) return CZ_ECUDA;
    auto got = [&](const Buf &b) { return pin + (static_cast<const char *>(b.p) - down); };
    cudaEventElapsedTime(&s.ms_h2d, h->ev[9], h->ev[10]);
    cudaEventElapsedTime(&s.ms_d2h, h->ev[6], h->ev[11]);
    read_times(h, &s);
    s.d2h_bytes = h->down_bytes;
    s.n_primes = n; s.n_dense = h->ndense; s.n_sparse = h->nsparse; s.n_profiles = h->nprof;
    s.kernels = launches;
    const OutRecord *ho = reinterpret_cast<const OutRecord *>(got(h->b_out));
    h->hout.assign(ho, ho + h->nprof);
    if (flags & CZ_A4) std::memcpy(a4_out, got(h->b_a4), 4ull * n);
    const u32 a4err = reinterpret_cast<const u32 *>(got(h->b_counter))[8];
    const ProfState *hs = reinterpret_cast<const ProfState *>(got(h->b_state));
    for (u32 g = 0; g < h->nprof; ++g) {
        s.words += hs[g].words; s.completions += hs[g].completions; s.tests += hs[g].tests;
        s.staged_bytes += 16ull * hs[g].staged16;
    }
    // records first: a refusal names the prime and its status
    std::vector<u32> fb, rs;
    rc = check_records(h, allow_fallback ? &fb : nullptr, allow_fallback ? &rs : nullptr);
    if (rc) return rc;
    if ((flags & CZ_A4) && a4err) { h->err = "refused: A4 point count not certified"; return CZ_EREFUSED; }
    for (u32 g = 0; g < h->nprof; ++g) {
        const OutRecord &o = h->hout[g];
        CZ_RECORD &d = out[g];
        d.p = o.p; d.r = o.r; d.M = o.M; d.L = o.L; d.witness = o.witness; d.status = o.status; d.K = o.K;
    }
    // the re-runs below re-plan the handle: take the primes and record slots first
    std::vector<pw_t> fb_p;
    std::vector<u32> fb_first, fb_mask;
    for (u32 pi : fb) {
        fb_p.push_back(h->hp[pi].p);
        fb_first.push_back(h->hp[pi].first_prof);
        fb_mask.push_back(h->hp[pi].mask);
    }
    if (!rs.empty()) {
        // profiles whose best run stayed below the speculative threshold: the
        // speculation was not certified.  Their orders alone are run again with
        // the threshold one lower, and what misses that too without one, on a
        // handle of their own, so this call's plan stays resident for a replay.
        if (!h->sub) h->sub = open_sub(h);
        std::vector<pw_t> sp;
        std::vector<u32> sm;
        u32 last = 0xFFFFFFFFu;
        for (u32 g : rs) {
            const ProfDesc &D = h->hprof[g];
            if (D.prime != last) { sp.push_back(h->hp[D.prime].p); sm.push_back(0u); }
            last = D.prime;
            sm.back() |= 1u << (D.r - 2u);
        }
        u32 fflags = (flags & ~(CZ_AUTO | CZ_A4)) | CZ_SPARSE;
        if (level) fflags |= CZ_NOSPEC;
        std::vector<CZ_RECORD> tmp(rs.size());
        cz_stats s2{};
        rc = census_impl(h->sub, sp.data(), (u32)sp.size(), fflags, tmp.data(), (u32)tmp.size(), nullptr, &s2, true,
                         sm.data(), level + 1u);
        if (rc == CZ_EINVAL)                             // no filter for these orders alone
            rc = census_impl(h->sub, sp.data(), (u32)sp.size(), (fflags & ~CZ_AUTO) | CZ_DENSE, tmp.data(),
                             (u32)tmp.size(), nullptr, &s2, false, sm.data(), 0u);
        if (rc) { h->err = h->sub->err; return rc; }
        for (size_t k = 0; k < rs.size(); ++k) out[rs[k]] = tmp[k];
        s.n_respec = (u32)sp.size();
        s.n_fallback += s2.n_fallback;
        s.ms_respec = s2.ms_device + s2.ms_respec;
        s.kernels += s2.kernels;
        s.h2d_bytes += s2.h2d_bytes;
        s.d2h_bytes += s2.d2h_bytes;
        h->sub_live = true;
        h->have_plan = h->have_plan && h->sub->have_plan;
    }
    if (!fb.empty()) {
        // sparse primes whose seed could not certify a threshold: dense re-run
        const u32 fflags = (flags & ~CZ_AUTO & ~CZ_A4) | CZ_DENSE;
        u32 np = 0;
        for (u32 m : fb_mask) np += popc(m);
        std::vector<CZ_RECORD> tmp(np);
        cz_stats s2{};
        rc = census_impl(h, fb_p.data(), (u32)fb_p.size(), fflags, tmp.data(), np, nullptr, &s2, false,
                         fb_mask.data());
        if (rc) return rc;
        u32 t = 0;
        for (size_t k = 0; k < fb_p.size(); ++k)
            for (u32 j = 0; j < popc(fb_mask[k]); ++j) out[fb_first[k] + j] = tmp[t++];
        s.n_fallback += (u32)fb.size();
        s.h2d_bytes += s2.h2d_bytes;
        s.d2h_bytes += s2.d2h_bytes;
        h->have_plan = false;   // the plan now describes the fallback batch
    }
    h->last = s;
    if (stats) *stats = s;
    return CZ_OK;
}

// a census call: waves when the plane pool of the batch exceeds its budget
int census_entry(CZ_HANDLE *h, const pw_t *primes, uint32_t n, uint32_t flags, CZ_RECORD *out,
                 uint32_t out_cap, uint32_t *a4_out, cz_stats *stats) {
    if (!h) return CZ_EINVAL;
    if (n && primes && out && ((flags & CZ_A4) == 0 || a4_out)) {
        if ((flags & CZ_AUTO) == 0) flags |= CZ_AUTO;
        if (out_cap < count_profiles(primes, n)) { h->err = "output capacity below profile count"; return CZ_EINVAL; }
        u64 tot = 0;
        for (u32 i = 0; i < n && tot <= ((u64)h->cfg.plane_budget_mb << 20); ++i) tot += plane_bytes(h->cfg, primes[i], flags);
        if (tot > ((u64)h->cfg.plane_budget_mb << 20)) return census_waves(h, primes, n, flags, out, out_cap, a4_out, stats);
    }
    int rc = census_impl(h, primes, n, flags, out, out_cap, a4_out, stats, true);
    if (!rc && stats) stats->waves = 1;
    return rc;
}

}  // namespace
