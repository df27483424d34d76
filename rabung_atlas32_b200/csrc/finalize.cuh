// finalize.cuh -- per-prime setup and per-profile finalisation kernels.
//
// setup_kernel: Montgomery constants, deterministic primality (the worker's
// "worker primality" check, src/census/worker32.cu:18), a root z of exact order
// m = lcm(r) (frozen_entry.cu:18-24), the label of -1, and the r-th roots of
// unity omega^j = z^(j m / r) used by direct colour evaluation.
//
// finalize_kernel: M and witness from the packed key, L by direct powers from
// x = 2 (the reference's prefix verification, worker32.cu:38), optional direct
// certification of the witness run (certify_witness, B2/src/advance.cpp:7-13),
// K by the scientific contract (docs/METHODS.md:11-18) and the output record.
#pragma once
#include "labels.cuh"

namespace CZ_NS {

// deterministic Miller-Rabin with bases 2, 3, 5, 7, 11: no strong pseudoprime
// to all five below 2.15e12, so exact for every n < 2^33 (host and device:
// the serving runtime refuses a caller's non-prime before any device work)
__host__ __device__ inline bool is_prime_word(pw_t n) {
    if (n < 2u) return false;
    const u32 bases[5] = {2, 3, 5, 7, 11};
    for (int i = 0; i < 5; ++i) {
        if (n == bases[i]) return true;
        if (n % bases[i] == 0u) return false;
    }
    const Mont M = make_mont(n);
    pw_t d = n - 1u;
    u32 s = 0;
    while (!(d & 1u)) { d >>= 1; ++s; }
    const pw_t mone = n - M.one;          // Montgomery form of -1
    for (int i = 0; i < 5; ++i) {
        pw_t x = mpow(to_mont((pw_t)bases[i], M), d, M);
        if (x == M.one || x == mone) continue;
        bool pass = false;
        for (u32 j = 1; j < s; ++j) {
            x = mmul(x, x, M);
            if (x == mone) { pass = true; break; }
            if (x == M.one) return false;
        }
        if (!pass) return false;
    }
    return true;
}

// is_prime_word with one base per lane: the same answer, its five strong tests
// at once
__device__ __forceinline__ bool is_prime_warp(pw_t n, u32 lane) {
    if (n < 2u) return false;
    const u32 base = lane == 0 ? 2u : lane == 1 ? 3u : lane == 2 ? 5u : lane == 3 ? 7u : 11u;
    if (__any_sync(0xFFFFFFFFu, n == base)) return true;
    if (__any_sync(0xFFFFFFFFu, n % base == 0u)) return false;
    const Mont M = make_mont(n);
    pw_t d = n - 1u;
    u32 s = 0;
    while (!(d & 1u)) { d >>= 1; ++s; }
    const pw_t mone = n - M.one;          // Montgomery form of -1
    pw_t x = mpow(to_mont((pw_t)base, M), d, M);
    bool pass = x == M.one || x == mone;
    for (u32 j = 1; j < s; ++j) {
        x = mmul(x, x, M);
        pass = pass || x == mone;
    }
    return __all_sync(0xFFFFFFFFu, pass);
}

constexpr int SETUP_WARPS = 4;     // primes per CTA

// One warp per prime: every step is a power of some 50 dependent products, so
// a thread per prime takes as long as its longest chain of them (0.19 ms for
// any call); lanes take the primality bases, 32 candidates of the root of
// order m, z = a^((p-1)/m) with z^(m/q) != 1 for each prime q | m (the least a
// is taken; the reference's character_root) and the profiles
// (measured: 4096 primes 0.19 -> 0.026 ms).
__global__ void __launch_bounds__(SETUP_WARPS * 32)
setup_kernel(PrimeDesc *primes, ProfDesc *profs, ProfState *state, u32 n) {
    const u32 i = blockIdx.x * SETUP_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (i >= n) return;
    PrimeDesc P = primes[i];
    u32 status = 0;
    if (!is_prime_warp(P.p, lane)) status |= ST_ROOT;
    if (P.p > 2u) {
        const Mont M = make_mont(P.p);
        P.pinv = M.pinv; P.one = M.one; P.r2 = M.r2;
        P.z = M.one;
        if (P.m > 1u) {
            P.z = 0u;
            for (u32 a0 = 2; a0 < P.p && a0 < 100000u && !P.z; a0 += 32u) {
                const u32 a = a0 + lane;
                bool ok = a < P.p && a < 100000u;
                const pw_t z = mpow(to_mont((pw_t)(ok ? a : 1u), M), P.e, M);
                const u32 qs[4] = {2, 3, 5, 7};
                for (int k = 0; k < 4; ++k)
                    if (P.m % qs[k] == 0u && mpow(z, (pw_t)(P.m / qs[k]), M) == M.one) ok = false;
                const u32 bal = __ballot_sync(0xFFFFFFFFu, ok);
                if (bal) {
                    const int f = __ffs(bal) - 1;
#if CZ_WIDE
                    P.z = ((u64)__shfl_sync(0xFFFFFFFFu, (u32)(z >> 32), f) << 32) |
                          __shfl_sync(0xFFFFFFFFu, (u32)z, f);
#else
                    P.z = __shfl_sync(0xFFFFFFFFu, z, f);
#endif
                }
            }
            if (!P.z) status |= ST_ROOT;
        }
        P.sigma = (P.e & 1u) ? P.m / 2u : 0u;
        if (lane < P.nprof) {
            ProfDesc &D = profs[P.first_prof + lane];
            const pw_t w = mpow(P.z, (pw_t)(P.m / D.r), M);
            pw_t v = M.one;
            for (u32 j = 0; j < 9; ++j) {
                D.omega[j] = j < D.r ? v : 0u;
                v = mmul(v, w, M);
            }
            ProfState &S = state[P.first_prof + lane];
            S.best = 0; S.claim = 0; S.seed = 0; S.firstnz = 0xFFFFFFFFu;
            S.status = 0; S.active = 0; S.done = 0; S.staged16 = 0; S.words = 0; S.completions = 0; S.tests = 0;
        }
    }
    P.status = status;
    if (lane == 0) primes[i] = P;
}

// mirrors cz_profile (32-bit words) or cz_profile64 (64-bit words) in
// include/rabung_census.h; the canonical witness is at most (p-1)/2 < 2^32
struct OutRecord {
    pw_t p;
    u32 r, M, L, witness, status;
#if CZ_WIDE
    u32 reserved;
#endif
    unsigned long long K;
};

__device__ __forceinline__ u32 colour_pow(pw_t x, const Mont &M, pw_t ex, const pw_t *om, u32 r) {
    const pw_t y = mpow(to_mont(x, M), ex, M);
    for (u32 j = 0; j < r; ++j)
        if (om[j] == y) return j;
    return 0xFFFFFFFFu;
}

// least k in [0, n) where pred fails, or n: by one thread, or 32 at a time by a warp
template <bool WARP, class F>
__device__ __forceinline__ u32 first_fail(u32 n, u32 lane, F pred) {
    if constexpr (WARP) {
        for (u32 k0 = 0; k0 < n; k0 += 32u) {
            const u32 bad = __ballot_sync(0xFFFFFFFFu, k0 + lane < n && !pred(k0 + lane));
            if (bad) return k0 + (u32)__ffs(bad) - 1u;
        }
        return n;
    } else {
        u32 k = 0;
        while (k < n && pred(k)) ++k;
        return k;
    }
}

// the record of profile g: M and witness from its best key, L (dense: from the
// scan; sparse: by direct powers), optional certification, K; by one thread
// (the serving runtime) or by a warp, whose lanes take the positions.  The key
// and status words are read through volatile loads: in the serving runtime the
// last CTA leaving a profile finalises it while other CTAs' atomics on them
// have just completed.  lost: status of the grouped profiles besides their own.
template <bool WARP>
__device__ inline void finalize_one(const PrimeDesc *primes, const ProfDesc *profs, const ProfState *state,
                                    const u32 *dense_prefix, u32 g, u32 verify, u32 lost, OutRecord *out, u32 lane) {
    const ProfDesc D = profs[g];
    const PrimeDesc P = primes[D.prime];
    const unsigned long long best = *(const volatile unsigned long long *)&state[g].best;
    const u32 sstatus = *(const volatile u32 *)&state[g].status;
    const Mont M{P.p, P.pinv, P.one, P.r2};
    const pw_t p = P.p, ex = (p - 1u) / D.r;
    const u32 r = D.r;
    u32 status = P.status | sstatus | (D.grouped ? lost : 0u);
    const u32 Mlen = key_len(best), w = key_witness(best);
    if (best == 0ull && !(D.qspec && P.route == 2u)) status |= ST_VERIFY;
    if (P.route == 2u && D.qspec && Mlen < D.qspec) status |= ST_SPEC;
    // colour(1) = 0; positions 2, 3, .. of colour 0
    auto zeros = [&](u32 n) {
        return first_fail<WARP>(n, lane, [&](u32 k) { return colour_pow((pw_t)k + 2u, M, ex, D.omega, r) == 0u; });
    };
    u32 L;
    if (P.route == 1u) {
        L = dense_prefix[g];
    } else {
        const u32 n = p - 2u < (pw_t)4096u ? (u32)(p - 2u) : 4096u;
        L = 1u + zeros(n);
        if (L > 4096u) status |= ST_PREFIX;
    }
    if (verify && !(status & (ST_ROOT | ST_LABEL)) && Mlen > 0u && Mlen <= 4096u) {
        // the run [w, w+M-1] (or its mirror) is monochromatic and maximal:
        // positions w - 1 .. w + M, of which the first and last differ
        const pw_t wx = w;
        const u32 c0 = colour_pow(wx, M, ex, D.omega, r);
        bool ok = c0 != 0xFFFFFFFFu && (u64)w + Mlen - 1u <= (u64)p - 1u;
        if (ok)
            ok = first_fail<WARP>(Mlen + 2u, lane, [&](u32 k) {
                     const bool end = k == 0u || k == Mlen + 1u;
                     if (end && ((k == 0u && w <= 1u) || (k && (u64)w + Mlen > (u64)p - 1u))) return true;
                     return (colour_pow(wx + k - 1u, M, ex, D.omega, r) == c0) != end;
                 }) == Mlen + 2u;
        if (ok && P.route == 1u) {               // prefix re-check from the scan result
            const u32 n = (u64)p - 2u < (u64)L ? (u32)(p - 2u) : L;
            ok = 1u + zeros(n) == L;
        }
        if (!ok) status |= ST_VERIFY;
    }
    if (lane) return;
    OutRecord o;
    o.p = p; o.r = r; o.M = Mlen; o.L = L; o.witness = w; o.status = status;
#if CZ_WIDE
    o.reserved = 0u;
#endif
    const u64 b = ((((u64)p - 1u) / 2u) % r == 0u) ? 2ull * L + 2ull : (u64)L + 2ull;
    o.K = (u64)Mlen + 1ull > b ? (u64)Mlen + 1ull : b;
    out[D.out_slot] = o;
}

constexpr int FINAL_WARPS = 4;     // profiles per CTA

// One warp per profile: certification is M + 2 powers and the prefix another
// few, independent of one another, so a thread per profile waits for some 40
// powers in a row (measured: 13,706 profiles 0.15 -> 0.066 ms).  *claimed of
// the group filter's nitems items were handed out; where some were not (every
// loading warp gave up on a wait), no grouped profile's search was complete.
__global__ void __launch_bounds__(FINAL_WARPS * 32)
finalize_kernel(const PrimeDesc *primes, const ProfDesc *profs, const ProfState *state,
                const u32 *dense_prefix, u32 nprof, u32 verify, const u32 *claimed, u32 nitems, OutRecord *out) {
    const u32 g = blockIdx.x * FINAL_WARPS + (threadIdx.x >> 5);
    if (g >= nprof) return;
    const u32 lost = nitems && *claimed < nitems ? (u32)ST_QUEUE : 0u;
    finalize_one<true>(primes, profs, state, dense_prefix, g, verify, lost, out, threadIdx.x & 31u);
}

}  // namespace CZ_NS
