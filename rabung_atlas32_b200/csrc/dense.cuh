// dense.cuh -- exhaustive half-interval census scan (the dense oracle).
//
// Behaviour follows the reference's dense oracle (src/census/dense_oracle.cu:12-66)
// and historical dense engine (src/census/engine32/build/original_scan_gpu.cu:311-389):
// colour every x in [1, (p-1)/2] by x^((p-1)/m) mod p (one power per x, shared
// by all admissible r of p), keep per-segment run summaries, merge them in
// order, and recover the full profile by reflection with an explicit centre
// join.  The B200 design is its own: integer Montgomery powers (no FP64),
// root labels from a shared-memory hash, run boundaries from warp ballots and
// per-lane __clz on the change mask, segment summaries reduced per CTA in
// shared memory and merged per profile on the device.
//
// Within [1, (p-1)/2] the canonical witness min(s, p-(s+len-1)) of a run
// equals its start s, and the centre run (when r | (p-1)/2) has witness equal
// to its start as well, so summaries carry starts.
#pragma once
#include "labels.cuh"

namespace CZ_NS {

constexpr int DENSE_WARPS = 8;           // warps per CTA = segments per chunk
constexpr int DENSE_STEPS = 256;         // 32-wide steps per segment
constexpr u32 DENSE_SEG = 32u * DENSE_STEPS;

// ordered run summary of a contiguous interval [start, start+len)
struct Summ {
    u32 start, len;
    u32 pre, suf;        // length of the run touching the left / right end
    u32 best, bstart;    // longest run touching neither end, least start
    u32 cf, cl;          // first / last colour
};

__device__ __forceinline__ void take_best(u32 &bl, u32 &bs, u32 l, u32 s) {
    if (l > bl || (l == bl && l != 0 && s < bs)) { bl = l; bs = s; }
}

// a (left) then b (right)
__device__ __forceinline__ Summ merge_summ(const Summ &a, const Summ &b) {
    Summ o;
    o.start = a.start;
    o.len = a.len + b.len;
    o.cf = a.cf;
    o.cl = b.cl;
    bool join = a.cl == b.cf;
    o.pre = (join && a.pre == a.len) ? a.len + b.pre : a.pre;
    o.suf = (join && b.suf == b.len) ? b.len + a.suf : b.suf;
    o.best = a.best; o.bstart = a.bstart;
    take_best(o.best, o.bstart, b.best, b.bstart);
    bool a_closed_left = a.suf < a.len;   // a's suffix run does not touch a's left end
    bool b_closed_right = b.pre < b.len;
    if (join) {
        if (a_closed_left && b_closed_right)
            take_best(o.best, o.bstart, a.suf + b.pre, a.start + a.len - a.suf);
    } else {
        if (a_closed_left) take_best(o.best, o.bstart, a.suf, a.start + a.len - a.suf);
        if (b_closed_right) take_best(o.best, o.bstart, b.pre, b.start);
    }
    return o;
}

// warp-uniform run state of one profile within a warp's segment; starts are
// offsets in the segment
struct DRun {
    u32 r, mg;                   // order, its division magic
    u32 carry_c, carry_start;    // colour of the last x, start of the open run (NO_RUN: none yet)
    u32 pre, bl, bs, cf, inpre;  // prefix run, best closed run (length, start), first colour, prefix open
    u32 pad[3];
};
constexpr u32 NO_RUN = 0xFFFFFFFFu;

// longest gap between set bits of C, with its start: gaps starting at offset 0
// of the segment (o0 + bit == 0) are its prefix run and go to *pre
__device__ __forceinline__ void longest_gap(u32 C, u32 o0, u32 &len, u32 &start, u32 &pre) {
    u32 a = (u32)__ffs((int)C) - 1u;
    for (u32 rest = C & (C - 1u); rest; rest &= rest - 1u) {
        const u32 b = (u32)__ffs((int)rest) - 1u, n = b - a;
        if (o0 + a == 0u) pre = n;
        else if (n > len) { len = n; start = o0 + a; }
        a = b;
    }
}

// runs of one block of up to 32 steps: lane k holds the change bits of step k
// (bit i: the colour changes at offset base + 32 k + i).  A run closes where the
// next begins; only a run longer than the best matters, and gaps inside a word
// are looked at only if one is long enough.
__device__ __forceinline__ void block_runs(DRun &R, u32 C, u32 base, u32 lane) {
    const u32 has = __ballot_sync(0xFFFFFFFFu, C != 0u);
    if (!has) return;
    const u32 o0 = base + 32u * lane;
    const u32 own = o0 + 31u - (u32)__clz((int)(C | 1u));          // last change of the word (C != 0)
    const u32 lower = has & ((1u << lane) - 1u);
    const u32 last = __shfl_sync(0xFFFFFFFFu, own, lower ? 31 - __clz((int)lower) : 0);
    const u32 open = lower ? last : R.carry_start;
    u32 len = 0u, start = 0u, pre = 0u;
    if (C && open != NO_RUN) {
        len = o0 + (u32)__ffs((int)C) - 1u - open;
        start = open;
        if (open == 0u) { pre = len; len = 0u; }
    }
    // a gap longer than bl inside the word: bl + 1 bits from a set bit on without another
    bool look = R.inpre != 0u || R.bl == 0u;
    if (!look && R.bl < 32u) {
        u32 z = ~C, w = 1u;
        while (w < R.bl) {
            const u32 s = min(w, R.bl - w);
            z &= z >> s;
            w += s;
        }
        look = z != 0u;
    }
    if (look && C) {
        u32 gl = 0u, gs = 0u;
        longest_gap(C, o0, gl, gs, pre);
        if (gl > len) { len = gl; start = gs; }
    }
    if (R.inpre) {
        const u32 p = __reduce_max_sync(0xFFFFFFFFu, pre);
        if (p) { R.pre = p; R.inpre = 0u; }
    }
    const u32 m = __reduce_max_sync(0xFFFFFFFFu, len);
    if (m > R.bl) {
        R.bl = m;
        R.bs = __reduce_min_sync(0xFFFFFFFFu, len == m ? start : 0xFFFFFFFFu);
    }
    R.carry_start = __shfl_sync(0xFFFFFFFFu, own, 31 - __clz((int)has));
}

struct DenseArgs {
    const PrimeDesc *primes;       // all primes of the call
    const u32 *dense_idx;          // dense-local index -> prime index
    const ProfDesc *profs;
    const u32 *chunk_prefix;       // [nprimes+1] CTA chunks per prime (prefix)
    const u32 *summ_prefix;        // [nprimes] first chunk-summary slot of the prime
    u32 nprimes;
    u32 nchunks;                   // total chunks
    Summ *summ;                    // per prime: nprof x nchunks chunk summaries, profile-major
    ProfState *state;
    u32 seg;                       // x per segment (a multiple of 32; DENSE_SEG by default)
    u32 chunk0;                    // first chunk of this launch (nchunks: one past its last)
    // labels of the x coprime to 210, precomputed (dlabel_kernel): per dense-local
    // prime its offset in the label pool, or NO_LABELS; nullptr: none
    const u64 *lab_off;
    const unsigned short *lab;
};

constexpr u64 NO_LABELS = ~0ull;
constexpr u32 DLABEL_CHUNK = 16384;      // label indices per CTA
constexpr u32 DLABEL_HEAD = 8;           // labels of 2, 3, 5, 7 before a prime's array (16 bytes)

// x coprime to 210 <-> index: 48 residues in every 210 numbers
__device__ __constant__ const unsigned char W210[48] = {
    1, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71, 73, 79, 83, 89, 97, 101, 103,
    107, 109, 113, 121, 127, 131, 137, 139, 143, 149, 151, 157, 163, 167, 169, 173, 179, 181, 187, 191, 193, 197, 199,
    209};
CZ_HD u32 labels_below(u32 nh) { return (nh / 210u + 1u) * 48u; }

struct DLabelArgs {
    const PrimeDesc *primes;
    const u32 *dense_idx;
    const u32 *chunk_prefix;       // label chunks per dense-local prime (prefix)
    u32 i0, i1;                    // dense-local primes of this launch
    u32 chunk0;                    // first label chunk of this launch
    const u64 *lab_off;
    unsigned short *lab;
    ProfState *state;
};

// Labels of the x in [1, (p-1)/2] coprime to 2, 3, 5 and 7 by one power each,
// 0.23 of all x; the scan adds those of the stripped factors (the colour is a
// character).  Bound by integer multiplies, two powers in flight per thread.
__global__ void __launch_bounds__(256)
dlabel_kernel(DLabelArgs a) {
    extern __shared__ __align__(16) u32 dlsm[];
    const u32 chunk = a.chunk0 + blockIdx.x;
    u32 lo = a.i0, hi = a.i1;                     // last i with prefix[i] <= chunk
    while (hi - lo > 1u) {
        const u32 mid = (lo + hi) >> 1;
        if (a.chunk_prefix[mid] <= chunk) lo = mid; else hi = mid;
    }
    const PrimeDesc P = a.primes[a.dense_idx[lo]];
    const Mont M{P.p, P.pinv, P.one, P.r2};
    const u32 slots = hash_slots(P.m);
    pw_t *keys = reinterpret_cast<pw_t *>(dlsm);
    unsigned short *hl = reinterpret_cast<unsigned short *>(keys + slots);
    build_root_hash(keys, hl, slots, M, P.z, P.m);
    unsigned short *out = a.lab + a.lab_off[lo] + DLABEL_HEAD;
    const u32 local = chunk - a.chunk_prefix[lo], nlab = labels_below((u32)((P.p - 1u) >> 1));
    u32 bad = 0;
    auto put = [&](unsigned short *at, pw_t y, bool need) {
        u32 l = lookup_label(keys, hl, slots, y);
        if (l == 0xFFFFu) { bad |= need ? 1u : 0u; l = 0u; }
        *at = (unsigned short)l;
    };
    const u32 nh = (u32)((P.p - 1u) >> 1);
    auto number = [&](u32 k) { const u32 t = k / 48u; return (pw_t)210u * t + W210[k - 48u * t]; };
    const u32 end = min(nlab, (local + 1u) * DLABEL_CHUNK);
    for (u32 k = local * DLABEL_CHUNK + threadIdx.x; k < end; k += 512u) {
        const u32 k2 = k + 256u < end ? k + 256u : k;
        const pw_t x1 = number(k), x2 = number(k2);          // past (p-1)/2 only in the last 210: below p
        pw_t y1, y2;
        mpow2(to_mont(x1, M), to_mont(x2, M), P.e, M, y1, y2);
        put(out + k, y1, x1 <= nh);
        if (k2 != k) put(out + k2, y2, x2 <= nh);
    }
    if (local == 0u && threadIdx.x < 4u) {
        const u32 q = threadIdx.x == 0u ? 2u : threadIdx.x == 1u ? 3u : threadIdx.x == 2u ? 5u : 7u;
        put(a.lab + a.lab_off[lo] + threadIdx.x, mpow(to_mont((pw_t)q, M), P.e, M), true);
    }
    if (__syncthreads_or((int)bad) && threadIdx.x == 0) atomicOr(&a.state[P.first_prof].status, ST_LABEL);
}

// divide y by the odd q while it divides: iq = q^-1 mod 2^32, lim = floor((2^32 - 1) / q)
__device__ __forceinline__ void strip(u32 &y, u32 iq, u32 lim, u32 l, u32 &sum) {
    for (u32 t = y * iq; t <= lim; t = y * iq) { y = t; sum += l; }
}

// One CTA per (prime, chunk of DENSE_WARPS segments); one warp per segment, in
// blocks of 32 steps of 32 x: labels first, then, profile by profile, one ballot
// a step for the change bits, whose runs are closed once per block (lane k holds
// step k).  A block's bookkeeping is some 150 instructions instead of 70 a step.
// Bound by issue (61 % busy): about 80 instructions a step for the labels (the
// factors 2, 3, 5, 7 are stripped by exact divisions), 11 for each profile.
// Measured, 700 primes from 2^24 (2370 profiles): a power for every x and a
// shuffle-and-reduce a step 171 ms, with three-multiply products 134, labels
// of the x coprime to 210 kept 96, blocks of 32 steps 57 ms; 400 small primes
// from 5000 (powers in the scan) 0.33 -> 0.18 ms.  Four CTAs per SM: 3 and 5 are
// 13 % and 7 % slower.
__global__ void __launch_bounds__(DENSE_WARPS * 32, 4)
dense_scan_kernel(DenseArgs a) {
    extern __shared__ __align__(16) u32 dsm[];
    __shared__ Summ wsum[DENSE_WARPS][8];
    __shared__ __align__(16) DRun drun[DENSE_WARPS][8];
    __shared__ u32 cur_prime;
    __shared__ unsigned short slab[DENSE_WARPS][32][32];   // labels of a block of 32 steps
    __shared__ unsigned char w210[210];      // index of a residue coprime to 210
    if (a.lab_off && threadIdx.x < 48) w210[W210[threadIdx.x]] = (unsigned char)threadIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    u32 prev_prime = 0xFFFFFFFFu;
    pw_t *keys = reinterpret_cast<pw_t *>(dsm);
    unsigned short *labs = nullptr;
    u32 slots = 0;
    for (u32 chunk = a.chunk0 + blockIdx.x; chunk < a.nchunks; chunk += gridDim.x) {
        if (threadIdx.x == 0) {
            u32 lo = 0, hi = a.nprimes;           // last i with prefix[i] <= chunk
            while (hi - lo > 1) {
                u32 mid = (lo + hi) >> 1;
                if (a.chunk_prefix[mid] <= chunk) lo = mid; else hi = mid;
            }
            cur_prime = lo;
        }
        __syncthreads();
        const u32 pi = cur_prime;
        const PrimeDesc P = a.primes[a.dense_idx[pi]];
        const Mont M{P.p, P.pinv, P.one, P.r2};
        const u64 loff = a.lab_off ? a.lab_off[pi] : NO_LABELS;
        const bool stored = loff != NO_LABELS;
        if (pi != prev_prime && !stored) {
            slots = hash_slots(P.m);
            labs = reinterpret_cast<unsigned short *>(keys + slots);
            build_root_hash(keys, labs, slots, M, P.z, P.m);
            prev_prime = pi;
        }
        const unsigned short *lab = a.lab + (stored ? loff : 0ull);
        const u32 local_chunk = chunk - a.chunk_prefix[pi];
        const u32 nh = (u32)((P.p - 1u) >> 1);             // p < 2^33: fits 32 bits
        const u32 seg = local_chunk * DENSE_WARPS + warp;
        // x of the segment's first element; in 64 bits, since (p-1)/2 reaches
        // 2^32 - 1 in 64-bit words and the chunk's last segments lie past it
        const u64 seg_start64 = 1ull + (u64)seg * a.seg;
        const u32 seg_start = (u32)seg_start64;
        const u32 nprof = P.nprof;
        // per-profile run state: warp-uniform, so it lives in this warp's shared
        // records, read and written once per block of 1024 x
        if ((u32)lane < nprof) {
            const u32 r = a.profs[P.first_prof + lane].r;
            drun[warp][lane] = DRun{r, magic_of(r), 0xFFFFFFFFu, NO_RUN, 0u, 0u, 0u, 0u, 1u, {0u, 0u, 0u}};
        }
        __syncwarp();
        const bool active = seg_start64 <= (u64)nh;
        const u32 seg_end = active ? (u32)min((u64)nh, seg_start64 + a.seg - 1u) : 0u;   // inclusive
        // x is compared through its offset in the segment: seg_start + offset
        // may pass 2^32 - 1 beyond seg_end, the offset never wraps
        const u32 seg_last = seg_end - seg_start;
        u32 bad = 0;
        const u32 nsteps = active ? seg_last / 32u + 1u : 0u;
        const u32 mgm = magic_of(P.m);
        for (u32 blk = 0; blk < nsteps; blk += 32u) {
            const u32 ns = min(32u, nsteps - blk);
            // labels of the block's steps, 32 consecutive x each
            if (stored) {
                // label(x) = sum of the labels of its factors 2, 3, 5, 7 + that of the
                // rest (below 64 m < 2^18: reduced by mod_small exactly)
                const u32 l2 = lab[0], l3 = lab[1], l5 = lab[2], l7 = lab[3];
                for (u32 k = 0; k < ns; ++k) {
                    u32 y = seg_start + min((blk + k) * 32u + (u32)lane, seg_last);
                    const u32 tz = (u32)__ffs((int)y) - 1u;
                    u32 sum = tz * l2;
                    y >>= tz;
                    strip(y, 0xAAAAAAABu, 0x55555555u, l3, sum);
                    strip(y, 0xCCCCCCCDu, 0x33333333u, l5, sum);
                    strip(y, 0xB6DB6DB7u, 0x24924924u, l7, sum);
                    const u32 t = y / 210u;
                    sum += lab[DLABEL_HEAD + 48u * t + w210[y - 210u * t]];
                    slab[warp][k][lane] = (unsigned short)mod_small(sum, P.m, mgm);
                }
            } else {
                // two steps at a time: each lane's two powers are independent chains
                auto label_of = [&](pw_t y, bool valid) {
                    if (!valid) return 0u;
                    u32 l = lookup_label(keys, labs, slots, y);
                    if (l == 0xFFFFu) { bad = 1; l = 0; }
                    return l;
                };
                for (u32 k = 0; k < ns; k += 2u) {
                    const u32 o0 = (blk + k) * 32u + (u32)lane, o1 = o0 + 32u;
                    const bool v0 = o0 <= seg_last, v1 = k + 1u < ns && o1 <= seg_last;
                    const u32 x0 = seg_start + o0, x1 = seg_start + o1;
                    pw_t y0, y1;
                    mpow2(to_mont((pw_t)(v0 ? x0 : 1u), M), to_mont((pw_t)(v1 ? x1 : 1u), M), P.e, M, y0, y1);
                    slab[warp][k][lane] = (unsigned short)label_of(y0, v0);
                    if (k + 1u < ns) slab[warp][k + 1u][lane] = (unsigned short)label_of(y1, v1);
                }
            }
            __syncwarp();
            const u32 base = blk * 32u, left = seg_last + 1u - base;     // x of the segment from the block on
            for (u32 s = 0; s < nprof; ++s) {
                DRun R = drun[warp][s];
                // change bits: colour against that of the x before (the lane below,
                // lane 31 of the step before for lane 0)
                u32 mine = 0u, before = R.carry_c, c = 0u;
                for (u32 k = 0; k < ns; ++k) {
                    c = mod_small(slab[warp][k][lane], R.r, R.mg);
                    const u32 rot = __shfl_sync(0xFFFFFFFFu, c, (lane + 31) & 31);
                    const u32 C = __ballot_sync(0xFFFFFFFFu, c != (lane ? rot : before));
                    before = rot;
                    if ((u32)lane == k) mine = C;
                }
                if (blk == 0u) R.cf = mod_small(slab[warp][0][0], R.r, R.mg);
                const u32 n = left - min(left, 32u * (u32)lane);         // x of the segment in the lane's step and after
                if (n < 32u) mine &= (1u << n) - 1u;
                R.carry_c = __shfl_sync(0xFFFFFFFFu, c, (left >= 32u * ns ? 31u : (left - 1u) & 31u));
                block_runs(R, mine, base, (u32)lane);
                __syncwarp();
                drun[warp][s] = R;                         // every lane writes the same record
                __syncwarp();
            }
        }
        bad = __reduce_or_sync(0xFFFFFFFFu, bad);
        if (lane == 0) {
            if (bad) atomicOr(&a.state[P.first_prof].status, ST_LABEL);
            for (u32 s = 0; s < nprof; ++s) {
                const DRun &R = drun[warp][s];
                Summ o;
                if (active) {
                    o.start = seg_start; o.len = seg_end - seg_start + 1u;
                    o.suf = o.len - R.carry_start;
                    o.pre = R.inpre ? o.len : R.pre;
                    o.best = R.bl; o.bstart = seg_start + R.bs;
                    o.cf = R.cf; o.cl = R.carry_c;
                } else {
                    o.start = 0; o.len = 0; o.pre = o.suf = o.best = o.bstart = 0; o.cf = o.cl = 0;
                }
                wsum[warp][s] = o;
            }
        }
        __syncthreads();
        // thread s merges the CTA's segments for profile s, in order
        if (threadIdx.x < nprof) {
            const int s = threadIdx.x;
            Summ acc = wsum[0][s];
            for (int w = 1; w < DENSE_WARPS; ++w)
                if (wsum[w][s].len) acc = merge_summ(acc, wsum[w][s]);
            const u32 nch = a.chunk_prefix[pi + 1] - a.chunk_prefix[pi];
            a.summ[a.summ_prefix[pi] + (u32)s * nch + local_chunk] = acc;
        }
        __syncthreads();
    }
}

struct DenseMergeArgs {
    const PrimeDesc *primes;
    const ProfDesc *profs;
    const u32 *chunk_prefix;
    const u32 *summ_prefix;
    u32 nprimes;
    const Summ *summ;
    ProfState *state;        // indexed by global profile index
    u32 *prefix_out;         // L per global profile index
};

// one warp per dense profile: lanes merge contiguous runs of chunk summaries,
// lane 0 merges the 32 partial summaries, applies the reflection centre join.
__global__ void dense_merge_kernel(DenseMergeArgs a, const u32 *dense_prof_list, u32 ndprof) {
    const u32 gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (gw >= ndprof) return;
    const u32 gprof = dense_prof_list[gw];
    const ProfDesc D = a.profs[gprof];
    const u32 pi = D.local;                  // dense-local prime index
    const PrimeDesc P = a.primes[D.prime];
    const u32 s = gprof - P.first_prof;
    const u32 nch = a.chunk_prefix[pi + 1] - a.chunk_prefix[pi];
    const Summ *base = a.summ + a.summ_prefix[pi] + s * nch;
    const u32 per = (nch + 31u) / 32u;
    const u32 lo = min(nch, lane * per), hi = min(nch, lo + per);
    Summ acc{};
    bool have = false;
    for (u32 i = lo; i < hi; ++i) {
        Summ v = base[i];
        if (!v.len) continue;
        acc = have ? merge_summ(acc, v) : v;
        have = true;
    }
    __shared__ Summ part[32 * 8];
    Summ *mine = part + (threadIdx.x >> 5) * 32;
    mine[lane] = have ? acc : Summ{};
    __syncwarp();
    if (lane != 0) return;
    Summ tot{};
    bool h2 = false;
    for (int l = 0; l < 32; ++l) {
        if (!mine[l].len) continue;
        tot = h2 ? merge_summ(tot, mine[l]) : mine[l];
        h2 = true;
    }
    const pw_t p = P.p;
    const u32 nh = (u32)((p - 1u) >> 1), r = D.r;
    const bool sym = (nh % r) == 0u;     // r | (p-1)/2: colour(p-x) = colour(x)
    u32 bl = tot.best, bs = tot.bstart;
    u32 L;
    if (tot.pre == nh) {
        // the whole half interval is one run
        if (sym) { bl = (u32)(p - 1u); bs = 1u; L = (u32)(p - 1u); }
        else { bl = nh; bs = 1u; L = nh; }
    } else {
        take_best(bl, bs, tot.pre, 1u);                       // run from x = 1
        if (sym) take_best(bl, bs, 2u * tot.suf, nh - tot.suf + 1u);   // centre join
        else take_best(bl, bs, tot.suf, nh - tot.suf + 1u);
        L = tot.pre;                                          // colour(1) = 0
    }
    a.state[gprof].best = pack_key(bl, bs);
    a.prefix_out[gprof] = L;
}

}  // namespace CZ_NS
