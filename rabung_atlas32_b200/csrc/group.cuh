// group.cuh -- the anchor filter on groups of 32 profiles, one per word bit.
//
// Profiles of one order r whose primes lie close together share one cover
// (B, D, q), so they visit the same (numerator, denominator) anchors.  A group
// holds up to 32 of them; its colour planes are stored bit-sliced: the word of
// numerator n and plane k holds bit k of colour(n) for every member, member m
// in bit m.  One 32-bit comparison then tests one anchor position of all
// members at once, and every word is read aligned: no window has to be cut out
// of two words, a row's shift j d is a shift of the word index.  The
// mathematics (cover, anchor selection, exact completion) is that of
// sparse.cuh; what differs is stated here.
//
//  * Classes.  Numerators are stored by residue modulo 6: n = 6 i + c lives at
//    word c CL + i + I0 of its plane array.  For a row d the anchors b with
//    gcd(b, d, 6) > 1 belong to no primitive pair, so those classes are not
//    visited: 2/3 of all (b, d) remain (the odd-numerator view of sparse.cuh
//    keeps 3/4), and within a class consecutive anchors are consecutive words,
//    so a warp's loads are conflict-free.
//  * Compared planes.  The filter compares F planes: all of r = 2, 3, 4, and for
//    r >= 5 either the low two or the low three bits of the colour (two colours
//    agree in the low two with probability 0.25 to 0.28, which makes a compared
//    word worth 0.92 to 1 bit; all planes of r = 5 are worth 0.77 bit a word).
//    Which of the two, and how many stages, follows from a cost model (group_plan
//    in core.cuh).  A plane left out is read by the exact completion.
//  * Selection.  A row visits the bands [c_k, c_k + d), c_k = c_0 + k sp, with
//    6 | c_0 <= beta = ceil((t-1) d / 2) and 6 | sp <= s d.  A row's residue
//    class (step d) meets each band exactly once, two successive bands are at
//    most s steps apart, and the band c_0 and its mirror image under
//    b -> (t-1) d - b overlap or touch; so every s consecutive anchors of a row
//    hold a visited one or the mirror of a visited one, and a run of length q
//    (which holds s = q - t + 1 anchors) is found.  Visiting more only costs
//    time: every candidate is completed exactly.
//  * Cover.  The pairs (c, d), c = a + (q-1) d / 2 the centre of a window
//    a, a + d, .., a + (q-1) d of row d, a = d x mod p, form a lattice of
//    determinant p for every x; a lattice has a nonzero vector with
//    (c / E)^2 + (d / D)^2 <= 1 once E D >= 2 p / sqrt 3 (Hermite's constant of
//    dimension two; the least such vector is primitive).  So rows d <= D with
//    window centres inside the ellipse meet every window, with pi / (2 sqrt 3)
//    = 0.907 of the area that the rectangle of sparse.cuh needs (4 p by
//    Minkowski's theorem).
//  * Threshold.  q is the least speculative threshold of the members and stays
//    fixed; a member whose best run ends below it is re-run (ST_SPEC), as in
//    sparse.cuh.
//
// What bounds it, and the layout: one anchor of 32 members costs F words of
// shared memory per stage and little else (an aligned load of consecutive words
// and 3/4 of a logic operation a word), so the bound is the shared-memory load
// path, 32 words a clock and SM.  An item's tile holds one segment per stage:
// the words of the anchors' positions b - j d for 48 neighbouring rows d, whose
// segments nearly coincide, so a staged word is used about 30 times.  Measured
// on 128 primes from 4.2e9 (421 profiles): 29.9 ms on per-profile planes
// (sparse.cuh) -> 13.7 ms, load path 74 % and issue 64 % busy, 5.0e12 words
// compared a second of the 9.3e12 the load path could deliver; a block of 4096
// primes below 2^32: 757 -> 375 ms, its tables 71 -> 7 ms.  18 testing warps with
// 96 registers: 14, 16, 20, 22, 26 warps take 16.3, 15.4, 16.1, 16.0, 16.0 ms
// against 14.8 (before rows were paired), rows per item 24, 36, 72 against 48
// 16.7, 15.2, 15.6 ms.  Members of a group should be many: the cost does not
// depend on their number.
#pragma once
#include "sparse.cuh"

namespace CZ_NS {

#ifndef CZ_GROUP_TILE_WORDS               // shared-memory words of one item's tile; two tiles per CTA
#define CZ_GROUP_TILE_WORDS 22272         // 87 KiB each
#endif
#ifndef CZ_GROUP_WARPS                    // warps per CTA that test anchors (two more load items)
#define CZ_GROUP_WARPS 18
#endif
constexpr u32 G_TILE_WORDS = CZ_GROUP_TILE_WORDS;
constexpr int G_WARPS = CZ_GROUP_WARPS;
constexpr u32 G_ROWS = 48;                // rows of an item (multiple of 6)
constexpr u32 G_UNITS = G_ROWS / 6u * 24u;    // (row, class) pairs with gcd(c, d, 6) = 1
constexpr u32 G_TMIN1 = 5, G_TMAX1 = 13;  // anchor stages compiled for one plane
constexpr u32 G_TMIN2 = 3, G_TMAX2 = 8;   // for two
constexpr u32 G_TMIN3 = 3, G_TMAX3 = 6;   // and for three
constexpr u32 G_TMAX = 16;                // stage slots of a tabulated unit
constexpr u32 G_TILE3 = G_TILE_WORDS / 3u / 4u * 4u * 8u;    // byte offset of plane 2 in a tile of three planes
constexpr u32 G_OFFS = G_UNITS * G_TMAX / 8u; // 16-byte words of an offset table (16-bit tile positions)
constexpr u32 G_SMEM = 8u * G_TILE_WORDS + 32u * G_OFFS;   // dynamic shared memory of the filter
constexpr u32 G_PAD = 384;                // guard indices at both ends of a class array
#ifndef CZ_GROUP_FULL_TRIES               // bounds of the waits for an item and for a free slot
#define CZ_GROUP_FULL_TRIES MBAR_SPIN_LIMIT
#endif
#ifndef CZ_GROUP_EMPTY_TRIES
#define CZ_GROUP_EMPTY_TRIES MBAR_SPIN_LIMIT
#endif
constexpr int G_SCR_CAP = 96;             // queued anchors per warp (< 32 + two rows' step of 32)
constexpr int G_CAND_CAP = 48;            // queued candidates per warp (<= 16 + one round of 32)

struct GroupDesc {
    u32 r, np, F;         // order, planes, compared planes (the first F)
    u32 B, D, q, t, s;    // table radius, denominators, threshold, anchor stages, s = q - t + 1
    u32 E;                // elliptic cover: windows centred at |c| <= E sqrt(1 - d^2 / D^2)
    u32 n;                // members
    u32 I0, CL;           // index of i = 0 in a class array, its length (multiples of 4)
    u32 nq;               // primes <= B
    u32 rg0, nrg;         // its row groups
    u32 item0;            // its first work item
    u32 sig;              // members with colour(-1) = r/2 (0 for the others)
    u32 pad;
    u64 off, off2;        // word offsets: planes 0 and 1 interleaved (r = 2: plane 0); planes 2 and 3, one array each
    u64 pwoff;            // word offset of the colours of the primes <= B
    u32 prof[32];         // global profile index of each member
    u32 job[32];          // row of each member's prime in the label matrix
};

// rows d0 .. d0 + nrows - 1 of a group (6 | d0; d = 0 is skipped).  Wide rows
// (ncol > 0): an item is (band, chunk of W indices of the band), its tile one
// segment of W indices per stage.  Narrow rows (ncol == 0): an item is a span
// of W indices of anchors, its tile one contiguous range of numerators.
struct RowGroup {
    u32 item;             // first item, relative to the group's
    u32 d0, nrows, W, ncol;
};

// largest numerator a row visits: the windows of row d have their centre within
// E sqrt(1 - d^2/D^2) and reach (q-1) d / 2 to each side.  Single precision is
// off by less than 1 below 2^21 (D - d and D + d are exact); slack covers it.
CZ_HD u32 row_limit(u32 E, u32 D, u32 B, u32 q, u32 d, u32 slack) {
    const float f = (float)E * sqrtf((float)(D - d) * (float)(D + d)) / (float)D;
    const u32 lim = (u32)f + ((q - 1u) * d + 1u) / 2u + slack;
    return lim < B ? lim : B;
}

CZ_HD i32 floor6(i32 n) { return n >= 0 ? n / 6 : -((5 - n) / 6); }

// one work item
struct GItem {
    u32 d0, nrows, W;
    u32 wide;             // 1: segments, 0: contiguous tile
    i32 i0;               // index of the first anchor (b = 6 i0 + 6 i + c)
    u32 x;                // wide: indices of the band before this chunk
};

// index range [S, S + L) (in class-array positions) of stage j's segment
CZ_HD void seg_range(const GItem &it, u32 t, u32 j, u32 I0, u32 CL, u32 &S, u32 &L) {
    const i32 dmax = (i32)(it.d0 + it.nrows - 1u), dmin = it.d0 ? (i32)it.d0 : 1;
    i32 lo, hi;
    if (it.wide) {
        lo = floor6(6 * it.i0 - (i32)j * dmax);
        hi = floor6(6 * it.i0 + 5 - (i32)j * dmin) + (i32)it.W;
    } else {
        lo = floor6(6 * it.i0 - (i32)(t - 1u) * dmax);
        hi = it.i0 + (i32)it.W + dmax / 6 + 2;
    }
    const i32 a = (lo + (i32)I0) & ~3;                  // the layout keeps lo + I0 >= 0 (group_layout)
    i32 b = (hi + (i32)I0 + 3) & ~3;
    if (b > (i32)CL) b = (i32)CL;                       // a narrow item at the table's end
    S = (u32)a;
    L = (u32)(b - a);
}

// layout of a group's class arrays: every segment of every item starts at an
// index >= -I0 (wide rows: 6 i0 >= (t-1) d0 / 2 - 6 and (t-1) D <= 2 B, plus the
// rows' spread; narrow rows d < dn: (t-1) dn before numerator 0)
CZ_HD void group_layout(GroupDesc &G, u32 dn) {
    const u32 low = (G.t - 1u) * (dn + G_ROWS) > G.B ? (G.t - 1u) * (dn + G_ROWS) : G.B;
    G.I0 = (low / 6u + G_PAD + 3u) & ~3u;
    G.CL = (G.I0 + G.B / 6u + 1u + G_PAD + 3u) & ~3u;
}

// first row of the wide row groups (a multiple of 6): rows below it use
// contiguous tiles, whose halo of t row steps is kept under about half the tile
CZ_HD u32 group_narrow_end(u32 t, u32 F) {
    const u32 cap = G_TILE_WORDS / F / 6u;
    return cap * 9u / 20u * 6u / t / G_ROWS * G_ROWS;
}

// anchor indices of a contiguous tile whose rows end at dmax
CZ_HD u32 group_narrow_span(u32 t, u32 F, u32 dmax) {
    return G_TILE_WORDS / F / 6u - t * dmax / 6u - 16u;
}

// widest chunk (indices, a multiple of 32) of a wide item: t segments of 6
// classes, each with the rows' spread j (G_ROWS - 1) and its alignment
CZ_HD u32 group_wide_max(u32 t, u32 F) {
    u32 extra = 0u;
    for (u32 j = 0; j < t; ++j) extra += (j * (G_ROWS - 1u) + 5u) / 6u + 9u;
    return (G_TILE_WORDS / (6u * F) - extra) / t & ~31u;
}

// the class of slot k (0..23) of a block of six rows and its row: rows
// d = 0..5 mod 6 visit {1,5}, all, {1,3,5}, {1,2,4,5}, {1,3,5}, all
__device__ __constant__ const unsigned char G_UNIT[24] = {
    0x01, 0x05, 0x10, 0x11, 0x12, 0x13, 0x14, 0x15, 0x21, 0x23, 0x25, 0x31,
    0x32, 0x34, 0x35, 0x41, 0x43, 0x45, 0x50, 0x51, 0x52, 0x53, 0x54, 0x55};

// bands of row d (numerators up to lim) whose first index lies in [i0, i0 + W), for narrow rows:
// first index relative to i0, band spacing and count; ny indices per band and class c
CZ_HD void narrow_bands(const GItem &it, u32 d, u32 t, u32 s, u32 lim, u32 &first, u32 &spi, u32 &nb) {
    const u32 c0 = (((t - 1u) * d + 1u) >> 1) / 6u, i0 = (u32)it.i0, i1 = i0 + it.W, ib = lim / 6u + 1u;
    spi = s * d / 6u;
    first = 0u;
    nb = 0u;
    if (c0 >= i1 || c0 >= ib) return;
    if (spi == 0u) {                       // s d < 6: every index is visited, as one band
        first = c0 > i0 ? c0 - i0 : 0u;
        nb = 1u;
        return;
    }
    const u32 end = i1 < ib ? i1 : ib;
    const u32 klo = c0 >= i0 ? 0u : (i0 - c0 + spi - 1u) / spi;
    const u32 khi = end > c0 ? (end - c0 + spi - 1u) / spi : 0u;
    if (khi <= klo) return;
    nb = khi - klo;
    first = c0 + klo * spi - i0;
}

// ---- bit-sliced tables -----------------------------------------------------

// o = a + b mod R on bit-sliced residues below R
template <int R> struct Sliced {
    static constexpr int NP = R <= 2 ? 1 : R <= 4 ? 2 : R <= 8 ? 3 : 4;
    static constexpr bool POW2 = (R & (R - 1)) == 0;
    static __device__ __forceinline__ void add(const u32 *a, const u32 *b, u32 *o) {
        u32 s[NP + 1], c = 0u;
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            s[k] = a[k] ^ b[k] ^ c;
            c = (a[k] & b[k]) | (c & (a[k] ^ b[k]));
        }
        s[NP] = c;
        if constexpr (POW2) {
#pragma unroll
            for (int k = 0; k < NP; ++k) o[k] = s[k];
        } else {
            constexpr u32 K = (2u << NP) - (u32)R;      // s - R mod 2^(NP+1); carry out iff s >= R
            u32 v[NP + 1], g = 0u;
#pragma unroll
            for (int k = 0; k <= NP; ++k) {
                if ((K >> k) & 1u) { v[k] = ~(s[k] ^ g); g = s[k] | g; }
                else { v[k] = s[k] ^ g; g = s[k] & g; }
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) o[k] = (v[k] & g) | (s[k] & ~g);
        }
    }
};

struct LabelArgs {
    const PrimeDesc *primes;
    ProfState *state;
    const LabelJob *jobs;
    u32 nchunk;                   // CTAs per job
    unsigned short *lab;          // label pool
    const u32 *small_primes;
};

// labels of the primes up to the table end, one row per prime of the call: the
// only powers a table needs.  nchunk CTAs share a row, so calls of few primes
// fill the GPU too; two interleaved powers per thread.
__global__ void __launch_bounds__(256)
plabel_kernel(LabelArgs a) {
    extern __shared__ __align__(16) u32 lsm[];
    const LabelJob job = a.jobs[blockIdx.x / a.nchunk];
    const u32 chunk = blockIdx.x % a.nchunk;
    const PrimeDesc P = a.primes[job.prime];
    if (P.status & ST_ROOT) return;              // refused: its member is masked out of the filter
    const Mont M{P.p, P.pinv, P.one, P.r2};
    const u32 slots = hash_slots(P.m);
    pw_t *keys = reinterpret_cast<pw_t *>(lsm);
    unsigned short *hl = reinterpret_cast<unsigned short *>(keys + slots);
    build_root_hash(keys, hl, slots, M, P.z, P.m);
    const u32 per = ((job.nq + a.nchunk - 1u) / a.nchunk + 63u) & ~63u;
    const u32 lo = chunk * per, hi = min(job.nq, lo + per);
    unsigned short *row = a.lab + job.off;
    u32 bad = 0;
    for (u32 i = lo + threadIdx.x; i < hi; i += 2u * blockDim.x) {
        const u32 i2 = i + blockDim.x;
        const u32 q1 = a.small_primes[i], q2 = i2 < hi ? a.small_primes[i2] : 2u;
        pw_t y1, y2;
        mpow2(to_mont((pw_t)q1, M), to_mont((pw_t)q2, M), P.e, M, y1, y2);
        const u32 l1 = lookup_label(keys, hl, slots, y1);
        bad |= l1 == 0xFFFFu;
        row[i] = (unsigned short)(l1 == 0xFFFFu ? 0u : l1);
        if (i2 < hi) {
            const u32 l2 = lookup_label(keys, hl, slots, y2);
            bad |= l2 == 0xFFFFu;
            row[i2] = (unsigned short)(l2 == 0xFFFFu ? 0u : l2);
        }
    }
    if (__syncthreads_or((int)bad) && threadIdx.x == 0) atomicOr(&a.state[P.first_prof].status, ST_LABEL);
}

struct GTableArgs {
    const GroupDesc *groups;
    u32 ngroups;
    const unsigned short *lab;
    const LabelJob *jobs;
    u32 *pw;                      // bit-sliced colours of the primes <= B, per group
    u32 *planes, *planes2;        // pools of planes 0, 1 and of planes 2, 3
    const uint2 *chain;
    const u32 *small_primes;
};

// bit-sliced colours of 32 primes of one group per warp: lane m holds member
// m's 32 labels (four 16-byte loads), 32 ballots per plane transpose them
__global__ void __launch_bounds__(256)
gpack_kernel(GTableArgs a, u32 nblk) {
    const u32 w = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    const u32 g = w / nblk, i0 = (w % nblk) * 32u;
    if (g >= a.ngroups) return;
    const GroupDesc &G = a.groups[g];
    if (i0 >= G.nq) return;
    const u32 r = G.r, np = G.np, mg = magic_of(r);
    const bool in = lane < G.n;
    uint4 v[4];
    if (in) {
        const uint4 *row = reinterpret_cast<const uint4 *>(a.lab + a.jobs[G.job[lane]].off + i0);
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = row[k];
    }
    u32 o[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        const uint4 x = v[k >> 3];
        const u32 y = (k & 4) ? ((k & 2) ? x.w : x.z) : ((k & 2) ? x.y : x.x);
        const u32 c = in ? mod_small((k & 1) ? y >> 16 : y & 0xFFFFu, r, mg) : 0u;
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (b < (int)np) {
                const u32 bal = __ballot_sync(0xFFFFFFFFu, (c >> b) & 1u);
                if (lane == (u32)k) o[b] = bal;
            }
    }
    u32 *dst = a.pw + G.pwoff + (u64)(i0 + lane) * np;
    if (i0 + lane < G.nq)
        for (u32 b = 0; b < np; ++b) dst[b] = o[b];
}

// all planes of one position; P2 and P2 + n6 hold planes 2 and 3
template <int R>
__device__ __forceinline__ void gload(const u32 *P1, const u32 *P2, u32 n6, u32 idx, u32 *o) {
    constexpr int NP = Sliced<R>::NP;
    if constexpr (NP == 1) {
        o[0] = P1[idx];
    } else {
        const uint2 v = reinterpret_cast<const uint2 *>(P1)[idx];
        o[0] = v.x; o[1] = v.y;
        if constexpr (NP >= 3) o[2] = P2[idx];
        if constexpr (NP == 4) o[3] = P2[n6 + idx];
    }
}
template <int R>
__device__ __forceinline__ void gstore(u32 *P1, u32 *P2, u32 n6, u32 idx, const u32 *o) {
    constexpr int NP = Sliced<R>::NP;
    if constexpr (NP == 1) {
        P1[idx] = o[0];
    } else {
        reinterpret_cast<uint2 *>(P1)[idx] = make_uint2(o[0], o[1]);
        if constexpr (NP >= 3) P2[idx] = o[2];
        if constexpr (NP == 4) P2[n6 + idx] = o[3];
    }
}

// colours of +-(6 i + c), c = 0..5, for the numerators n in [lo, hi): the
// colour is a character, colour(n) = colour(q) + colour(n / q) with q the least
// prime factor of n, and n / q < lo is known already
template <int R>
__device__ __forceinline__ void gtable_index(const GTableArgs &a, const GroupDesc &G, u32 *P1, u32 *P2, u32 i,
                                             u32 lo, u32 hi) {
    constexpr int NP = Sliced<R>::NP;
    const u32 *pw = a.pw + G.pwoff;
    const u32 I0 = G.I0, CL = G.CL, n6 = 6u * CL;
    uint2 ch[6];
    const uint4 *cp = reinterpret_cast<const uint4 *>(a.chain + 6u * i);   // 48 i bytes: 16-byte aligned
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint4 v = cp[k];
        ch[2 * k] = make_uint2(v.x, v.y);
        ch[2 * k + 1] = make_uint2(v.z, v.w);
    }
    u32 sig[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) sig[k] = (R % 2 == 0 && (((u32)R / 2u) >> k & 1u)) ? G.sig : 0u;
#pragma unroll
    for (u32 c = 0; c < 6u; ++c) {
        const u32 n = 6u * i + c;
        if (n < lo || n >= hi) continue;
        u32 o[NP];
        if (n <= 1u) {
#pragma unroll
            for (int k = 0; k < NP; ++k) o[k] = 0u;
        } else {
            const u32 qi = ch[c].x & 0xFFFFFFu;
            const u32 m = (ch[c].x >> 24) == 1u ? ch[c].y : n / a.small_primes[qi];
            u32 y[NP];
#pragma unroll
            for (int k = 0; k < NP; ++k) y[k] = pw[(size_t)qi * NP + k];
            if (m > 1u) {
                u32 x[NP];
                const u32 mi = m / 6u;
                gload<R>(P1, P2, n6, (m - 6u * mi) * CL + mi + I0, x);
                Sliced<R>::add(x, y, o);
            } else {
#pragma unroll
                for (int k = 0; k < NP; ++k) o[k] = y[k];
            }
        }
        gstore<R>(P1, P2, n6, c * CL + i + I0, o);
        if (n) {
            if constexpr (R % 2 == 0) Sliced<R>::add(o, sig, o);
            gstore<R>(P1, P2, n6, (c ? 6u - c : 0u) * CL + I0 - i - (c ? 1u : 0u), o);
        }
    }
}

__device__ __forceinline__ void gtable_dispatch(const GTableArgs &a, const GroupDesc &G, u32 i, u32 lo, u32 hi) {
    u32 *P1 = a.planes + G.off, *P2 = a.planes2 + G.off2;
    switch (G.r) {
        case 2: gtable_index<2>(a, G, P1, P2, i, lo, hi); break;
        case 3: gtable_index<3>(a, G, P1, P2, i, lo, hi); break;
        case 4: gtable_index<4>(a, G, P1, P2, i, lo, hi); break;
        case 5: gtable_index<5>(a, G, P1, P2, i, lo, hi); break;
        case 6: gtable_index<6>(a, G, P1, P2, i, lo, hi); break;
        case 7: gtable_index<7>(a, G, P1, P2, i, lo, hi); break;
        case 8: gtable_index<8>(a, G, P1, P2, i, lo, hi); break;
        default: gtable_index<9>(a, G, P1, P2, i, lo, hi); break;
    }
}

constexpr u32 G_LOW = 4096;       // numerators below this: one CTA per group, level by level

// numerators below G_LOW, doubling levels [L, 2 L) with a barrier between them
__global__ void __launch_bounds__(512)
gtable_low_kernel(GTableArgs a) {
    const GroupDesc &G = a.groups[blockIdx.x];
    const u32 end = min(G_LOW, G.B + 1u);
    for (u32 lo = 0u; lo < end;) {
        const u32 hi = min(end, lo ? 2u * lo : 2u);
        for (u32 i = lo / 6u + threadIdx.x; 6u * i < hi; i += blockDim.x) gtable_dispatch(a, G, i, lo, hi);
        __syncthreads();
        lo = hi;
    }
}

// numerators [lo, 2 lo) of every group, lo >= G_LOW; one launch per level
__global__ void __launch_bounds__(256)
gtable_level_kernel(GTableArgs a, u32 lo, u32 nblk) {
    const GroupDesc &G = a.groups[blockIdx.x / nblk];
    const u32 i = lo / 6u + (blockIdx.x % nblk) * 256u + threadIdx.x;
    const u32 hi = min(2u * lo, G.B + 1u);
    if (6u * i < hi) gtable_dispatch(a, G, i, lo, hi);
}

// ---- filter ------------------------------------------------------------------

struct GFilterArgs {
    const PrimeDesc *primes;
    const ProfDesc *profs;
    ProfState *state;
    const GroupDesc *groups;
    const u32 *item0;             // first item of each group, ascending; [ngroups] = all items
    const RowGroup *rgs;
    u32 ngroups, nitems;
    const u32 *planes, *planes2;
    u32 *next;                    // work counter
};

struct GCand { u32 b, dm; };      // numerator; d << 5 | member
struct GEnt { u32 b, alive, d; }; // anchor awaiting the screen

// a warp's queues and counters, in shared memory; the length of its screen
// queue stays in a register (the stage loop would otherwise reload it)
struct GWarp {
    GEnt scr[G_SCR_CAP];
    GCand cand[G_CAND_CAP];
    u32 ncand, words, comps, err;
};

// one staged item: its group, geometry, offsets and tile (the tile in dynamic
// shared memory).  The loading warp fills it and completes `full`; every
// testing warp arrives on `empty` when it has left it.
struct GSlot {
    GroupDesc G;
    GItem it;
    u32 group;                    // 0xFFFFFFFF: no further item
    u32 live;                     // members not refused
    u32 nunits;                   // units of the item
    u32 unit;                     // next unit to claim
    u32 base[G_TMAX], S[G_TMAX], L[G_TMAX];
    u32 lim[G_ROWS], first[G_ROWS], spi[G_ROWS], nb[G_ROWS];
    // narrow: row d, numerator of rank 0, ranks | last index << 16, ny | spacing << 16;
    // wide: row d, numerator of rank 0, ranks of d | ranks of d + 6 << 16, 0
    uint4 units[G_UNITS];
    unsigned long long full, empty;
};

struct GShared {
    GFilterArgs a;                // the kernel's arguments (a copy: calls would put them on the stack)
    GSlot slot[2];
};

__device__ __forceinline__ u32 gindex(const GroupDesc &G, i32 n) {
    const u32 m = (u32)(n + (i32)(6u * G.I0)), i = m / 6u;      // n >= -B > -6 I0
    return (m - 6u * i) * G.CL + i;
}

// the F compared planes of one position in global memory
template <int F>
__device__ __forceinline__ void gplanes(const u32 *P, const u32 *P2, u32 idx, u32 *x) {
    if constexpr (F == 1) {
        x[0] = __ldg(P + idx);
    } else {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(P) + idx);
        x[0] = v.x;
        x[1] = v.y;
        if constexpr (F == 3) x[2] = __ldg(P2 + idx);
    }
}
// members that differ from the anchor's in any of them
template <int F>
__device__ __forceinline__ u32 gmismatch(const u32 *P, const u32 *P2, u32 idx, const u32 *x0) {
    u32 x[F], m = 0u;
    gplanes<F>(P, P2, idx, x);
#pragma unroll
    for (int f = 0; f < F; ++f) m |= x[f] ^ x0[f];
    return m;
}

// OR over a of R[a] & L[h - a], both indices below top, for one h
template <u32 H>
__device__ __forceinline__ u32 gpairs_h(const u32 *R, const u32 *L, u32 top) {
    u32 k = 0u;
#pragma unroll
    for (u32 a = 0; a < 6u; ++a)
        if (a < top && a <= H && H - a < top) k |= R[a] & L[H - a];
    return k;
}
__device__ __forceinline__ u32 gpairs(const u32 *R, const u32 *L, u32 h, u32 top) {
    switch (h) {
        case 1: return gpairs_h<1>(R, L, top);
        case 2: return gpairs_h<2>(R, L, top);
        case 3: return gpairs_h<3>(R, L, top);
        case 4: return gpairs_h<4>(R, L, top);
        case 5: return gpairs_h<5>(R, L, top);
        case 6: return gpairs_h<6>(R, L, top);
        case 7: return gpairs_h<7>(R, L, top);
        case 8: return gpairs_h<8>(R, L, top);
        case 9: return gpairs_h<9>(R, L, top);
        case 10: return gpairs_h<10>(R, L, top);
        default: return 0u;                                // no two tested counts below top reach h
    }
}

// bilateral screen of one anchor.  R[a] (L[a]): members that match the first a
// positions right (left) of its t; numerators outside [-B, B] are unknown and
// match.  A member's run can reach q only if it matches a positions on one side
// and h - a on the other (h = q - t), where a side that matches all tested
// positions is unbounded.  Three positions a side are tested first, the next
// three only where a member is left; the loads of a round are independent.
template <int F>
__device__ __forceinline__ u32 gscreen(const GroupDesc &G, const u32 *P, const u32 *P2, u32 b, u32 d, u32 alive) {
    const u32 h = G.q - G.t;
    if (h == 0u) return alive;
    const i32 B = (i32)G.B, t = (i32)G.t;
    u32 x0[F], R[7], L[7];
    gplanes<F>(P, P2, gindex(G, (i32)b), x0);
    R[0] = L[0] = alive;
    u32 keep = alive;
#pragma unroll
    for (u32 k0 = 0; k0 < 6u; k0 += 3u) {
        u32 mr[3], ml[3];
#pragma unroll
        for (u32 k = 0; k < 3u; ++k) {
            const i32 nr = (i32)(b + (k0 + k + 1u) * d), nl = (i32)b - (t + (i32)(k0 + k)) * (i32)d;
            mr[k] = nr <= B ? gmismatch<F>(P, P2, gindex(G, nr), x0) : 0u;
            ml[k] = nl >= -B ? gmismatch<F>(P, P2, gindex(G, nl), x0) : 0u;
        }
        const u32 top = k0 + 3u;
#pragma unroll
        for (u32 k = 0; k < 3u; ++k) {
            R[k0 + k + 1u] = R[k0 + k] & ~mr[k];
            L[k0 + k + 1u] = L[k0 + k] & ~ml[k];
        }
        keep = R[top] | L[top] | gpairs(R, L, h, k0 + 3u);
        if (!keep) return 0u;
    }
    return keep;
}

// colour of numerator n for member mb, all planes
__device__ __forceinline__ u32 gcolour(const GroupDesc &G, const u32 *P, const u32 *P2, i32 n, u32 mb) {
    const u32 u = gindex(G, n);
    if (G.np == 1u) return (__ldg(P + u) >> mb) & 1u;
    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(P) + u);
    u32 c = ((v.x >> mb) & 1u) | (((v.y >> mb) & 1u) << 1);
    if (G.np >= 3u) c |= ((__ldg(P2 + u) >> mb) & 1u) << 2;
    if (G.np == 4u) c |= ((__ldg(P2 + 6u * G.CL + u) >> mb) & 1u) << 3;
    return c;
}

__device__ __forceinline__ u32 gdirect(pw_t x, const Mont &M, pw_t ex, const pw_t *om, u32 r) {
    const pw_t y = mpow(to_mont(x, M), ex, M);
    for (u32 j = 0; j < r; ++j)
        if (om[j] == y) return j;
    return 0xFFFFFFFFu;
}

// exact completion of one candidate (member mb, anchor b / d): the run is
// walked both ways on the table first; a run closed on both sides inside the
// table that is shorter than the member's best (or than q) needs no position.
// Otherwise x = b / d mod p, and where the table ends the walk goes on by
// direct powers.
__device__ __forceinline__ void gcomplete(const GShared &sh, const GroupDesc &G, u32 b, u32 dm, u32 &err) {
    const GFilterArgs &a = sh.a;
    const u32 mb = dm & 31u, d = dm >> 5;
    const u32 *P = a.planes + G.off, *P2 = a.planes2 + G.off2;
    const i32 B = (i32)G.B;
    const u32 g = G.prof[mb];
    const u32 cb = gcolour(G, P, P2, (i32)b, mb);
    u32 right = 0, left = 0;
    bool openr = false, openl = false;
    for (u32 k = 1;; ++k) {                            // numerator b + k d
        if (k > RUN_CAP) { err = 1; return; }
        const i64 n = (i64)b + (i64)k * d;
        if (n > B) { openr = true; break; }
        if (gcolour(G, P, P2, (i32)n, mb) != cb) break;
        right = k;
    }
    for (u32 k = 1;; ++k) {                            // numerator b - k d; 0 is x = 0, outside the domain
        if (k > RUN_CAP) { err = 1; return; }
        const i64 n = (i64)b - (i64)k * d;
        if (n < -(i64)B) { openl = true; break; }
        if (n == 0 || gcolour(G, P, P2, (i32)n, mb) != cb) break;
        left = k;
    }
    ProfState *st = a.state + g;
    if (!openr && !openl) {
        const u32 len = right + left + 1u;
        if (len < G.q || len < key_len(*(volatile unsigned long long *)&st->best)) return;
    }
    const ProfDesc &D = a.profs[g];
    const PrimeDesc &Q = a.primes[D.prime];
    const pw_t p = Q.p;
    const Mont M{p, Q.pinv, Q.one, Q.r2};
    const u32 r = G.r;
    const pw_t dinv = mpow(to_mont((pw_t)d, M), p - 2u, M);
    const pw_t x = mmul((pw_t)b, dinv, M);
    if (x == 0u) return;
    if (openr || openl) {
        const pw_t ex = (p - 1u) / r;
        const u32 cd = gcolour(G, P, P2, (i32)d, mb);
        const u32 A = cb >= cd ? cb - cd : cb + r - cd;    // absolute colour of x
        if (openr)
            for (u32 k = right + 1u; (u64)x + k < (u64)p; ++k) {
                if (k > RUN_CAP) { err = 1; return; }
                if (gdirect(x + k, M, ex, D.omega, r) != A) break;
                right = k;
            }
        if (openl)
            for (u32 k = left + 1u; k < x; ++k) {
                if (k > RUN_CAP) { err = 1; return; }
                if (gdirect(x - k, M, ex, D.omega, r) != A) break;
                left = k;
            }
    }
    const pw_t s = x - left, e = x + right;
    const pw_t w = s < p - e ? s : p - e;
    atomicMax(&st->best, (unsigned long long)pack_key((u32)(e - s + 1u), (u32)w));
}

// complete the first `count` (<= 32) of n queued candidates, one per lane
__device__ __noinline__ void gflush(const GShared &sh, const GroupDesc &G, GWarp &w, u32 n, u32 count, u32 lane) {
    if (lane < count) {
        const GCand c = w.cand[lane];
        u32 e = 0;
        gcomplete(sh, G, c.b, c.dm, e);
        if (e) w.err = 1u;
    }
    __syncwarp();
    GCand mv{0u, 0u};
    const bool has = lane < n - count;
    if (has) mv = w.cand[count + lane];
    __syncwarp();
    if (has) w.cand[lane] = mv;
    if (lane == 0) w.comps += count;
    __syncwarp();
}

// screen the n queued anchors, 32 at a time and one per lane, and queue the
// members that survive; fewer than 32 stay (none with `all`).  Returns how many.
template <int F>
__device__ __noinline__ u32 gscreen_batch(const GShared &sh, const GroupDesc &G, GWarp &w, u32 n, bool all, u32 lane) {
    u32 nc = w.ncand;
    __syncwarp();
    while (n >= 32u || (all && n)) {
        // the last entries: the others need no move
        const u32 count = min(32u, n);
        n -= count;
        u32 keep = 0u, b = 0u, d = 0u;
        if (lane < count) {
            const GEnt e = w.scr[n + lane];
            b = e.b;
            d = e.d;
            keep = gscreen<F>(G, sh.a.planes + G.off, sh.a.planes2 + G.off2, b, d, e.alive);
        }
        for (u32 bal = __ballot_sync(0xFFFFFFFFu, keep != 0u); bal; bal = __ballot_sync(0xFFFFFFFFu, keep != 0u)) {
            if (keep) {
                const u32 mb = __ffs(keep) - 1u;
                keep &= keep - 1u;
                w.cand[nc + __popc(bal & ((1u << lane) - 1u))] = GCand{b, (d << 5) | mb};
            }
            nc += __popc(bal);
            __syncwarp();
            if (nc > 16u) {
                const u32 m = min(32u, nc);
                gflush(sh, G, w, nc, m, lane);
                nc -= m;
            }
        }
    }
    __syncwarp();
    if (lane == 0) w.ncand = nc;
    __syncwarp();
    return n;
}

// the F planes' words of all T stages for one anchor per lane.  ad[j] is the
// lane's shared byte address of stage j in the tile's planes 0 and 1, ad3[j]
// (F = 3) in its plane 2; disp (indices) is a compile-time displacement.
template <int F, int T, int J0 = 0>
__device__ __forceinline__ void gwords(const u32 *ad, const u32 *ad3, u32 disp, u32 (*x)[T]) {
#pragma unroll
    for (int j = J0; j < T; ++j) {
        if constexpr (F == 1) {
            x[0][j] = lds32(ad[j] + 4u * disp);
        } else {
            const uint2 v = lds64(ad[j] + 8u * disp);
            x[0][j] = v.x;
            x[1][j] = v.y;
            if constexpr (F == 3) x[2][j] = lds32(ad3[j] + 4u * disp);
        }
    }
}

// members that agree on all T stages.  Two words' differences from the base
// are one three-input operation, three partial results another, so a compared
// word costs 3/4 of a logic operation; two accumulators shorten the chains.
template <int F, int T>
__device__ __forceinline__ u32 gagree(const u32 (*x)[T]) {
    u32 m = 0u, a = 0u;
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
        for (int j = 1; j < T; j += 4) {
            u32 p = x[f][j] ^ x[f][0], q = 0u;
            if (j + 1 < T) p |= x[f][j + 1] ^ x[f][0];
            if (j + 2 < T) q = x[f][j + 2] ^ x[f][0];
            if (j + 3 < T) q |= x[f][j + 3] ^ x[f][0];
            if (j & 4) a = a | p | q;
            else m = m | p | q;
        }
    return ~(m | a);
}
template <int F, int T>
__device__ __forceinline__ u32 gtest(const u32 *ad, const u32 *ad3, u32 disp) {
    u32 x[F][T];
    gwords<F, T>(ad, ad3, disp, x);
    return gagree<F, T>(x);
}
// the same anchors (same numerators) of two rows: the base words are read once
template <int F, int T>
__device__ __forceinline__ void gtest2(const u32 *ad, const u32 *ad3, const u32 *bd, const u32 *bd3, u32 disp, u32 &r0,
                                       u32 &r1) {
    u32 x[F][T], y[F][T];
    gwords<F, T>(ad, ad3, disp, x);
    gwords<F, T, 1>(bd, bd3, disp, y);
#pragma unroll
    for (int f = 0; f < F; ++f) y[f][0] = x[f][0];
    r0 = gagree<F, T>(x);
    r1 = gagree<F, T>(y);
}

// queue the surviving anchors of one step behind the n queued ones; true when
// a full batch waits
__device__ __forceinline__ bool gqueue(GEnt *scr, u32 &n, u32 b, u32 d, u32 alive, u32 lane) {
    const u32 bal = __ballot_sync(0xFFFFFFFFu, alive != 0u);
    if (!bal) return false;
    if (alive) scr[n + __popc(bal & ((1u << lane) - 1u))] = GEnt{b, alive, d};
    n += __popc(bal);
    __syncwarp();
    return n >= 32u;
}

// byte addresses of a unit's stages: tabulated positions, from index l0 on
template <int F, int T>
__device__ __forceinline__ void gaddresses(const uint4 *of, u32 tile, u32 l0, u32 *ad, u32 *ad3) {
    constexpr u32 A = F == 1 ? 4u : 8u;                    // bytes of planes 0 and 1 per index
    u32 v[8];
    const uint4 p = of[0];
    v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w;
    if constexpr (T > 8) {
        const uint4 r = of[1];
        v[4] = r.x; v[5] = r.y; v[6] = r.z; v[7] = r.w;
    }
    const u32 t0 = tile + l0 * A, t3 = tile + G_TILE3 + l0 * 4u;
#pragma unroll
    for (int j = 0; j < T; ++j) {
        const u32 k = (j & 1) ? v[j >> 1] >> 16 : v[j >> 1] & 0xFFFFu;
        ad[j] = t0 + k * A;
        if constexpr (F == 3) ad3[j] = t3 + k * 4u;
    }
}

// One unit from rank `i` on: false when a full batch waits for the screen
// first (the caller screens with none of this state live and resumes at i),
// true when the unit is done.  A wide unit is a class of two rows d, d + 6,
// whose bands start together: ranks are the chunk's consecutive indices, the
// anchors' own words are read once for both rows (measured on 128 primes from
// 4.2e9: two steps of one row 14.8 ms, one step of two rows 13.7).  A narrow unit
// is a class of one row: ranks run over the indices of its bands, ny a band, spi apart.
template <int F, int T>
__device__ __forceinline__ bool gunit(const uint4 U, const uint4 *of, u32 tile, u32 live, u32 &i, GWarp &w, u32 &n,
                                      u32 lane) {
    constexpr u32 A = F == 1 ? 4u : 8u;
    u32 ad[T], ad3[F == 3 ? T : 1];
    if (U.w == 0u) {
        const u32 ca = U.z & 0xFFFFu, cb = U.z >> 16, most = max(ca, cb), least = min(ca, cb);
        u32 bd[T], bd3[F == 3 ? T : 1];
        gaddresses<F, T>(of, tile, i + lane, ad, ad3);
        gaddresses<F, T>(of + G_TMAX / 8u, tile, i + lane, bd, bd3);
        u32 b = U.y + 6u * (i + lane);
        for (;;) {
#pragma unroll
            for (u32 h = 0; h < 2u; ++h) {                 // the second step's displacement is a constant
                u32 x0, x1;
                gtest2<F, T>(ad, ad3, bd, bd3, 32u * h, x0, x1);
                x0 &= live;
                x1 &= live;
                if (i + 32u > least) {                     // partial in one row or both
                    if (i + lane >= ca) x0 = 0u;
                    if (i + lane >= cb) x1 = 0u;
                }
                i += 32u;
                if (__any_sync(0xFFFFFFFFu, (x0 | x1) != 0u)) {
                    gqueue(w.scr, n, b + 192u * h, U.x, x0, lane);
                    if (gqueue(w.scr, n, b + 192u * h, U.x + 6u, x1, lane) || n >= 32u) return i >= most;
                }
                if (i >= most) return true;
            }
#pragma unroll
            for (int j = 0; j < T; ++j) {
                ad[j] += 64u * A;
                if (j) bd[j] += 64u * A;
                if constexpr (F == 3) {
                    ad3[j] += 256u;
                    if (j) bd3[j] += 256u;
                }
            }
            b += 384u;
        }
    }
    gaddresses<F, T>(of, tile, 0u, ad, ad3);
    const u32 cnt = U.z & 0xFFFFu;
    const u32 ny = U.w & 0xFFFFu, spi = U.w >> 16, last = U.z >> 16;
    const float rny = __frcp_rn(__uint2float_rn(ny));
    const u32 k = div_rcp(i + lane, ny, rny);
    u32 y = i + lane - k * ny;
    const u32 q32 = div_rcp(32u, ny, rny), r32 = 32u - q32 * ny;
    u32 ix = k * spi + y;
    const u32 dA = q32 * spi + r32, dB = spi - ny;
    for (;;) {
        const bool ok = i + lane < cnt && ix <= last;
        const u32 o = ok ? ix : 0u;
        u32 am[T], am3[F == 3 ? T : 1];
#pragma unroll
        for (int j = 0; j < T; ++j) {
            am[j] = ad[j] + o * A;
            if constexpr (F == 3) am3[j] = ad3[j] + o * 4u;
        }
        u32 alive = gtest<F, T>(am, am3, 0u) & live;
        if (!ok) alive = 0u;
        i += 32u;
        if (gqueue(w.scr, n, U.y + 6u * ix, U.x, alive, lane)) return i >= cnt;
        if (i >= cnt) return true;
        y += r32;
        const bool wrap = y >= ny;
        if (wrap) y -= ny;
        ix += wrap ? dA + dB : dA;
    }
}

// the units of a staged item, claimed by warps
template <int F, int T>
__device__ __forceinline__ void gunits(const GShared &sh, GSlot &sl, const uint4 *offs, u32 tile, GWarp &w, u32 &n,
                                       u32 lane) {
    const u32 live = sl.live, nunits = sl.nunits;
    u32 words = 0u;
    for (;;) {
        u32 u = 0;
        if (lane == 0) u = atomicAdd(&sl.unit, 1u);
        u = __shfl_sync(0xFFFFFFFFu, u, 0);
        if (u >= nunits) break;
        const uint4 U = sl.units[u];
        const u32 cnt = (U.z & 0xFFFFu) + (U.w ? 0u : U.z >> 16);
        if (cnt == 0u) continue;
        words += cnt;
        u32 i = 0;
        for (;;) {
            const bool done = gunit<F, T>(U, offs + u * (U.w ? 1u : 2u) * (G_TMAX / 8u), tile, live, i, w, n, lane);
            if (n >= 32u) n = gscreen_batch<F>(sh, sl.G, w, n, false, lane);
            if (done) break;
        }
    }
    if (lane == 0) w.words += words;
}

__device__ __forceinline__ void gunits_t(const GShared &sh, GSlot &sl, const uint4 *offs, u32 tile, GWarp &w, u32 &n,
                                         u32 lane) {
    if (sl.G.F == 1u) {
        switch (sl.G.t) {
            case 5: gunits<1, 5>(sh, sl, offs, tile, w, n, lane); break;
            case 6: gunits<1, 6>(sh, sl, offs, tile, w, n, lane); break;
            case 7: gunits<1, 7>(sh, sl, offs, tile, w, n, lane); break;
            case 8: gunits<1, 8>(sh, sl, offs, tile, w, n, lane); break;
            case 9: gunits<1, 9>(sh, sl, offs, tile, w, n, lane); break;
            case 10: gunits<1, 10>(sh, sl, offs, tile, w, n, lane); break;
            case 11: gunits<1, 11>(sh, sl, offs, tile, w, n, lane); break;
            case 12: gunits<1, 12>(sh, sl, offs, tile, w, n, lane); break;
            default: gunits<1, 13>(sh, sl, offs, tile, w, n, lane); break;
        }
    } else if (sl.G.F == 2u) {
        switch (sl.G.t) {
            case 3: gunits<2, 3>(sh, sl, offs, tile, w, n, lane); break;
            case 4: gunits<2, 4>(sh, sl, offs, tile, w, n, lane); break;
            case 5: gunits<2, 5>(sh, sl, offs, tile, w, n, lane); break;
            case 6: gunits<2, 6>(sh, sl, offs, tile, w, n, lane); break;
            case 7: gunits<2, 7>(sh, sl, offs, tile, w, n, lane); break;
            default: gunits<2, 8>(sh, sl, offs, tile, w, n, lane); break;
        }
    } else {
        switch (sl.G.t) {
            case 3: gunits<3, 3>(sh, sl, offs, tile, w, n, lane); break;
            case 4: gunits<3, 4>(sh, sl, offs, tile, w, n, lane); break;
            case 5: gunits<3, 5>(sh, sl, offs, tile, w, n, lane); break;
            default: gunits<3, 6>(sh, sl, offs, tile, w, n, lane); break;
        }
    }
}

// every member of the group falls back (a failed item or candidate); one warp
__device__ __forceinline__ void gfail(const GFilterArgs &a, const GroupDesc &G, u32 st, u32 lane) {
    if (lane < G.n) atomicOr(&a.state[G.prof[lane]].status, st);
}

// a warp leaves its group: queues, counters and errors
__device__ __noinline__ void gleave(const GShared &sh, const GroupDesc &G, GWarp &w, u32 n, u32 lane) {
    if (n) {
        if (G.F == 1u) gscreen_batch<1>(sh, G, w, n, true, lane);
        else if (G.F == 2u) gscreen_batch<2>(sh, G, w, n, true, lane);
        else gscreen_batch<3>(sh, G, w, n, true, lane);
    }
    const u32 nc = w.ncand;
    if (nc) gflush(sh, G, w, nc, nc, lane);
    const u32 err = w.err;
    __syncwarp();
    if (lane == 0) {
        ProfState *st = sh.a.state + G.prof[0];
        atomicAdd(&st->words, (unsigned long long)w.words);
        atomicAdd(&st->tests, (unsigned long long)w.words * G.t * G.F);
        atomicAdd(&st->completions, (unsigned long long)w.comps);
        w.ncand = w.words = w.comps = w.err = 0u;
    }
    __syncwarp();
    if (err) gfail(sh.a, G, ST_QUEUE, lane);
}

__device__ __forceinline__ void mbar_arrive(u32 mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(mbar) : "memory");
}
// announce `bytes` of transaction without arriving
__device__ __forceinline__ void mbar_expect(u32 mbar, u32 bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" :: "r"(mbar), "r"(bytes) : "memory");
}

// last index k in [0, n) with key(k) <= v (key(0) <= v, ascending): 32 probes per round
template <class K>
__device__ __forceinline__ u32 warp_upper(u32 n, u32 v, u32 lane, K key) {
    u32 lo = 0;
    while (n > 1u) {
        const u32 step = (n + 31u) / 32u, k = lane * step;
        const bool le = k < n && key(lo + k) <= v;
        const u32 last = 31u - __clz(__ballot_sync(0xFFFFFFFFu, le));   // lane 0 always holds
        lo += last * step;
        n = min(step, n - last * step);
    }
    return lo;
}

// the next non-empty item: its group and geometry; false when none is left
__device__ __forceinline__ bool gclaim(const GFilterArgs &a, u32 lane, u32 &g, GItem &it) {
    for (;;) {
        u32 item = 0;
        if (lane == 0) item = atomicAdd(a.next, 1u);
        item = __shfl_sync(0xFFFFFFFFu, item, 0);
        if (item >= a.nitems) return false;
        g = warp_upper(a.ngroups, item, lane, [&](u32 k) { return a.item0[k]; });
        const GroupDesc &G = a.groups[g];
        const RowGroup *rg = a.rgs + G.rg0;
        const u32 rel = item - G.item0, t = G.t, s = G.s, B = G.B;
        const RowGroup Rg = rg[warp_upper(G.nrg, rel, lane, [&](u32 j) { return rg[j].item; })];
        const u32 j = rel - Rg.item;
        it.d0 = Rg.d0; it.nrows = Rg.nrows; it.W = Rg.W; it.wide = Rg.ncol != 0u; it.x = 0u;
        if (Rg.ncol) {
            const u32 band = j / Rg.ncol, x = j - band * Rg.ncol;
            it.x = x * Rg.W;
            it.i0 = (i32)((((t - 1u) * Rg.d0 + 1u) >> 1) / 6u + band * (s * Rg.d0 / 6u) + it.x);
        } else {
            it.i0 = (i32)(j * Rg.W);
        }
        if (6 * it.i0 <= (i32)B) return true;              // else: a last band's chunk past B, without anchors
    }
}

// a loading warp stages item `it` of group g in its slot: the bulk copies of
// the tile first, then, while they run, the group, the units and the tabulated
// offsets; the arrival on sl.full releases them.  false: the tile does not fit.
__device__ __noinline__ bool gstage(GShared &sh, GSlot &sl, unsigned short *offs, u32 tile, u32 g, const GItem it,
                                    u32 lane) {
    const GFilterArgs &a = sh.a;
    const u32 full = smem_addr(&sl.full);
    if (g != sl.group) {
        const u32 *src = reinterpret_cast<const u32 *>(a.groups + g);
        for (u32 i = lane; i < sizeof(GroupDesc) / 4u; i += 32u) reinterpret_cast<u32 *>(&sl.G)[i] = src[i];
        __syncwarp();
        // a refused member (not a prime) matches every window: it is left out
        const bool ok = lane < sl.G.n && !(a.primes[a.profs[sl.G.prof[lane]].prime].status & ST_ROOT);
        const u32 live = __ballot_sync(0xFFFFFFFFu, ok);
        if (lane == 0) { sl.live = live; sl.group = g; }
        __syncwarp();
    }
    const GroupDesc &G = sl.G;
    const u32 t = G.t, F = G.F, I0 = G.I0, nseg = it.wide ? t : 1u;
    u32 S = 0, L = 0;
    if (lane < nseg) seg_range(it, t, lane, I0, G.CL, S, L);
    u32 incl = 6u * L;
    for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (u32)o) incl += y;
    }
    const u32 total = __shfl_sync(0xFFFFFFFFu, incl, 31);  // positions of the tile
    if (total > (F == 3u ? G_TILE3 / 8u : G_TILE_WORDS / F) || total == 0u) { gfail(a, G, ST_COVER, lane); return false; }
    if (lane < nseg) { sl.base[lane] = incl - 6u * L; sl.S[lane] = S; sl.L[lane] = L; }
    __syncwarp();
    {
        const u32 A = F == 1u ? 1u : 2u;                   // planes 0 and 1 interleaved, plane 2 apart
        if (lane == 0) mbar_expect(full, total * F * 4u);
        __syncwarp();
        for (u32 k = lane; k < 6u * nseg; k += 32u) {
            const u32 j = k / 6u, c = k - 6u * j, Lj = sl.L[j], at = sl.base[j] + c * Lj;
            const u64 from = (u64)c * G.CL + sl.S[j];
            bulk_load(tile + at * A * 4u, a.planes + G.off + from * A, Lj * A * 4u, full);
            if (F == 3u) bulk_load(tile + G_TILE3 + at * 4u, a.planes2 + G.off2 + from, Lj * 4u, full);
        }
    }
    // rows: largest numerator, and the bands of narrow rows
    for (u32 k = lane; k < it.nrows; k += 32u) {
        const u32 d = it.d0 + k;
        u32 first = 0u, spi = 0u, nb = 0u;
        const u32 lim = d ? row_limit(G.E, G.D, G.B, G.q, d, 2u) : 0u;
        if (!it.wide && d) narrow_bands(it, d, t, G.s, lim, first, spi, nb);
        sl.lim[k] = lim; sl.first[k] = first; sl.spi[k] = spi; sl.nb[k] = nb;
    }
    __syncwarp();
    // units: their ranks (a narrow unit's rank 0 is its first band's first index)
    const u32 nunits = it.wide ? (it.nrows + 11u) / 12u * 24u : (it.nrows + 5u) / 6u * 24u;
    for (u32 u = lane; u < nunits; u += 32u) {
        const u32 blk = u / 24u, e = G_UNIT[u - 24u * blk], c = e & 15u;
        uint4 U = make_uint4(0u, 0u, 0u, 0u);
        if (it.wide) {
            // the chunk's part of the bands [c_k, c_k + d), up to lim, of rows d and d + 6
            const u32 row = 12u * blk + (e >> 4);
            U.x = it.d0 + row;
            U.y = 6u * (u32)it.i0 + c;
#pragma unroll
            for (u32 h = 0; h < 2u; ++h) {
                if (row + 6u * h >= it.nrows) continue;
                const i32 len = min(min((i32)(6u * it.W), (i32)(U.x + 6u * h) - (i32)(6u * it.x)),
                                    (i32)sl.lim[row + 6u * h] + 1 - 6 * it.i0);
                if (len > (i32)c) U.z |= ((u32)len - c + 5u) / 6u << (16u * h);
            }
        } else {
            const u32 row = 6u * blk + (e >> 4), d = it.d0 + row;
            U.x = d;
            if (row < it.nrows && d && sl.nb[row]) {
                // indices of the class in a band (6 | c_k); without spacing: up to the tile's end
                const u32 lim = sl.lim[row], spi = sl.spi[row], first = sl.first[row];
                const u32 ny = spi ? (d > c ? (d - c + 5u) / 6u : 0u) : it.W - first;
                U.y = 6u * ((u32)it.i0 + first) + c;
                const u32 cnt = sl.nb[row] * ny;
                if (cnt && U.y <= lim) {
                    U.z = cnt | min((lim - U.y) / 6u, 0xFFFFu) << 16;
                    U.w = ny | spi << 16;
                }
            }
        }
        sl.units[u] = U;
    }
    // offsets: the tile position of stage j of the anchor at index 0, row d, class
    // c is that of n = 6 i0 + c - j d, i.e. base + (n mod 6) L + floor(n / 6) + I0 - S
    // of the stage's segment; lane (row, j) divides j d by 6 once for the row's
    // classes.  A wide unit's two rows follow each other; where the second is
    // past the item's rows, it reads as the first (its ranks are none).
    for (u32 k = lane, n = it.nrows * t; k < n; k += 32u) {
        const u32 row = k / t, j = k - row * t, sj = it.wide ? j : 0u;
        const u32 blk = row / 6u, m6 = row - 6u * blk, e = j * (it.d0 + row), q6 = e / 6u;
        const i32 rho = (i32)(e - 6u * q6), Lj = (i32)sl.L[sj];
        const i32 at = (i32)(sl.base[sj] + sl.first[row] + (u32)it.i0 + I0 - sl.S[sj]) - (i32)q6;
        const u32 u0 = (u32)(0x120F0B080200ull >> (8u * m6)) & 0xFFu;          // first slot of the row: 0 2 8 11 15 18
        const u32 u1 = m6 == 5u ? 24u : (u32)(0x120F0B080200ull >> (8u * m6 + 8u)) & 0xFFu;
        const bool twice = it.wide && !(blk & 1u) && row + 6u >= it.nrows;
        for (u32 u = u0; u < u1; ++u) {
            const i32 cc = (i32)(G_UNIT[u] & 15u) - rho;
            const unsigned short o = (unsigned short)(at + cc * Lj + (cc < 0 ? 6 * Lj - 1 : 0));
            const u32 slot = it.wide ? 2u * (24u * (blk >> 1) + u) + (blk & 1u) : 24u * blk + u;
            offs[slot * G_TMAX + j] = o;
            if (twice) offs[(slot + 1u) * G_TMAX + j] = o;
        }
    }
    if (lane == 0) {
        sl.it = it;
        sl.nunits = nunits;
        sl.unit = 0u;
        atomicAdd(&a.state[G.prof[0]].staged16, total * F / 4u);
    }
    __threadfence_block();
    __syncwarp();
    if (lane == 0) mbar_arrive(full);
    __syncwarp();
    return true;
}

// One CTA per SM.  The last two warps each stage items into a slot of their
// own; the others test the slots in turn, each moving to the next as soon as
// no unit is left for it, so neither a tile's copy nor an item's end holds the
// SM up.  Every wait is bounded.  A testing warp whose wait runs out marks the
// group it held and leaves; the loading warps then find their slots taken, mark
// the group in the slot and the one of the item claimed for it, and leave too,
// so every item handed out is tested or its group falls back.  Items that
// nobody claims any more are seen by finalize_kernel.
__global__ void __launch_bounds__((G_WARPS + 2) * 32, 1)
gfilter_kernel(GFilterArgs a) {
    extern __shared__ __align__(128) uint4 s_tile[];     // two tiles of G_TILE_WORDS words, two offset tables
    __shared__ GShared sh;
    __shared__ GWarp ws[G_WARPS];
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (threadIdx.x == 0) {
        sh.a = a;
        for (int k = 0; k < 2; ++k) {
            sh.slot[k].group = 0xFFFFFFFEu;
            mbar_init(smem_addr(&sh.slot[k].full), 1u);
            mbar_init(smem_addr(&sh.slot[k].empty), (u32)G_WARPS);
        }
    }
    __syncthreads();
    uint4 *offs = s_tile + 2u * G_TILE_WORDS / 4u;       // G_OFFS 16-byte words each
    if (warp >= (u32)G_WARPS) {
        const u32 k = warp - (u32)G_WARPS;
        GSlot &sl = sh.slot[k];
        for (u32 r = 0;;) {                              // fill r waits until every warp left fill r - 1
            u32 g = 0xFFFFFFFFu;
            GItem it;
            const bool has = gclaim(sh.a, lane, g, it);
            if (r && !mbar_wait_bounded(smem_addr(&sl.empty), (r - 1u) & 1u, CZ_GROUP_EMPTY_TRIES)) {
                gfail(sh.a, sl.G, ST_QUEUE, lane);
                if (has) gfail(sh.a, sh.a.groups[g], ST_QUEUE, lane);
                mbar_wait_bounded(smem_addr(&sl.full), (r - 1u) & 1u);     // let the copies land before leaving
                return;
            }
            if (!has) {
                if (lane == 0) {
                    sl.group = 0xFFFFFFFFu;
                    mbar_arrive(smem_addr(&sl.full));
                }
                return;
            }
            while (!gstage(sh, sl, reinterpret_cast<unsigned short *>(offs + k * G_OFFS),
                           smem_addr(s_tile) + k * G_TILE_WORDS * 4u, g, it, lane))
                if (!gclaim(sh.a, lane, g, it)) {
                    if (lane == 0) {
                        sl.group = 0xFFFFFFFFu;
                        mbar_arrive(smem_addr(&sl.full));
                    }
                    return;
                }
            ++r;
        }
    }
    GWarp &w = ws[warp];
    u32 nscr = 0u;                                       // anchors in the warp's screen queue
    u32 prev = 2u, ended = 0u;                           // slot it holds (2: none), slots without further items
    if (lane == 0) w.ncand = w.words = w.comps = w.err = 0u;
    __syncwarp();
    for (u32 n = 0;; ++n) {
        const u32 k = n & 1u;
        if (ended & (1u << k)) continue;
        if (prev == k) {                                 // the only slot left: it has to be free to be refilled
            gleave(sh, sh.slot[k].G, w, nscr, lane);
            nscr = 0u;
            if (lane == 0) mbar_arrive(smem_addr(&sh.slot[k].empty));
            prev = 2u;
        }
        GSlot &sl = sh.slot[k];
        const bool ok = mbar_wait_bounded(smem_addr(&sl.full), (n >> 1) & 1u, CZ_GROUP_FULL_TRIES);
        const bool end = ok && sl.group == 0xFFFFFFFFu;
        if (end) ended |= 1u << k;
        if (prev < 2u) {
            // the other slot is left once this one's group is known: the queue
            // goes on within a group
            GSlot &pv = sh.slot[prev];
            if (!ok || ended == 3u || (!end && sl.group != pv.group)) {
                gleave(sh, pv.G, w, nscr, lane);
                nscr = 0u;
            }
            if (!ok) gfail(sh.a, pv.G, ST_QUEUE, lane);
            __syncwarp();
            if (!end && lane == 0) mbar_arrive(smem_addr(&pv.empty));
        }
        if (!ok || ended == 3u) return;
        if (end) continue;
        gunits_t(sh, sl, offs + k * G_OFFS, smem_addr(s_tile) + k * G_TILE_WORDS * 4u, w, nscr, lane);
        prev = k;
    }
}

}  // namespace CZ_NS
