// Band indexing by triplet voting on the device: tripletvote.BandIndexer.bandindex
// (tripletvote.py:492-633) with high_fidelity on -- the triplet vote (:1021-1210), the TRIAD
// band assignment over band pairs (:1483-1690), the QUEST band weights and orientation fit
// (:856-1020, rotlib.py:1641-1674) and the vote confidence (:2057-2075) -- plus the indexer's
// band weights and pattern quality (_ebsd_index_single.py:751-763).
//
// One warp indexes one pattern; a block of kWarps warps shares the phase library in shared
// memory.  Arithmetic follows the reference as numpy evaluates it: float32 where the reference
// works on float32 arrays (band angles, votes, the TRIAD fit), float64 for the QUEST fit, every
// add/multiply rounded on its own (no contraction), 3-term dot products as the fused
// multiply-add chain BLAS uses for these shapes, sums in numpy's pairwise order.  arccos is
// CUDA's float32 acosf (within two ulp, as numpy's own float32 arccos is).
//
// Two steps are reorganised for the GPU without changing their result:
//   * the vote's library test |T - a| <= angTol (float64, T a library angle, a a float32 band
//     angle) becomes a <= / >= test against the float32 interval of a that passes it, computed
//     once per library on the host;
//   * a lane tests one band triplet against the library rows that can hold it, 32 triplets at
//     once; the warp lists the matches in triplet and library order, a lane takes one match's
//     weights, and the votes are cast in that order with a lane per band, so that every float32
//     vote sum adds in the reference's order.
//   * the TRIAD candidates of a band pair are tried several at once, a lane per candidate and
//     band, and the first of the best scores is kept, as a scan in order would keep it.
// What bounds the kernel is instructions issued.  FCC library (167 triplets, 50 poles), nine
// bands: 84 band triplets, 85 matches and 14 candidates a pattern cost 63,800 warp instructions
// with a warp per triplet, lane 0 casting the votes and a candidate at a time, and 15.2 ms per
// 200,000 patterns; 19,800 and 5.0 ms now (four blocks an SM; three: 6.0).
#include "ebsd_internal.cuh"

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>

struct ebsd_vote_plan_s {
    int device = 0;
    int nfam = 0, ntrip = 0, npoles = 0;
    double tol = 0.0;
    int early = 0, simpleq = 0;
    uint8_t lut[27] = {};         // lut[:, s0, s1, s2] as 3 x 2 bits, index s0 * 9 + s1 * 3 + s2
    float* d_iv = nullptr;        // [6][ntrip] acceptance intervals lo0, hi0, lo1, hi1, lo2, hi2, rows sorted by lo0
    uint32_t* d_tfam = nullptr;   // [ntrip] f0 | f1 << 8 | f2 << 16
    double* d_tang = nullptr;     // [ntrip][3]
    float* d_pole = nullptr;      // [npoles][4] float32 poles with their family (int bits)
    float* d_triad = nullptr;     // [nfam][npoles][8] TRIAD frame of (family's first pole, pole)
    double* d_pole64 = nullptr;   // [npoles][3]
    double* d_angtab = nullptr;   // [npoles][npoles]
    int32_t* d_famcnt = nullptr;  // [nfam]
    int32_t* d_famidx = nullptr;  // [nfam]
    float* d_cand = nullptr;      // [nfam][npoles][2] band-pair cosine interval per library column
    float* d_par = nullptr;       // [1] largest |cosine| of a band pair that is not parallel
    float par = -1.0f;            // host copy of *d_par
    int32_t* d_orig = nullptr;    // [ntrip] library index of each interval row (rows sorted by lo0)
    void* d_quest = nullptr;      // QUEST hand-over scratch, quest_cap patterns
    int64_t quest_cap = 0;
    float win = 0.0f;             // widest first-angle interval (hi0 - lo0), plus a margin
};

namespace ebsd {
namespace {

constexpr int kWarps = 8;
constexpr int kList = 160;  // matches held at once for casting in triplet and library order
constexpr unsigned kFull = 0xffffffffu;
constexpr double kRadeg = 57.29577951308232;  // 180 / pi
constexpr float kRadegF = 57.29577951308232f;

// What the warp hands to the QUEST solve for one pattern: the bands chosen for the weights
// (bit j: band j) and the number of matched bands; k_quest adds the bands in the fit (mask, m;
// m < 3: no fit) for k_quest_fit.
struct QuestInput {
    uint32_t sel;
    int32_t ngood;
    uint32_t mask;
    int32_t m;
};

struct VoteArgs {
    const float* iv;
    const uint32_t* tfam;
    const double* tang;
    const float* pole;
    const float* triad;
    const double* pole64;
    const double* angtab;
    const int32_t* famcnt;
    const int32_t* famidx;
    const float* cand;
    const int32_t* orig;
    float par, win;
    int nfam, ntrip, npoles, nb;
    float tol_f;
    double tol;
    int early, simpleq;
    uint8_t lut[28];
    const float* norms;
    const float* inten;
    int64_t n;
    ebsd_index_out out;
    QuestInput* quest;  // [n] scratch, device
};

__device__ __forceinline__ float addf(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double addf(double a, double b) { return __dadd_rn(a, b); }

// numpy's pairwise summation (the add reduction of a contiguous float32 / float64 run), over
// get(0 .. n-1): below 8 elements a running sum from 0; up to 128 eight interleaved partial
// sums combined as ((r0 + r1) + (r2 + r3)) + ((r4 + r5) + (r6 + r7)), then the tail; above
// 128 the two halves (split at a multiple of 8) summed the same way.
template <class T, class G>
__device__ T np_sum_block(G get, int lo, int n) {
    if (n < 8) {
        T r = T(0);
        for (int i = 0; i < n; ++i) r = addf(r, get(lo + i));
        return r;
    }
    T r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = get(lo + j);
    int i = 8;
    for (; i < n - (n % 8); i += 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) r[j] = addf(r[j], get(lo + i + j));
    }
    T res = addf(addf(addf(r[0], r[1]), addf(r[2], r[3])), addf(addf(r[4], r[5]), addf(r[6], r[7])));
    for (; i < n; ++i) res = addf(res, get(lo + i));
    return res;
}

template <class T, class G>
__device__ T np_sum_half(G get, int lo, int n) {  // n <= 256
    if (n <= 128) return np_sum_block<T>(get, lo, n);
    int h = n / 2;
    h -= h % 8;
    return addf(np_sum_block<T>(get, lo, h), np_sum_block<T>(get, lo + h, n - h));
}

template <class T, class G>
__device__ T np_sum_get(G get, int n) {  // n <= 512
    if (n <= 256) return np_sum_half<T>(get, 0, n);
    int h = n / 2;
    h -= h % 8;
    return addf(np_sum_half<T>(get, 0, h), np_sum_half<T>(get, h, n - h));
}

template <class T>
__device__ T np_sum(const T* a, int n) {
    return np_sum_get<T>([a](int i) { return a[i]; }, n);
}

// float32 3-term dot product as BLAS sgemm forms it: fma(a2, b2, fma(a1, b1, a0 * b0))
__device__ __forceinline__ float dot3(float a0, float a1, float a2, float b0, float b1, float b2) {
    return __fmaf_rn(a2, b2, __fmaf_rn(a1, b1, __fmul_rn(a0, b0)));
}

// numpy.cross of float32 3-vectors: each component a product difference, each op rounded
__device__ __forceinline__ void cross3(const float* a, const float* b, float* c) {
    c[0] = __fsub_rn(__fmul_rn(a[1], b[2]), __fmul_rn(a[2], b[1]));
    c[1] = __fsub_rn(__fmul_rn(a[2], b[0]), __fmul_rn(a[0], b[2]));
    c[2] = __fsub_rn(__fmul_rn(a[0], b[1]), __fmul_rn(a[1], b[0]));
}

__device__ __forceinline__ float norm3(const float* a) {
    return __fsqrt_rn(dot3(a[0], a[1], a[2], a[0], a[1], a[2]));
}

// float32 arccos(x) * RADEG.  The reference's float32 arccos is numpy's (SIMD, not correctly
// rounded: one or two ulp off for about a third of the inputs on x86); CUDA's acosf is within
// two ulp as well, so either may sit an ulp or two from the reference's value.
__device__ __forceinline__ float acos_deg(float x) {
    return __fmul_rn(acosf(x), kRadegF);
}

// Sorts (v0, v1, v2) with the reference's exchanges; s0, s1, s2: where the sorted values were.
template <class T>
__device__ __forceinline__ void sort3(T& v0, T& v1, T& v2, int& s0, int& s1, int& s2) {
    auto order = [](T& a, T& b, int& i, int& j) {
        const bool x = a > b;
        const T t = a;
        const int k = i;
        a = x ? b : a;
        i = x ? j : i;
        b = x ? t : b;
        j = x ? k : j;
    };
    s0 = 0; s1 = 1; s2 = 2;
    order(v0, v2, s0, s2);
    order(v0, v1, s0, s1);
    order(v1, v2, s1, s2);
}

__device__ __forceinline__ double np_maximum(double a, double b) {  // NaN-propagating
    if (a != a) return a;
    if (b != b) return b;
    return a > b ? a : b;
}

__host__ __device__ inline size_t align8(size_t words) { return (words + 1) & ~size_t(1); }

// 4-byte words of one warp's region
__host__ __device__ inline size_t warp_words(int nb, int nfam) {
    return align8(3 * size_t(nb) + nb + nb * nb + 2 * size_t(nfam) * nb + nb + nb + kList);
}

__host__ __device__ inline size_t block_words(int ntrip, int npoles) {
    return align8(6 * size_t(ntrip) + ntrip + 3 * size_t(npoles) + npoles);
}

// Length of the run of [0, n) on which a monotone predicate holds.
template <class P>
__device__ __forceinline__ int count_leading(int n, P pred) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (pred(mid)) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// ---------------------------------------------------------------------------------------
__device__ void index_pattern(const VoteArgs& A, int64_t p, int lane, const float* s_iv,
                              const int* s_orig, const float4* s_pole, float* w) {
    const int nb = A.nb, nfam = A.nfam, ntrip = A.ntrip, npoles = A.npoles;
    const float tolf = A.tol_f;
    auto pole_family = [s_pole](int P) { return __float_as_int(s_pole[P].w); };
    float2* acc = (float2*)w;            // [nfam][nb] vote weight and count
    float* bn = w + 2 * nfam * nb;       // [nb][3]
    float* inten = bn + 3 * nb;          // [nb]
    float* ang = inten + nb;             // [nb][nb]
    int* rarg = (int*)(ang + nb * nb);   // [nb] band order, ascending rank
    int* bfam = rarg + nb;               // [nb]
    int* mlist = bfam + nb;              // [kList] matches: triplet lane << 16 | library index
    float* fscr = (float*)mlist;         // [32] band fits (after the vote)
    const unsigned lt_mask = (1u << lane) - 1u;

    for (int t = lane; t < 3 * nb; t += 32) bn[t] = A.norms[p * 3 * nb + t];
    for (int t = lane; t < nb; t += 32) inten[t] = A.inten ? A.inten[p * nb + t] : 1.0f;
    for (int t = lane; t < nfam * nb; t += 32) acc[t] = make_float2(0.0f, 0.0f);
    __syncwarp();

    // band-band angles, tripletvote.py:1181-1188 (the vote reads the upper triangle only)
    for (int t = lane; t < nb * (nb - 1) / 2; t += 32) {
        int i = 0, r = t;
        while (r >= nb - 1 - i) {
            r -= nb - 1 - i;
            ++i;
        }
        const int j = i + 1 + r;
        const float* a = bn + 3 * i;
        const float* b = bn + 3 * j;
        float d = fabsf(dot3(a[0], a[1], a[2], b[0], b[1], b[2]));
        d = fminf(fmaxf(d, -1.0f), 1.0f);
        float v = acos_deg(d);
        if (inten[i] < 1e-6f || inten[j] < 1e-6f) v = 10000.0f;
        ang[i * nb + j] = v;
    }
    __syncwarp();

    // ---- triplet vote, tripletvote.py:1023-1135 ----
    // a match's votes, cast by the lanes of its three bands, each into its own column: meta holds
    // the bands i, j, k (5 bits each), the families f0, f1, f2 (4 bits each) and e1, e2, e3
    auto cast = [&](unsigned meta, float w1, float w2, float w3) {
        const bool ri = lane == (int)(meta & 31u), rj = lane == (int)((meta >> 5) & 31u);
        if (!(ri || rj || lane == (int)((meta >> 10) & 31u))) return;
        float2* const a0 = acc + (int)((meta >> 15) & 15u) * nb + lane;
        float2* const a1 = acc + (int)((meta >> 19) & 15u) * nb + lane;
        float2* const a2 = acc + (int)((meta >> 23) & 15u) * nb + lane;
        auto vote = [&](int role) {  // 0: (f0, w1), 1: (f1, w2), 2: (f2, w3)
            float2* const t = role == 0 ? a0 : role == 1 ? a1 : a2;
            float2 v = *t;
            v.x = __fadd_rn(v.x, role == 0 ? w1 : role == 1 ? w2 : w3);
            v.y = __fadd_rn(v.y, 1.0f);
            *t = v;
        };
        vote(ri ? 0 : rj ? 1 : 2);
        const unsigned ee = meta >> 27;
        if (ee & 1u) vote(ri ? 1 : rj ? 0 : 2);
        if (ee & 2u) vote(ri ? 0 : rj ? 2 : 1);
        if (ee & 4u) vote(ri ? 2 : rj ? 1 : 0);
        if (ee == 7u) {
            vote(ri ? 1 : rj ? 2 : 0);
            vote(ri ? 2 : rj ? 0 : 1);
        }
    };
    // the weights and families of library triplet q for a band triplet (angles a0..a2; tri: its
    // bands, the library's family order as 2-bit fields from bit 15, e1..e3 from bit 27)
    auto weigh = [&](int q, float a0, float a1, float a2, unsigned tri, float& w1, float& w2, float& w3) -> unsigned {
        const double* T = A.tang + 3 * (size_t)q;
        const float t0 = __double2float_rn(fabs(__dsub_rn(T[0], (double)a0)));
        const float t1 = __double2float_rn(fabs(__dsub_rn(T[1], (double)a1)));
        const float t2 = __double2float_rn(fabs(__dsub_rn(T[2], (double)a2)));
        const uint32_t fw = A.tfam[q];
        w1 = __fsub_rn(tolf, __fmul_rn(0.5f, __fadd_rn(t0, t1)));
        w2 = __fsub_rn(tolf, __fmul_rn(0.5f, __fadd_rn(t0, t2)));
        w3 = __fsub_rn(tolf, __fmul_rn(0.5f, __fadd_rn(t1, t2)));
        const unsigned f0 = (fw >> (8 * ((tri >> 15) & 3u))) & 15u, f1 = (fw >> (8 * ((tri >> 17) & 3u))) & 15u;
        const unsigned f2 = (fw >> (8 * ((tri >> 19) & 3u))) & 15u;
        return (tri & 0x38007fffu) | f0 << 15 | f1 << 19 | f2 << 23;
    };
    const int nt3 = nb * (nb - 1) * (nb - 2) / 6;
    for (int t0 = 0; t0 < nt3; t0 += 32) {
        // this lane's band triplet i < j < k, in the order of the nested loops over them
        int i = 0, j, k;
        {
            int r = t0 + lane < nt3 ? t0 + lane : 0, c = (nb - 1) * (nb - 2) / 2;
            while (r >= c) {
                r -= c;
                ++i;
                c -= nb - 1 - i;
            }
            j = i + 1;
            c = nb - 1 - j;
            while (r >= c) {
                r -= c;
                ++j;
                --c;
            }
            k = j + 1 + r;
        }
        // (a band without intensity has angles 10000: no library triplet matches)
        const bool on = t0 + lane < nt3 && !(inten[i] < 1e-6f) && !(inten[j] < 1e-6f) && !(inten[k] < 1e-6f);
        float a0 = ang[i * nb + j], a1 = ang[i * nb + k], a2 = ang[j * nb + k];
        int s0, s1, s2, u0, u1, u2;
        sort3(a0, a1, a2, s0, s1, s2);
        const int code = A.lut[s0 * 9 + s1 * 3 + s2];
        int r0 = code & 3, r1 = (code >> 2) & 3, r2 = (code >> 4) & 3;
        sort3(r0, r1, r2, u0, u1, u2);
        unsigned tri = (unsigned)(i | j << 5 | k << 10 | u0 << 15 | u1 << 17 | u2 << 19);
        tri |= (fabsf(__fsub_rn(a0, a1)) < tolf ? 1u << 27 : 0u) | (fabsf(__fsub_rn(a1, a2)) < tolf ? 2u << 27 : 0u) |
               (fabsf(__fsub_rn(a2, a0)) < tolf ? 4u << 27 : 0u);
        // library rows whose first-angle interval can hold a0: sorted by its lower end, so
        // [s, e) with lo0 in [a0 - win, a0]
        const float tgt = a0 - A.win;
        const int e = on ? count_leading(ntrip, [&](int q) { return s_iv[q] <= a0; }) : 0;
        const int s = count_leading(e, [&](int q) { return s_iv[q] < tgt; });
        auto test = [&](const float* r, float b0, float b1, float b2) {
            return (b1 >= r[2 * ntrip]) & (b1 <= r[3 * ntrip]) & (b0 >= r[0]) & (b0 <= r[ntrip]) & (b2 >= r[4 * ntrip]) &
                   (b2 <= r[5 * ntrip]);
        };
        int cnt = 0;
        unsigned long long hits = 0;  // of the first 64 rows
#pragma unroll 2
        for (int q = s; q < e; ++q)
            if (test(s_iv + q, a0, a1, a2)) {
                if (q - s < 64) hits |= 1ull << (q - s);
                ++cnt;
            }
        int off = cnt;  // matches of the lanes before
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, off, o);
            if (lane >= o) off += v;
        }
        const int total = __shfl_sync(kFull, off, 31);
        off -= cnt;
        int last = -1;
        for (int base = 0; base < total;) {
            // the lanes whose matches fit in the list from `base` on
            const bool in = cnt > 0 && off >= base && off + cnt <= base + kList;
            const unsigned inm = __ballot_sync(kFull, in);
            int n;
            if (inm == 0) {
                // one band triplet with more matches than the list holds: 32 at a time, each the
                // smallest library index above the last one
                const int l = __ffs(__ballot_sync(kFull, cnt > 0 && off == base)) - 1;
                const float b0 = __shfl_sync(kFull, a0, l), b1 = __shfl_sync(kFull, a1, l), b2 = __shfl_sync(kFull, a2, l);
                const int bs = __shfl_sync(kFull, s, l), be = __shfl_sync(kFull, e, l);
                for (n = 0; n < 32; ++n) {
                    int mine = INT_MAX;
                    for (int q = bs + lane; q < be; q += 32)
                        if (test(s_iv + q, b0, b1, b2) && s_orig[q] > last && s_orig[q] < mine) mine = s_orig[q];
                    last = __reduce_min_sync(kFull, mine);
                    if (last == INT_MAX) break;
                    if (lane == 0) mlist[n] = l << 16 | last;
                }
                if (last == INT_MAX) {
                    base += __shfl_sync(kFull, cnt, l);
                    last = -1;
                }
            } else {
                n = __shfl_sync(kFull, off + cnt, 31 - __clz(inm)) - base;
            }
            if (in) {  // into the lane's part of the list, sorted into library order
                int* seg = mlist + (off - base);
                int have = 0;
                auto put = [&](int q) {
                    const int v = lane << 16 | s_orig[q];
                    int b = have - 1;
                    while (b >= 0 && seg[b] > v) {
                        seg[b + 1] = seg[b];
                        --b;
                    }
                    seg[b + 1] = v;
                    ++have;
                };
                for (unsigned long long m = hits; m; m &= m - 1) put(s + __ffsll((long long)m) - 1);
                for (int q = s + 64; q < e && have < cnt; ++q)
                    if (test(s_iv + q, a0, a1, a2)) put(q);
            }
            if (inm != 0) base += n;
            __syncwarp();
            for (int m0 = 0; m0 < n; m0 += 32) {
                const int v = m0 + lane < n ? mlist[m0 + lane] : 0, l = v >> 16;
                const float b0 = __shfl_sync(kFull, a0, l), b1 = __shfl_sync(kFull, a1, l), b2 = __shfl_sync(kFull, a2, l);
                const unsigned btri = __shfl_sync(kFull, tri, l);
                float w1, w2, w3;
                const unsigned meta = weigh(v & 0xffff, b0, b1, b2, btri, w1, w2, w3);
                const int nm = n - m0 < 32 ? n - m0 : 32;
                for (int m = 0; m < nm; ++m)
                    cast(__shfl_sync(kFull, meta, m), __shfl_sync(kFull, w1, m), __shfl_sync(kFull, w2, m),
                         __shfl_sync(kFull, w3, m));
            }
            __syncwarp();
        }
    }
    __syncwarp();

    // ---- vote metrics per band, tripletvote.py:1137-1171, and rank, :1189-1191 ----
    float rank = 0.0f;
    int fam = 0;
    if (lane < nb) {
        float sum = 0.0f, mx = -1.0e12f, m1 = -INFINITY, m2 = -INFINITY;
        for (int f = 0; f < nfam; ++f) {
            const float v = acc[f * nb + lane].x;
            sum = __fadd_rn(sum, v);
            if (v > mx) { mx = v; fam = f; }
            if (v > m1) { m2 = m1; m1 = v; } else if (v > m2) { m2 = v; }
        }
        const int mxvote = (int)mx, tvotes = (int)sum;
        const float cm = tvotes < 1 ? 0.0f
                                    : __double2float_rn(__ddiv_rn((double)__fsub_rn(m1, m2), (double)tvotes));
        const double lead = __ddiv_rn((double)(nb - lane), (double)nb);
        rank = __double2float_rn(__dmul_rn(__dmul_rn(lead, (double)cm), (double)mxvote));
        bfam[lane] = fam;
    }
    {
        int pos = 0;
        for (int c = 0; c < nb; ++c) {
            const float rc = __shfl_sync(kFull, rank, c);
            pos += (rc < rank) || (rc == rank && c < lane);
        }
        if (lane < nb) rarg[pos] = lane;
    }
    __syncwarp();

    // ---- TRIAD assignment over band pairs in rank order, tripletvote.py:1600-1690 ----
    // groups of nb lanes try a candidate each, lane tj of a group with band tj
    const int ngrp = 32 / nb, grp = lane / nb, tj = lane - grp * nb;
    const unsigned grp_mask = nb == 32 ? kFull : (1u << nb) - 1u;
    int best_n = 0;
    float best_fit = 360.0f;
    int bij[4] = {-1, -1, -1, -1};
    int best_pm = -1000, best_pv = 0;
    bool stop = false;
    for (int ii = 0; ii < nb - 1 && !stop; ++ii) {
        for (int jj = ii + 1; jj < nb; ++jj) {
            const int b1 = rarg[nb - 1 - ii], b2 = rarg[nb - 1 - jj];
            const float* v1 = bn + 3 * b1;
            const float* v2 = bn + 3 * b2;
            const int f1 = bfam[b1], f2 = bfam[b2];
            float c12 = dot3(v1[0], v1[1], v1[2], v2[0], v2[1], v2[2]);
            if (c12 > 1.0f) c12 = 1.0f;
            if (c12 < -1.0f) c12 = -1.0f;
            int ngood = 0;
            float afit = 0.0f;
            int pm = -1, pv = 0;
            // arccos(|c12|) > angTol and |angTable - arccos(c12)| < angTol (tripletvote.py:1517-1524) as
            // cosine intervals precomputed with the same arccos (k_vote_thresholds)
            if (fabsf(c12) <= A.par) {
                const float* cint = A.cand + (size_t)f1 * npoles * 2;
                const int row = A.famidx[f1], lo = A.famidx[f2], cnt = A.famcnt[f2];
                float x[3];
                cross3(v1, v2, x);
                const float nx = norm3(x);
                x[0] = __fdiv_rn(x[0], nx); x[1] = __fdiv_rn(x[1], nx); x[2] = __fdiv_rn(x[2], nx);
                float y[3];
                cross3(v1, x, y);
                const float B[3][3] = {{v1[0], v1[1], v1[2]}, {x[0], x[1], x[2]}, {y[0], y[1], y[2]}};
                const float4 p1 = s_pole[row];
                const float* bj = bn + 3 * tj;
                const float bj0 = bj[0], bj1 = bj[1], bj2 = bj[2];
                float score = -1.0f;
                bool any = false;
                for (int cb = 0; cb < cnt; cb += 32) {
                    const int col = lo + cb + lane;
                    const bool hit = cb + lane < cnt && c12 >= cint[2 * col] && c12 <= cint[2 * col + 1];
                    unsigned m = __ballot_sync(kFull, hit);
                    any = any || m != 0;
                    while (m) {
                        // the next ngrp candidates, one a group (a group past the last takes the first)
                        int cand = lo + cb + __ffs(m) - 1, ntry = 0;
                        for (; ntry < ngrp && m; ++ntry, m &= m - 1)
                            if (ntry == grp) cand = lo + cb + __ffs(m) - 1;
                        // the frame of (p1, candidate): p1, their unit cross product, the cross of the two
                        const float4* fr = (const float4*)(A.triad + ((size_t)f1 * npoles + cand) * 8);
                        const float4 fa = __ldg(fr), fb = __ldg(fr + 1);
                        const float Am[3][3] = {{p1.x, fa.x, fa.w}, {p1.y, fa.y, fb.x}, {p1.z, fa.z, fb.y}};
                        float t[3];
#pragma unroll
                        for (int r = 0; r < 3; ++r) {
                            float AB[3];
#pragma unroll
                            for (int c = 0; c < 3; ++c)
                                AB[c] = dot3(Am[r][0], Am[r][1], Am[r][2], B[0][c], B[1][c], B[2][c]);
                            t[r] = dot3(AB[0], AB[1], AB[2], bj0, bj1, bj2);
                        }
                        // this lane's band: rotated normal, best library pole
                        float best = -INFINITY;
                        int arg = 0;
#pragma unroll 4
                        for (int P = 0; P < npoles; ++P) {
                            const float4 po = s_pole[P];
                            const float v = dot3(po.x, po.y, po.z, t[0], t[1], t[2]);
                            if (v > best) { best = v; arg = P; }
                        }
                        best = best < -1.0f ? -1.0f : best;
                        best = best > 1.0f ? 1.0f : best;
                        const float ftry = acos_deg(best);
                        const bool ok = grp < ntry && ftry < tolf;
                        const unsigned okm = (__ballot_sync(kFull, ok) >> (grp * nb < 32 ? grp * nb : 0)) & grp_mask;
                        const int nmatch = __popc(okm);
                        if (ok) fscr[grp * nb + __popc(okm & ((1u << tj) - 1u))] = ftry;
                        __syncwarp();
                        float stry = 0.0f;
                        if (grp < ntry && tj == 0) {
                            const float mean = __fdiv_rn(np_sum(fscr + lane, nmatch), (float)nmatch);
                            stry = __fdiv_rn((float)nmatch, __fadd_rn(mean, 1e-6f));
                        }
                        int sel = -1;
                        for (int g = 0; g < ntry; ++g) {
                            const float sg = __shfl_sync(kFull, stry, g * nb);
                            if (sg > score) {
                                score = sg;
                                sel = g;
                            }
                        }
                        if (sel >= 0) {
                            const int src = (sel * nb + lane) & 31;  // lanes from nb on hold no band
                            afit = __shfl_sync(kFull, ftry, src);
                            pm = __shfl_sync(kFull, arg, src);
                            pv = afit < tolf;
                        }
                        __syncwarp();
                    }
                }
                if (any) ngood = __popc(__ballot_sync(kFull, lane < nb && afit < tolf));
            }
            if (ngood >= 3) {
                float fit = 0.0f;
                for (int j = 0; j < nb; ++j) {
                    const float v = __shfl_sync(kFull, afit, j);
                    if (v < tolf) fit = __fadd_rn(fit, v);
                }
                fit = __fdiv_rn(fit, (float)ngood);
                if (best_n < ngood || (best_n == ngood && best_fit > fit)) {
                    best_fit = fit;
                    best_n = ngood;
                    best_pm = pm;
                    best_pv = pv;
                    bij[0] = ii; bij[1] = jj; bij[2] = b1; bij[3] = b2;
                }
            }
            if (best_n >= A.early) {
                stop = true;
                break;
            }
        }
    }

    // ---- QUEST weights, tripletvote.py:856-901: the band selection here (its scores need the
    // votes); the float64 weights, B and z and the solve in k_quest, one thread per pattern ----
    const bool good = lane < nb && best_pv != 0;
    const unsigned goodm = __ballot_sync(kFull, good);
    const int ngood = __popc(goodm);
    unsigned selm = 0;
    if (ngood >= 3) {
        float sc = -1.0f;
        if (!A.simpleq) {
            if (good) {
                const int a = pole_family(best_pm);
                const float2 v = acc[a * nb + lane];
                sc = __fdiv_rn(v.x, v.y > 0.0f ? v.y : 1.0e-12f);
            }
        } else if (good) {
            sc = inten[__popc(goodm & lt_mask)];
        }
        int pos = 0;
        for (int c = 0; c < nb; ++c) {
            const float s = __shfl_sync(kFull, sc, c);
            pos += (s < sc) || (s == sc && c < lane);
        }
        const int nfit = ngood < 6 ? ngood : 6;
        selm = __ballot_sync(kFull, lane < nb && (nb - 1 - pos) < nfit);
    }
    if (lane == 0) {
        QuestInput* qi = A.quest + p;
        qi->sel = selm;
        qi->ngood = ngood;
    }

    // ---- vote confidence of the matched bands, tripletvote.py:2057-2075 ----
    float cm2 = -1.0f;
    if (ngood >= 3) {
        float num = 0.0f;
        for (int j = 0; j < nb; ++j) {
            const int pmj = __shfl_sync(kFull, best_pm, j);
            if ((goodm >> j) & 1u) num = __fadd_rn(num, acc[pole_family(pmj) * nb + j].x);
        }
        float den = 0.0f;
        if (lane == 0)  // accumulator.clip(1) summed over all families and bands
            den = np_sum_get<float>([acc](int t) { const float v = acc[t].x; return (v != v || v >= 1.0f) ? v : 1.0f; },
                                    nfam * nb);
        den = __shfl_sync(kFull, den, 0);
        cm2 = __fdiv_rn(num, den);
    }

    // ---- outputs ----
    const ebsd_index_out& o = A.out;
    const int accc = __popc(__ballot_sync(kFull, good && pole_family(best_pm > 0 ? best_pm : 0) == fam));
    if (lane < nb) {
        const int64_t e = p * nb + lane;
        o.polematch[e] = best_pm;
        if (o.bandfam) o.bandfam[e] = fam;
        if (o.bandrank) o.bandrank[e] = rank;
        if (o.polevalid) o.polevalid[e] = (uint8_t)best_pv;
    }
    if (o.accw)
        for (int t = lane; t < nfam * nb; t += 32) o.accw[p * nfam * nb + t] = acc[t].x;
    if (o.accn)
        for (int t = lane; t < nfam * nb; t += 32) o.accn[p * nfam * nb + t] = acc[t].y;
    if (lane == 0) {
        o.cm[p] = cm2;
        o.nmatch[p] = best_n;
        for (int t = 0; t < 4; ++t) o.ij[4 * p + t] = bij[t];
        o.acc_correct[p] = accc;
    }
    __syncwarp();
}

// Plan-time thresholds of the TRIAD step, evaluated with the kernel's own arccos so that the
// float comparisons replace the reference's tests exactly (acos_deg is monotone in x):
//   par: the largest y in [0, 1] with acos_deg(y) > angTol, so that the pair test
//        arccos(|c|) * RADEG > angTol (tripletvote.py:1517) is |c| <= par;
//   cand[f][c] = [lo, hi]: the cosines x in [-1, 1] with |angTable[famIndex[f]][c] - acos_deg(x)|
//        < angTol in float64 (tripletvote.py:1521-1522); empty as [+inf, -inf];
//   triad[f][c]: what the TRIAD solution of a candidate c needs of the library alone.
__device__ __forceinline__ int64_t okey(float f) {
    const uint32_t u = __float_as_uint(f);
    return (int64_t)((u & 0x80000000u) ? ~u : (u | 0x80000000u));
}
__device__ __forceinline__ float okey_float(int64_t k) {
    const uint32_t v = (uint32_t)k;
    return __uint_as_float((v & 0x80000000u) ? (v & 0x7fffffffu) : ~v);
}

__global__ void k_vote_thresholds(const double* __restrict__ angtab, const int32_t* __restrict__ famidx,
                                  const float4* __restrict__ pole, int nfam, int npoles, double tol, float tolf,
                                  float* __restrict__ cand, float* __restrict__ par, float* __restrict__ triad) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) {
        int64_t a = okey(0.0f), b = okey(1.0f);
        if (!(acos_deg(0.0f) > tolf)) {
            *par = -1.0f;
        } else {
            while (a < b) {  // last key with the test true
                const int64_t mid = a + (b - a + 1) / 2;
                if (acos_deg(okey_float(mid)) > tolf) a = mid; else b = mid - 1;
            }
            *par = okey_float(a);
        }
    }
    if (t >= nfam * npoles) return;
    const int f = t / npoles, c = t - f * npoles;
    {  // the frame of the family's first pole and pole c: their unit cross product, its cross with the first
        const float4 a = pole[famidx[f]], b = pole[c];
        const float p1[3] = {a.x, a.y, a.z};
        float p2[3] = {b.x, b.y, b.z};
        const float n2 = __fadd_rn(norm3(p2), 1.0e-35f);
        p2[0] = __fdiv_rn(p2[0], n2); p2[1] = __fdiv_rn(p2[1], n2); p2[2] = __fdiv_rn(p2[2], n2);
        float pc[3];
        cross3(p1, p2, pc);
        const float npc = __fadd_rn(norm3(pc), 1.0e-35f);
        pc[0] = __fdiv_rn(pc[0], npc); pc[1] = __fdiv_rn(pc[1], npc); pc[2] = __fdiv_rn(pc[2], npc);
        float a2[3];
        cross3(p1, pc, a2);
        float* fr = triad + (size_t)t * 8;
        for (int i = 0; i < 3; ++i) {
            fr[i] = pc[i];
            fr[3 + i] = a2[i];
        }
        fr[6] = fr[7] = 0.0f;
    }
    const double T = angtab[(size_t)famidx[f] * npoles + c];
    const int64_t k0 = okey(-1.0f), k1 = okey(1.0f);
    // d(x) = T - acos_deg(x) does not decrease with x; the test is -tol < d < tol
    int64_t a = k0, b = k1 + 1;
    while (a < b) {  // first key with d > -tol (k1 + 1: none)
        const int64_t mid = a + (b - a) / 2;
        if (__dsub_rn(T, (double)acos_deg(okey_float(mid))) > -tol) b = mid; else a = mid + 1;
    }
    const int64_t lo = a;
    a = k0 - 1;
    b = k1;
    while (a < b) {  // last key with d < tol (k0 - 1: none)
        const int64_t mid = a + (b - a + 1) / 2;
        if (__dsub_rn(T, (double)acos_deg(okey_float(mid))) < tol) a = mid; else b = mid - 1;
    }
    const int64_t hi = a;
    if (lo > k1 || hi < k0 || lo > hi) {
        cand[2 * t] = INFINITY;
        cand[2 * t + 1] = -INFINITY;
    } else {
        cand[2 * t] = okey_float(lo);
        cand[2 * t + 1] = okey_float(hi);
    }
}


// ---- the scalar QUEST solve (tripletvote.py:955-993), one thread per pattern so that every
// float64 instruction carries a full warp of patterns ----
__global__ void k_quest(QuestInput* __restrict__ qin, int64_t n, int nb, const float* __restrict__ norms,
                        const float* __restrict__ inten, const int64_t* __restrict__ polematch,
                        const double* __restrict__ pole64, double* __restrict__ quat) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        QuestInput& qi = qin[p];
        double qout[4] = {1.0, 0.0, 0.0, 0.0};
        // band weights (tripletvote.py:885-899): the chosen bands' intensities normalised to
        // sum one, stored as float32
        float wsel[32];
        double wq[32];
        for (int j = 0; j < nb; ++j) {
            const float it = inten ? inten[p * nb + j] : 1.0f;
            wq[j] = (qi.ngood >= 3 && ((qi.sel >> j) & 1u)) ? (double)it : 0.0;
        }
        double tot = np_sum(wq, nb);
        for (int j = 0; j < nb; ++j) wsel[j] = qi.ngood >= 3 ? __double2float_rn(__ddiv_rn(wq[j], tot)) : 0.0f;
        // the fit's weights (tripletvote.py:912-914, 940-947)
        for (int j = 0; j < nb; ++j) wq[j] = (double)wsel[j];
        tot = np_maximum(np_sum(wq, nb), 1e-12);
        double wn[32];
        int idx[32];
        int m = 0;
        uint32_t mask = 0;
        for (int j = 0; j < nb; ++j) {
            const double w = __ddiv_rn((double)wsel[j], tot);
            if (w > 1.0e-7) {
                wn[m] = w;
                idx[m] = j;
                mask |= 1u << j;
                ++m;
            }
        }
        qi.mask = m >= 3 ? mask : 0u;
        qi.m = m >= 3 ? m : 0;
        if (m >= 3) {
            const double ws = np_sum(wn, m);
            for (int k = 0; k < m; ++k) wn[k] = __ddiv_rn(wn[k], ws);
            auto bcomp = [&](int k, int c) { return (double)norms[(p * nb + idx[k]) * 3 + c]; };
            auto pcomp = [&](int k, int c) {
                const int64_t pm = polematch[p * nb + idx[k]];
                return pole64[3 * (pm > 0 ? pm : 0) + c];
            };
            // B = (w b)^T p and z = sum_k w_k (b_k x p_k), in the reference's operation order
            double Bm[3][3];
            for (int r = 0; r < 3; ++r)
                for (int c = 0; c < 3; ++c) {
                    double acc = __dmul_rn(__dmul_rn(wn[0], bcomp(0, r)), pcomp(0, c));
                    for (int k = 1; k < m; ++k) acc = __fma_rn(__dmul_rn(wn[k], bcomp(k, r)), pcomp(k, c), acc);
                    Bm[r][c] = acc;
                }
            double z[3];
            for (int c = 0; c < 3; ++c) {
                const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
                double zc = 0.0;
                for (int k = 0; k < m; ++k) {
                    const double cr = __dsub_rn(__dmul_rn(bcomp(k, c1), pcomp(k, c2)), __dmul_rn(bcomp(k, c2), pcomp(k, c1)));
                    const double v = __dmul_rn(wn[k], cr);
                    zc = k == 0 ? v : __dadd_rn(zc, v);
                }
                z[c] = zc;
            }
            double S[3][3];
            for (int r = 0; r < 3; ++r)
                for (int c = 0; c < 3; ++c) S[r][c] = __dadd_rn(Bm[r][c], Bm[c][r]);
            double S2[3][3];
            for (int r = 0; r < 3; ++r)
                for (int c = 0; c < 3; ++c)
                    S2[r][c] = __fma_rn(S[r][2], S[2][c], __fma_rn(S[r][1], S[1][c], __dmul_rn(S[r][0], S[0][c])));
            const double det =
                __dadd_rn(__dsub_rn(__dmul_rn(S[0][0], __dsub_rn(__dmul_rn(S[1][1], S[2][2]), __dmul_rn(S[1][2], S[2][1]))),
                                    __dmul_rn(S[0][1], __dsub_rn(__dmul_rn(S[1][0], S[2][2]), __dmul_rn(S[1][2], S[2][0])))),
                          __dmul_rn(S[0][2], __dsub_rn(__dmul_rn(S[1][0], S[2][1]), __dmul_rn(S[1][1], S[2][0]))));
            const double kk = __dadd_rn(__dadd_rn(__dsub_rn(__dmul_rn(S[1][1], S[2][2]), __dmul_rn(S[1][2], S[2][1])),
                                                  __dsub_rn(__dmul_rn(S[0][0], S[2][2]), __dmul_rn(S[0][2], S[2][0]))),
                                        __dsub_rn(__dmul_rn(S[0][0], S[1][1]), __dmul_rn(S[1][0], S[0][1])));
            const double sig = __dmul_rn(0.5, __dadd_rn(__dadd_rn(S[0][0], S[1][1]), S[2][2]));
            const double sig2 = __dmul_rn(sig, sig);
            double u[3], v[3];
            for (int c = 0; c < 3; ++c) {
                u[c] = __fma_rn(z[2], S2[2][c], __fma_rn(z[1], S2[1][c], __dmul_rn(z[0], S2[0][c])));
                v[c] = __fma_rn(z[2], S[2][c], __fma_rn(z[1], S[1][c], __dmul_rn(z[0], S[0][c])));
            }
            const double d = __fma_rn(u[2], z[2], __fma_rn(u[1], z[1], __dmul_rn(u[0], z[0])));
            const double c = __dadd_rn(det, __fma_rn(v[2], z[2], __fma_rn(v[1], z[1], __dmul_rn(v[0], z[0]))));
            const double b = __dadd_rn(sig2, __fma_rn(z[2], z[2], __fma_rn(z[1], z[1], __dmul_rn(z[0], z[0]))));
            const double a = __dsub_rn(sig2, kk);
            const double apb = __dadd_rn(a, b);
            const double cst = __dsub_rn(__dadd_rn(__dmul_rn(a, b), __dmul_rn(c, sig)), d);
            double lam = 1.0, dlam = 1e6;
            for (int it = 0; dlam > 1.0e-12 && it < 10; ++it) {
                const double lam0 = lam;
                const double l2 = __dmul_rn(lam, lam);
                const double num = __dadd_rn(__dsub_rn(__dsub_rn(__dmul_rn(l2, l2), __dmul_rn(apb, l2)), __dmul_rn(c, lam)), cst);
                const double den = __dsub_rn(__dsub_rn(__dmul_rn(4.0, __dmul_rn(l2, lam)), __dmul_rn(__dmul_rn(2.0, apb), lam)), c);
                lam = __dsub_rn(lam, __ddiv_rn(num, den));
                dlam = fabs(__dsub_rn(lam0, lam));
            }
            const double beta = __dsub_rn(lam, sig);
            const double alpha = __dadd_rn(__dsub_rn(__dmul_rn(lam, lam), sig2), kk);
            const double gamma = __dsub_rn(__dmul_rn(__dadd_rn(lam, sig), alpha), det);
            double X[3];
            for (int r = 0; r < 3; ++r) {
                double M[3];
                for (int cc = 0; cc < 3; ++cc)
                    M[cc] = __dadd_rn(__dadd_rn(r == cc ? alpha : 0.0, __dmul_rn(beta, S[r][cc])), S2[r][cc]);
                X[r] = __fma_rn(M[2], z[2], __fma_rn(M[1], z[1], __dmul_rn(M[0], z[0])));
            }
            const double qn = __dsqrt_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(gamma, gamma), __dmul_rn(X[0], X[0])),
                                                             __dmul_rn(X[1], X[1])), __dmul_rn(X[2], X[2])));
            qout[0] = __ddiv_rn(gamma, qn);
            qout[1] = __ddiv_rn(X[0], qn);
            qout[2] = __ddiv_rn(X[1], qn);
            qout[3] = __ddiv_rn(X[2], qn);
            if (gamma < 0.0)
                for (int t = 0; t < 4; ++t) qout[t] = -qout[t];
        }
        for (int t = 0; t < 4; ++t) quat[4 * p + t] = qout[t];
    }
}

// ---- per-band and mean fit (tripletvote.py:994-1018, rotlib.quat_vectorL1N with p = 1, and
// the arccos of bandindex, :601-604), one thread per pattern ----
__global__ void k_quest_fit(const QuestInput* __restrict__ qin, const float* __restrict__ norms,
                            const int64_t* __restrict__ polematch, const double* __restrict__ pole64,
                            const double* __restrict__ quat, int64_t n, int nb, double* __restrict__ fit,
                            double* __restrict__ bandfit) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const QuestInput& qi = qin[p];
        const int m = qi.m >= 3 ? qi.m : 0;
        const double w0 = quat[4 * p], r0 = quat[4 * p + 1], r1 = quat[4 * p + 2], r2 = quat[4 * p + 3];
        double dots[32];
        int k = 0;
        for (int j = 0; j < nb; ++j) {
            double bd = -1.0;
            if (m > 0 && ((qi.mask >> j) & 1u)) {
                const float* f = norms + (p * nb + j) * 3;
                const double vv[3] = {(double)f[0], (double)f[1], (double)f[2]};
                const int64_t pm = polematch[p * nb + j];
                const double* pp = pole64 + 3 * (pm > 0 ? pm : 0);
                double t[3] = {__dsub_rn(__dmul_rn(r1, vv[2]), __dmul_rn(r2, vv[1])),
                               __dsub_rn(__dmul_rn(r2, vv[0]), __dmul_rn(r0, vv[2])),
                               __dsub_rn(__dmul_rn(r0, vv[1]), __dmul_rn(r1, vv[0]))};
                for (int cc = 0; cc < 3; ++cc) t[cc] = __dadd_rn(t[cc], __dmul_rn(w0, vv[cc]));
                const double t2[3] = {__dsub_rn(__dmul_rn(r1, t[2]), __dmul_rn(r2, t[1])),
                                      __dsub_rn(__dmul_rn(r2, t[0]), __dmul_rn(r0, t[2])),
                                      __dsub_rn(__dmul_rn(r0, t[1]), __dmul_rn(r1, t[0]))};
                double sd = 0.0;
                for (int cc = 0; cc < 3; ++cc)
                    sd = __dadd_rn(sd, __dmul_rn(__dadd_rn(__dmul_rn(2.0, t2[cc]), vv[cc]), pp[cc]));
                bd = sd;
                dots[k++] = sd;
            }
            const double bc = bd < -1.0 ? -1.0 : (bd > 1.0 ? 1.0 : bd);
            bandfit[p * nb + j] = __dmul_rn(acos(bc), kRadeg);
        }
        double mad = -1.0;
        if (m > 0) mad = __ddiv_rn(np_sum(dots, m), (double)m);
        const double mc = mad < -1.0 ? -1.0 : (mad > 1.0 ? 1.0 : mad);
        fit[p] = __dmul_rn(acos(mc), kRadeg);
    }
}

__global__ void __launch_bounds__(kWarps * 32, 4) k_band_index(VoteArgs A) {
    extern __shared__ __align__(16) float vsm[];
    float4* s_pole = (float4*)vsm;
    float* s_iv = vsm + 4 * A.npoles;
    int* s_orig = (int*)(s_iv + 6 * A.ntrip);
    for (int t = threadIdx.x; t < 6 * A.ntrip; t += blockDim.x) s_iv[t] = A.iv[t];
    for (int t = threadIdx.x; t < A.ntrip; t += blockDim.x) s_orig[t] = A.orig[t];
    for (int t = threadIdx.x; t < A.npoles; t += blockDim.x) s_pole[t] = ((const float4*)A.pole)[t];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* w = vsm + block_words(A.ntrip, A.npoles) + warp * warp_words(A.nb, A.nfam);
    const int64_t stride = (int64_t)gridDim.x * kWarps;
    for (int64_t p = (int64_t)blockIdx.x * kWarps + warp; p < A.n; p += stride)
        index_pattern(A, p, lane, s_iv, s_orig, s_pole, w);
}

// ---- band weights and pattern quality, _ebsd_index_single.py:751-763 ----
__global__ void k_band_intensity(const float* __restrict__ mx, const float* __restrict__ nmx,
                                 const float* __restrict__ theta, const float* __restrict__ rho,
                                 const int8_t* __restrict__ valid, int64_t n, int nb, float rhomax,
                                 float* __restrict__ adj, float* __restrict__ pq, float* __restrict__ iq) {
    const float lo = (float)(2.0 * 3.141592653589793 / 180.0);
    const float hi = (float)(178.0 * 3.141592653589793 / 180.0);
    float a[128];
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        for (int b = 0; b < nb; ++b) {
            const int64_t e = p * nb + b;
            const float v = (float)valid[e];
            float t = __fmul_rn(__fmul_rn(-1.0f, fabsf(rho[e])), 0.5f);
            t = __fmul_rn(__fadd_rn(__fdiv_rn(t, rhomax), 1.0f), mx[e]);
            t = __fmul_rn(t, __fdiv_rn(__fadd_rn(theta[e] > lo ? 1.0f : 0.0f, 0.5f), 2.0f));
            t = __fmul_rn(t, __fdiv_rn(__fadd_rn(theta[e] < hi ? 1.0f : 0.0f, 0.5f), 2.0f));
            adj[e] = __fmul_rn(t, v);
        }
        if (pq) {
            for (int b = 0; b < nb; ++b) a[b] = __fmul_rn(mx[p * nb + b], (float)valid[p * nb + b]);
            pq[p] = __fdiv_rn(np_sum(a, nb), (float)nb);
        }
        if (iq) {
            for (int b = 0; b < nb; ++b) a[b] = __fmul_rn(nmx[p * nb + b], (float)valid[p * nb + b]);
            iq[p] = __fdiv_rn(np_sum(a, nb), (float)nb);
        }
    }
}

// ---- host: float32 acceptance interval of |T - a| <= tol (evaluated in float64) ----
inline uint32_t fkey(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
inline float funkey(uint32_t k) {
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
inline bool within(double T, float a, double tol) { return std::fabs(T - (double)a) <= tol; }

void accept_interval(double T, double tol, float* lo, float* hi) {
    const float fT = (float)T;
    if (!(tol >= 0.0) || !std::isfinite(T) || !within(T, fT, tol)) {
        *lo = INFINITY;
        *hi = -INFINITY;
        return;
    }
    const uint32_t kT = fkey(fT);
    uint32_t a = fkey(-FLT_MAX), b = kT;  // smallest key in [a, b] that passes
    while (a < b) {
        const uint32_t mid = a + (b - a) / 2;
        if (within(T, funkey(mid), tol)) b = mid; else a = mid + 1;
    }
    *lo = funkey(a);
    a = kT;
    b = fkey(FLT_MAX);  // largest key in [a, b] that passes
    while (a < b) {
        const uint32_t mid = a + (b - a + 1) / 2;
        if (within(T, funkey(mid), tol)) a = mid; else b = mid - 1;
    }
    *hi = funkey(a);
}

}  // namespace
}  // namespace ebsd

using namespace ebsd;

extern "C" int ebsd_vote_plan_create(const ebsd_triplib_desc* d, int device, ebsd_vote_plan_t* out) {
    if (!d || !out) return EBSD_E_ARG;
    *out = nullptr;
    if (d->nfam < 2 || d->nfam > 16 || d->ntrip < 1 || d->ntrip > 8192 || d->npoles < 1 || d->npoles > 512)
        return EBSD_E_ARG;
    if (!d->trip_angles || !d->trip_family || !d->lut || !d->poles_cart || !d->pole_family || !d->ang_table ||
        !d->fam_count || !d->fam_index)
        return EBSD_E_ARG;
    const int nt = d->ntrip, np_ = d->npoles, nf = d->nfam;
    for (int i = 0; i < 81; ++i)
        if (d->lut[i] < 0 || d->lut[i] > 2) return EBSD_E_ARG;
    for (int i = 0; i < 3 * nt; ++i)
        if (d->trip_family[i] < 0 || d->trip_family[i] >= nf) return EBSD_E_ARG;
    for (int i = 0; i < np_; ++i)
        if (d->pole_family[i] < 0 || d->pole_family[i] >= nf) return EBSD_E_ARG;
    for (int f = 0; f < nf; ++f)
        if (d->fam_index[f] < 0 || d->fam_count[f] < 0 || d->fam_index[f] + d->fam_count[f] > np_) return EBSD_E_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return EBSD_E_DEVICE;
    if (cudaSetDevice(device) != cudaSuccess) return EBSD_E_DEVICE;

    auto* p = new ebsd_vote_plan_s();
    p->device = device;
    p->nfam = nf;
    p->ntrip = nt;
    p->npoles = np_;
    p->tol = d->ang_tol;
    p->early = d->nband_earlyexit;
    p->simpleq = d->simple_qweights ? 1 : 0;
    for (int s0 = 0; s0 < 3; ++s0)
        for (int s1 = 0; s1 < 3; ++s1)
            for (int s2 = 0; s2 < 3; ++s2) {
                int code = 0;
                for (int r = 0; r < 3; ++r) code |= int(d->lut[((r * 3 + s0) * 3 + s1) * 3 + s2]) << (2 * r);
                p->lut[s0 * 9 + s1 * 3 + s2] = (uint8_t)code;
            }
    std::vector<float> iv0(6 * (size_t)nt);
    std::vector<uint32_t> tf(nt);
    for (int q = 0; q < nt; ++q) {
        for (int c = 0; c < 3; ++c)
            accept_interval(d->trip_angles[3 * q + c], d->ang_tol, &iv0[(2 * c) * nt + q], &iv0[(2 * c + 1) * nt + q]);
        tf[q] = uint32_t(d->trip_family[3 * q]) | uint32_t(d->trip_family[3 * q + 1]) << 8 |
                uint32_t(d->trip_family[3 * q + 2]) << 16;
    }
    // interval rows sorted by the lower end of the first angle's interval (library order kept
    // in d_orig), so that a band triplet scans only the rows whose first interval can hold it
    std::vector<int32_t> order(nt);
    for (int q = 0; q < nt; ++q) order[q] = q;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return iv0[a] < iv0[b]; });
    std::vector<float> iv(6 * (size_t)nt);
    double wmax = 0.0;
    for (int r = 0; r < nt; ++r) {
        const int q = order[r];
        for (int c = 0; c < 6; ++c) iv[(size_t)c * nt + r] = iv0[(size_t)c * nt + q];
        if (iv0[q] <= iv0[nt + q]) wmax = std::max(wmax, (double)iv0[nt + q] - (double)iv0[q]);
    }
    p->win = (float)(wmax + 1e-3);
    std::vector<float> pole(4 * (size_t)np_);
    for (int i = 0; i < np_; ++i) {
        for (int c = 0; c < 3; ++c) pole[4 * (size_t)i + c] = (float)d->poles_cart[3 * i + c];
        const int32_t fam = d->pole_family[i];
        std::memcpy(&pole[4 * (size_t)i + 3], &fam, 4);
    }
    std::vector<int32_t> fidx(nf);
    for (int f = 0; f < nf; ++f) fidx[f] = (int32_t)d->fam_index[f];

    auto up = [](void** dst, const void* src, size_t bytes) -> int {
        if (cudaMalloc(dst, bytes) != cudaSuccess) return EBSD_E_NOMEM;
        if (cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice) != cudaSuccess) return EBSD_E_LAUNCH;
        return EBSD_OK;
    };
    int rc = EBSD_OK;
    if (!rc) rc = up((void**)&p->d_iv, iv.data(), iv.size() * 4);
    if (!rc) rc = up((void**)&p->d_tfam, tf.data(), tf.size() * 4);
    if (!rc) rc = up((void**)&p->d_tang, d->trip_angles, 3 * (size_t)nt * 8);
    if (!rc) rc = up((void**)&p->d_pole, pole.data(), pole.size() * 4);
    if (!rc) rc = up((void**)&p->d_pole64, d->poles_cart, 3 * (size_t)np_ * 8);
    if (!rc) rc = up((void**)&p->d_angtab, d->ang_table, (size_t)np_ * np_ * 8);
    if (!rc) rc = up((void**)&p->d_famcnt, d->fam_count, (size_t)nf * 4);
    if (!rc) rc = up((void**)&p->d_famidx, fidx.data(), (size_t)nf * 4);
    if (!rc) rc = up((void**)&p->d_orig, order.data(), (size_t)nt * 4);
    if (!rc && cudaMalloc((void**)&p->d_cand, (size_t)nf * np_ * 2 * 4) != cudaSuccess) rc = EBSD_E_NOMEM;
    if (!rc && cudaMalloc((void**)&p->d_triad, (size_t)nf * np_ * 8 * 4) != cudaSuccess) rc = EBSD_E_NOMEM;
    if (!rc && cudaMalloc((void**)&p->d_par, 4) != cudaSuccess) rc = EBSD_E_NOMEM;
    if (!rc) {
        const int total = nf * np_;
        k_vote_thresholds<<<(total + 127) / 128, 128>>>(p->d_angtab, p->d_famidx, (const float4*)p->d_pole, nf, np_,
                                                        p->tol, (float)p->tol, p->d_cand, p->d_par, p->d_triad);
        rc = launch_status();
        if (!rc && cudaMemcpy(&p->par, p->d_par, 4, cudaMemcpyDeviceToHost) != cudaSuccess) rc = EBSD_E_LAUNCH;
    }
    if (rc) {
        ebsd_vote_plan_destroy(p);
        return rc;
    }
    *out = p;
    return EBSD_OK;
}

extern "C" int ebsd_vote_plan_destroy(ebsd_vote_plan_t p) {
    if (!p) return EBSD_OK;
    cudaSetDevice(p->device);
    cudaFree(p->d_iv);
    cudaFree(p->d_tfam);
    cudaFree(p->d_tang);
    cudaFree(p->d_pole);
    cudaFree(p->d_pole64);
    cudaFree(p->d_triad);
    cudaFree(p->d_angtab);
    cudaFree(p->d_famcnt);
    cudaFree(p->d_famidx);
    cudaFree(p->d_cand);
    cudaFree(p->d_par);
    cudaFree(p->d_orig);
    cudaFree(p->d_quest);
    delete p;
    return EBSD_OK;
}

extern "C" int ebsd_band_index(ebsd_vote_plan_t p, const float* d_norms, const float* d_intensity, int64_t n,
                               int32_t nBands, const ebsd_index_out* out, void* stream) {
    if (!p || !out || n < 0 || nBands < 1 || nBands > 32) return EBSD_E_ARG;
    if (n == 0) return EBSD_OK;
    if (!d_norms || !out->quat || !out->fit || !out->cm || !out->polematch || !out->nmatch || !out->ij ||
        !out->acc_correct || !out->bandfit)
        return EBSD_E_ARG;
    if (cudaSetDevice(p->device) != cudaSuccess) return EBSD_E_DEVICE;
    const size_t words = block_words(p->ntrip, p->npoles) + kWarps * warp_words(nBands, p->nfam);
    const size_t smem = words * 4;
    int dev_max = 0;
    cudaDeviceGetAttribute(&dev_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, p->device);
    if (smem > (size_t)dev_max) return EBSD_E_UNSUPPORTED;
    static int raised[64] = {};
    if (smem > 48 * 1024 && raised[p->device] < (int)smem) {
        EBSD_CUDA_TRY(cudaFuncSetAttribute(k_band_index, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        raised[p->device] = (int)smem;
    }
    VoteArgs A;
    A.iv = p->d_iv;
    A.tfam = p->d_tfam;
    A.tang = p->d_tang;
    A.pole = p->d_pole;
    A.pole64 = p->d_pole64;
    A.triad = p->d_triad;
    A.angtab = p->d_angtab;
    A.famcnt = p->d_famcnt;
    A.famidx = p->d_famidx;
    A.cand = p->d_cand;
    A.par = p->par;
    A.orig = p->d_orig;
    A.win = p->win;
    A.nfam = p->nfam;
    A.ntrip = p->ntrip;
    A.npoles = p->npoles;
    A.nb = nBands;
    A.tol_f = (float)p->tol;
    A.tol = p->tol;
    A.early = p->early;
    A.simpleq = p->simpleq;
    std::memcpy(A.lut, p->lut, 27);
    A.lut[27] = 0;
    // patterns go in pieces of at most kQuestChunk; the hand-over scratch is allocated on the
    // first call (make it outside a CUDA-graph capture) and reused
    constexpr int64_t kQuestChunk = 1 << 20;
    const int64_t cap = std::min<int64_t>(n, kQuestChunk);
    if (cap > p->quest_cap) {
        cudaFree(p->d_quest);
        p->d_quest = nullptr;
        p->quest_cap = 0;
        EBSD_CUDA_TRY(cudaMalloc(&p->d_quest, (size_t)cap * sizeof(QuestInput)));
        p->quest_cap = cap;
    }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_band_index, kWarps * 32, smem);
    if (per_sm < 1) per_sm = 1;
    const int nf = p->nfam;
    for (int64_t off = 0; off < n; off += kQuestChunk) {
        const int64_t cnt = std::min<int64_t>(kQuestChunk, n - off);
        A.norms = d_norms + off * nBands * 3;
        A.inten = d_intensity ? d_intensity + off * nBands : nullptr;
        A.n = cnt;
        ebsd_index_out o = *out;
        o.quat += 4 * off;
        o.fit += off;
        o.cm += off;
        o.polematch += off * nBands;
        o.nmatch += off;
        o.ij += 4 * off;
        o.acc_correct += off;
        o.bandfit += off * nBands;
        if (o.accw) o.accw += off * nf * nBands;
        if (o.accn) o.accn += off * nf * nBands;
        if (o.bandfam) o.bandfam += off * nBands;
        if (o.bandrank) o.bandrank += off * nBands;
        if (o.polevalid) o.polevalid += off * nBands;
        A.out = o;
        A.quest = (QuestInput*)p->d_quest;
        const int64_t need = (cnt + kWarps - 1) / kWarps;
        const int blocks = (int)std::min<int64_t>(need, (int64_t)sms * per_sm);
        k_band_index<<<blocks, kWarps * 32, smem, (cudaStream_t)stream>>>(A);
        int rc = launch_status();
        if (rc != EBSD_OK) return rc;
        const int qb = (int)std::min<int64_t>((cnt + 127) / 128, (int64_t)sms * 16);
        k_quest<<<qb, 128, 0, (cudaStream_t)stream>>>(A.quest, cnt, nBands, A.norms, A.inten, o.polematch,
                                                     p->d_pole64, o.quat);
        if ((rc = launch_status()) != EBSD_OK) return rc;
        k_quest_fit<<<qb, 128, 0, (cudaStream_t)stream>>>(A.quest, A.norms, o.polematch, p->d_pole64, o.quat, cnt,
                                                         nBands, o.fit, o.bandfit);
        if ((rc = launch_status()) != EBSD_OK) return rc;
    }
    return EBSD_OK;
}

extern "C" int ebsd_band_intensity(const float* d_max, const float* d_normmax, const float* d_theta,
                                   const float* d_rho, const int8_t* d_valid, int64_t n, int32_t nBands,
                                   float rhomax, float* d_adj, float* d_pq, float* d_iq, void* stream) {
    if (n < 0 || nBands < 1 || nBands > 128) return EBSD_E_ARG;
    if (n == 0) return EBSD_OK;
    if (!d_max || !d_theta || !d_rho || !d_valid || !d_adj || (d_iq && !d_normmax)) return EBSD_E_ARG;
    const int blocks = (int)std::min<int64_t>((n + 127) / 128, 152 * 8);
    k_band_intensity<<<blocks, 128, 0, (cudaStream_t)stream>>>(d_max, d_normmax, d_theta, d_rho, d_valid, n,
                                                               nBands, rhomax, d_adj, d_pq, d_iq);
    return launch_status();
}
