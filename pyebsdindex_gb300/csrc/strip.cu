// Band detection of integer patterns in two kernels joined by the Radon image in L2 / HBM:
//
//   k_strip_pack    eight uint8 (or four uint16) patterns interleaved pixel by pixel, by image
//                   column and by image row, with a zero apron
//   k_strip_radon   their Radon means.  A ray of the reference's sampling (radon_fast.py:113-158)
//                   takes one pixel per image column (or row), and its row moves by 0 or 1 from
//                   column to column: over four columns it is one of eight step words.  The block
//                   builds the sums of all eight words at every row of a four-column strip once,
//                   in shared memory, and every ray then adds one table entry per strip instead
//                   of four pixels.  Integer sums are exact in any order, so the means equal
//                   the pixel-by-pixel sums' (rdn_loops, radon_fast.py:281-310).
//   k_strip_peaks   padding, LoG convolution, max filter, top-N and band fit of one pattern (or one
//                   theta slab of it): band_detect.py:562-809, rows along theta, columns along rho
//   k_strip_merge   theta slabs only: the slabs' peaks merged and the bands fitted
//
// Measured (GB300, 2.07 GHz): 262,144 uint8 patterns of 80x80 in 37.9 ms, against 46.3 ms for the
// one-tile kernel that gathers pixel by pixel (fused.cu); 9,000 uint16 patterns of 120x120 in 4.9 ms
// against 9.5 ms in theta slabs (slab.cu); 5,000 each of 60x60, 120x120 and 240x240 in 12.0 against
// 25.9 ms.  Of 353 us for 2,432 patterns of 80x80 the word sums take 164 (shared-memory wavefronts at
// 73 % of their rate, the rays' 16-byte entry loads being most of them), the peak kernel 155 (16 warps
// per SM, issue at 40 %: latency), packing 21, the fits 9.
//
// The convolution's multiply-adds run in the per-stage kernels' order (theta taps, then rho taps),
// so the records equal theirs bit for bit; normmax's mean is reduced in another order (last bit).
#include "ebsd_internal.cuh"
#include "label.cuh"

#include <cstring>
#include <new>
#include <type_traits>

namespace ebsd {

namespace {

constexpr int kRThreads = 512, kRWarps = kRThreads / 32;
constexpr int kSlots = 12;              // 32-ray groups a warp accumulates at once (four registers each)
constexpr int kTaskGroups = kRWarps * kSlots;
constexpr int kWords = 8;               // step words of a four-pixel strip
constexpr int kApron = 3;

constexpr int kPThreads = 256, kPWarps = kPThreads / 32;
constexpr int kCapBand = 11;            // slab peak: value, position, 3x3 convolved values

struct StripTask {
    int octant;                         // 2 * axis (0: strips of columns, 1: of rows) + (rows counted from the end)
    int nph;                            // phases (SB strips each)
    int lut;                            // first 16-byte LUT vector of the task
    int act, cr;                        // first activity word, first entry of the slots' rays
};

struct RadonArgs {
    const uint2* elems;                 // [unit][E0 | E1] interleaved pixels
    size_t unit_elems;                  // elements of a unit
    size_t axis1;                       // first element of the by-row copy
    int V[2], PV[2];                    // cross-axis extent and pitch, per axis
    const StripTask* tasks;
    int ntask, parts;                   // parts: CTAs a task's slots are dealt over (small calls)
    const uint4* lut;
    const uint32_t* act;
    const float4* cr;                   // [slot][thread] of each task: count, RN(1 / count), bias, byte offset of the ray
    float* means;                       // [pattern][nRaysPad]
    int nRaysPad;
    int P;                              // word table pitch (rows)
    int64_t n;                          // patterns of this launch
    int nitem;                          // units x tasks x parts
};

// ---- k_strip_pack -------------------------------------------------------------------------
// One block per 32x32 tile of a unit's image: elements of 8 bytes holding one pixel of each of the
// unit's patterns, written by row (axis 1) and, through shared memory, by column (axis 0).  The
// aprons (kApron on both sides of the cross axis, and the strips' spare columns) are zeroed here
// too: the buffer is shared scratch.  Pixels no ray holds (the detector mask) are stored as zero.
template <typename InT>
__global__ void __launch_bounds__(256) k_strip_pack(const InT* __restrict__ pats, int64_t n, int H, int W,
                                                    const uint8_t* __restrict__ used, uint2* __restrict__ elems,
                                                    size_t unit_elems, size_t axis1, int PV0, int PV1, int U0, int U1) {
    constexpr int kPer = 8 / sizeof(InT);
    __shared__ uint2 t[32][33];
    const int64_t q0 = (int64_t)blockIdx.z * kPer;
    const int npk = (int)(n - q0 < kPer ? n - q0 : kPer);
    uint2* e0 = elems + (size_t)blockIdx.z * unit_elems;  // [x < U0][PV0]: by column
    uint2* e1 = e0 + axis1;                               // [y < U1][PV1]: by row
    // the tile covers x, y from -kApron on: both copies' cross axes start there
    const int x0 = blockIdx.x * 32 - kApron, y0 = blockIdx.y * 32 - kApron;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const size_t px = (size_t)H * W;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int x = x0 + tx, y = y0 + ty + 8 * s;
        uint2 e = make_uint2(0u, 0u);
        if (x >= 0 && x < W && y >= 0 && y < H && __ldg(used + y * W + x)) {
            const InT* p = pats + (size_t)q0 * px + (size_t)y * W + x;
            unsigned w[kPer];
#pragma unroll
            for (int j = 0; j < kPer; ++j) w[j] = j < npk ? (unsigned)__ldcs(p + j * px) : 0u;
            if (kPer == 8) {
                e.x = w[0] | (w[1] << 8) | (w[2] << 16) | (w[3] << 24);
                e.y = w[4 % kPer] | (w[5 % kPer] << 8) | (w[6 % kPer] << 16) | (w[7 % kPer] << 24);
            } else {
                e.x = w[0] | (w[1] << 16);
                e.y = w[2] | (w[3] << 16);
            }
        }
        t[ty + 8 * s][tx] = e;
        if (y >= 0 && y < U1 && x + kApron < PV1) e1[(size_t)y * PV1 + x + kApron] = e;
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int x = x0 + ty + 8 * s, y = y0 + tx;
        if (x >= 0 && x < U0 && y + kApron < PV0) e0[(size_t)x * PV0 + y + kApron] = t[tx][ty + 8 * s];
    }
}

// ---- k_strip_radon ------------------------------------------------------------------------
__device__ __forceinline__ uint4 add4(const uint4& a, const uint4& b) {
    return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ uint4 add4(const uint4& a, const uint4& b, const uint4& c) {
    return make_uint4(a.x + b.x + c.x, a.y + b.y + c.y, a.z + b.z + c.z, a.w + b.w + c.w);
}

// An element's pixels as sums: eight 16-bit lanes (uint8 patterns) or four words (uint16)
template <bool kU16>
__device__ __forceinline__ uint4 spread(uint2 e) {
    if (kU16) return make_uint4(e.x & 0xFFFFu, e.x >> 16, e.y & 0xFFFFu, e.y >> 16);
    return make_uint4(__byte_perm(e.x, 0u, 0x4140), __byte_perm(e.x, 0u, 0x4342), __byte_perm(e.y, 0u, 0x4140),
                      __byte_perm(e.y, 0u, 0x4342));
}

// Two float32 values in a 64-bit register, two operations per instruction, each rounded as its own
typedef unsigned long long Pair;
__device__ __forceinline__ Pair pack2(float a, float b) {
    Pair d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 unpack2(Pair p) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(p));
    return d;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
    Pair d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
    Pair d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
    Pair d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// RN(s / c) of two sums, r = RN(1 / c): one correction step of Markstein's division (P. Markstein,
// IBM J. Res. Dev. 34(1), 1990).  The quotient of a 24-bit integer and a count below 2^9 lies at
// least 2^-34 (relative) from any rounding boundary, far beyond the corrected value's error.
__device__ __forceinline__ Pair div_count(Pair s, Pair minus_c, Pair r) {
    const Pair q = mul2(s, r);
    return fma2(fma2(q, minus_c, s), r, q);
}

__device__ __forceinline__ void copy16(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ uint2 first_slot(const uint4& o) { return make_uint2(o.x, o.y); }
__device__ __forceinline__ uint2 second_slot(const uint4& o) { return make_uint2(o.z, o.w); }
__device__ __forceinline__ unsigned first_slot(const uint2& o) { return o.x; }
__device__ __forceinline__ unsigned second_slot(const uint2& o) { return o.y; }
__device__ __forceinline__ void add_entries(uint4& acc, const unsigned char* tb, uint2 o) {
    const uint4 t0 = *(const uint4*)(tb + (o.x & 0xFFFFu)), t1 = *(const uint4*)(tb + (o.x >> 16));
    const uint4 t2 = *(const uint4*)(tb + (o.y & 0xFFFFu)), t3 = *(const uint4*)(tb + (o.y >> 16));
    acc = add4(add4(acc, t0, t1), t2, t3);
}
__device__ __forceinline__ void add_entries(uint4& acc, const unsigned char* tb, unsigned o) {
    const uint4 t0 = *(const uint4*)(tb + (o & 0xFFFFu)), t1 = *(const uint4*)(tb + (o >> 16));
    acc = add4(acc, t0, t1);
}

template <int SB, bool kU16>
__global__ void __launch_bounds__(kRThreads, 1) k_strip_radon(const __grid_constant__ RadonArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    typedef typename std::conditional<SB == 4, uint4, uint2>::type Vec;  // LUT entries of two slots
    constexpr int kNV = kSlots / 2, kPer = kU16 ? 4 : 8;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int P = a.P;
    const int tab = SB * kWords * P * 16 + 16;  // bytes of one table; its last entry stays zero
    unsigned char* esm = smem + 2 * tab;
    if (tid < 8) ((unsigned*)(smem + (tid < 4 ? 0 : tab) + SB * kWords * P * 16))[tid & 3] = 0u;

    // The block's items (a unit of patterns, a task, a part of its slots), one after the other; the
    // first loads of the next are issued before the means of the last are written.
    StripTask tk;
    int PV = 0, ebytes = 0, dir = 0, epos = 0, dpos = 0;
    bool builds = false;
    unsigned mine = 0u, act = 0u;  // the slots this part takes; those with pixels in the phase
    const char* epix = nullptr;
    const Vec* lp = nullptr;
    const uint32_t* ap = nullptr;
    int64_t q0 = 0;
    Vec lut[kNV];
    const unsigned ebase = (unsigned)__cvta_generic_to_shared(esm);
    auto fetch = [&](int ph) {
        const char* s = epix + (size_t)ph * ebytes;
        for (int b = tid * 16; b < ebytes; b += kRThreads * 16) copy16(ebase + (ph & 1) * ebytes + b, s + b);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto open = [&](int item) {
        const int per = a.ntask * a.parts, unit = item / per, tp = item - unit * per;
        const int task = tp / a.parts, part = tp - task * a.parts;
        tk = a.tasks[task];
        const int axis = tk.octant >> 1, V = a.V[axis], rows = V + kApron;
        PV = a.PV[axis];
        ebytes = SB * 4 * PV * 8;         // one phase's interleaved pixels
        q0 = (int64_t)unit * kPer;
        epix = (const char*)(a.elems + (size_t)unit * a.unit_elems + (axis ? a.axis1 : 0));
        // this thread's row of the table: strip k of the phase, first-pixel row r - kApron
        const int k = tid / rows, r = tid - k * rows;
        builds = k < SB;
        dir = (tk.octant & 1) ? -1 : 1;
        epos = 4 * k * PV + ((tk.octant & 1) ? V - 1 - (r - kApron) + kApron : r);
        dpos = (k * kWords * P + r) * 16;
        mine = 0u;
        for (int g = part; g < kSlots; g += a.parts) mine |= 1u << g;
        // LUT: [phase][pair of slots][thread], SB 16-bit byte offsets into the table each; a pair is
        // loaded for the next phase as soon as it is used
        lp = (const Vec*)(a.lut + tk.lut) + tid;
        ap = a.act + tk.act + warp;
#pragma unroll
        for (int m = 0; m < kNV; ++m) lut[m] = __ldg(lp + m * kRThreads);
        act = __ldg(ap) & mine;
        fetch(0);
        if (tk.nph > 1) fetch(1);
    };
    // words by their steps: bit 2 the step to the second pixel, bit 1 to the third, bit 0 to the fourth
    auto build = [&](int ph) {
        if (!builds) return;
        const uint2* e = (const uint2*)(esm + (ph & 1) * ebytes) + epos;
        unsigned char* d = smem + (ph & 1) * tab + dpos;
        const uint4 x0 = spread<kU16>(e[0]);
        uint4 x3[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) x3[v] = spread<kU16>(e[3 * PV + v * dir]);
#pragma unroll
        for (int b0 = 0; b0 < 2; ++b0) {
            const uint4 s1 = add4(x0, spread<kU16>(e[PV + b0 * dir]));
#pragma unroll
            for (int b1 = 0; b1 < 2; ++b1) {
                const uint4 x2 = spread<kU16>(e[2 * PV + (b0 + b1) * dir]);
#pragma unroll
                for (int b2 = 0; b2 < 2; ++b2)
                    *(uint4*)(d + ((b0 * 4 + b1 * 2 + b2) * P) * 16) = add4(s1, x2, x3[b0 + b1 + b2]);
            }
        }
    };

    int item = blockIdx.x;
    if (item >= a.nitem) return;
    open(item);
    for (;;) {
        uint4 acc[kSlots];
#pragma unroll
        for (int g = 0; g < kSlots; ++g) acc[g] = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        build(0);
        __syncthreads();
        const int nph = tk.nph;
        for (int ph = 0; ph < nph; ++ph) {
            const bool more = ph + 1 < nph;
            if (ph + 2 < nph) fetch(ph + 2);  // its buffer was last read in the previous phase
            lp += kNV * kRThreads;
            ap += kRWarps;
            const unsigned next = more ? __ldg(ap) & mine : 0u;
            // half of the warps build the next table before they add this one's entries, half after
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                if (half == (warp & 1)) {
                    const unsigned char* tb = smem + (ph & 1) * tab;
#pragma unroll
                    for (int m = 0; m < kNV; ++m) {
                        const Vec o = lut[m];
                        if (more) lut[m] = __ldg(lp + m * kRThreads);
                        if ((act >> (2 * m)) & 1u) add_entries(acc[2 * m], tb, first_slot(o));
                        if ((act >> (2 * m + 1)) & 1u) add_entries(acc[2 * m + 1], tb, second_slot(o));
                    }
                } else if (more) {
                    build(ph + 1);
                }
            }
            act = next;
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
        }

        // the means, one row of nRaysPad per pattern.  An empty ray's is -1 (radon_fast.py:265): its
        // count is stored as 1 and its bias takes 1 from the zero sum.
        const float4* crp = a.cr + tk.cr + tid;  // count, RN(1 / count), bias, byte offset of the ray (-1: none)
        const unsigned took = mine;
        const int npk = (int)(a.n - q0 < kPer ? a.n - q0 : kPer);
        char* out = (char*)(a.means + (size_t)q0 * a.nRaysPad);
        const unsigned rowb = (unsigned)a.nRaysPad * 4u;
        item += gridDim.x;
        const bool again = item < a.nitem;
        if (again) open(item);
#pragma unroll
        for (int g = 0; g < kSlots; ++g) {
            const float4 cr = __ldg(crp + g * kRThreads);
            const unsigned s[4] = {acc[g].x, acc[g].y, acc[g].z, acc[g].w};
            const unsigned at = __float_as_uint(cr.w);
            const bool there = ((took >> g) & 1u) && at != 0xffffffffu;
            const Pair minus_c = pack2(-cr.x, -cr.x), rc = pack2(cr.y, cr.y), bias = pack2(cr.z, cr.z);
#pragma unroll
            for (int j = 0; j < kPer; j += 2) {
                Pair f;
                if (kU16) f = pack2((float)s[j & 3], (float)s[(j + 1) & 3]);
                else  // 2^23 + s: the sum in the low mantissa bits
                    f = pack2(__uint_as_float(__byte_perm(s[(j >> 1) & 3], 0x4B00u, 0x5410)),
                              __uint_as_float(__byte_perm(s[(j >> 1) & 3], 0x4B00u, 0x5432)));
                const float2 m = unpack2(div_count(add2(f, bias), minus_c, rc));
                if (there && j < npk) *(float*)(out + (at + j * rowb)) = m.x;
                if (there && j + 1 < npk) *(float*)(out + (at + (j + 1) * rowb)) = m.y;
            }
        }
        if (!again) return;
    }
}

// ---- k_strip_peaks ------------------------------------------------------------------------
struct PeakArgs {
    const float* means;                 // [pattern][nRaysPad], row j at j * rowp
    int nRaysPad, rowp;                 // rowp = 32 * ceil(nRho / 32)
    int nRho, nTheta, nB;
    int nslab;
    int NC, PC;                         // stored columns (rho from -(H0 + 2) to nRho + H0), tile pitch
    int nseg, SW;                       // rho segments of a row and their width
    int nstrip, strip_rows;             // theta strips of a slab
    int hb;                             // floats of one row buffer (a warp has two)
    int FW;                             // mask bytes of a row: a nibble per lane and segment
    int FC;                             // NC rounded up to whole lanes
    int CTmax;                          // most tile rows of a slab
    int stat_hi;                        // interior columns in the statistics slice
    float stat_last;                    // how often column nRho + H0 counts
    int nspecial;                       // zero-extended statistics rows
    float special[4];                   // their values per unit of the last row's theta response
    float special_sum;
    int topk;                           // candidates the first threshold aims at
    float ku[9];
    Pair kw[9];                         // both halves alike
    int mask_fixed;                     // the mask is the same for every theta
    const uint8_t* mask;                // [nTheta][FW] Radon mask in the candidates' layout
    LabelConsts kc;
    ebsd_bands out;
    int64_t out_offset;
    float* cap;                         // slabs: [pattern][slab][capf]
    int capf;
    float stat_unit;                    // statistics sums are integers in units of 1 / stat_unit
    double stat_scale;                  // 1 / stat_unit / cells of the statistics slice
};

__device__ __forceinline__ bool ahead(float v, int p, float w, int q) { return v > w || (v == w && p < q); }

__device__ __forceinline__ void list_add(float v, int pos, float& lv, int& lp, int nB, int lane) {
    const unsigned better = __ballot_sync(0xffffffffu, lane < nB && lp >= 0 && ahead(lv, lp, v, pos));
    const int ins = __popc(better);
    if (ins < nB) {
        const float uv = __shfl_up_sync(0xffffffffu, lv, 1);
        const int up = __shfl_up_sync(0xffffffffu, lp, 1);
        if (lane > ins && lane < nB) { lv = uv; lp = up; }
        if (lane == ins) { lv = v; lp = pos; }
    }
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// k-way merge of up to 32 sorted lists by one warp (lane l walks list l of `stride` entries):
// lanes 0..nB-1 get the best entries' positions and owning lists
template <typename V, typename I>
__device__ __forceinline__ int merge_lists(V val, I pos, int nlist, int nB, int lane, int& from, int& slot) {
    int ptr = 0, mine = -1;
    float hv = lane < nlist ? val(lane, 0) : -INFINITY;
    int hp = lane < nlist ? pos(lane, 0) : -1;
    for (int k = 0; k < nB; ++k) {
        const unsigned key = hp < 0 ? 0u : __float_as_uint(hv);  // positive values: ordered as integers
        const unsigned kmax = __reduce_max_sync(0xffffffffu, key);
        if (kmax == 0u) break;
        const unsigned pmin = __reduce_min_sync(0xffffffffu, key == kmax ? (unsigned)hp : 0xffffffffu);
        const bool win = key == kmax && (unsigned)hp == pmin;
        const int wl = __ffs(__ballot_sync(0xffffffffu, win)) - 1;
        const int ws = __shfl_sync(0xffffffffu, ptr, wl);
        if (lane == k) { mine = (int)pmin; from = wl; slot = ws; }
        if (win) {
            ++ptr;
            hp = ptr < nB ? pos(lane, ptr) : -1;
            hv = ptr < nB ? val(lane, ptr) : -INFINITY;
        }
    }
    return mine;
}

// Statistics sums are kept as integers in a unit of the plan's: exact in any order, so a record does not
// depend on how a pattern was split over slabs and warps.  The unit is the finest power of two for which no
// sum of the plan's cells leaves 62 bits (80x80: 2^-37 for uint8, 2^-29 for uint16), far below the
// float sums of four cells that are added in it, a dim pattern's too; the weights of those sums carry it, so
// that it costs no instruction.
double stat_unit(const ebsd_plan_s* p, int dtype, int statR) {
    double gu = 0.0, gw = 0.0;
    for (int k = 0; k < p->k0; ++k) gu += std::fabs((double)p->h_ku[k]);
    for (int k = 0; k < p->k1; ++k) gw += std::fabs((double)p->h_kw[k]);
    // means lie in [-1, 255] or [-1, 65535]; the float convolution's own rounding stays far below 1/256
    const double most = (dtype == EBSD_U8 ? 256.0 : 65536.0) * gu * gw * ((double)std::max(statR, 1) * p->nTheta);
    int e = 0;
    std::frexp(most, &e);
    return std::ldexp(1.0, 62 - e);
}

template <int K0, int K1, int NP>
__global__ void __launch_bounds__(kPThreads, 2) k_strip_peaks(const __grid_constant__ PeakArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int D0 = K0, D1 = K1, H0 = K0 / 2, H1 = K1 / 2;
    constexpr int kOff = H0 + 2;                     // tile column of rho 0
    constexpr int NQ = (4 + 2 * H0 + 3) / 4;         // float4 of theta responses under four outputs
    constexpr int kRing = K1 == 5 ? 8 : K1 + 1;      // rows a step: the taps' and those loaded ahead
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int PC = a.PC, nB = a.nB, ntask = a.nstrip * a.nseg;

    float* conv = (float*)smem;                                    // [CT][PC]
    float* hrows = conv + (size_t)a.CTmax * PC;                    // two row buffers per warp
    float* bests = hrows + (size_t)kPWarps * 2 * a.hb;             // [ntask][32] largest candidate of each lane
    float* gmax = bests + ntask * 32;                              // [32]
    float* redf = gmax + 32;                                       // [kPWarps] minima
    long long* reds = (long long*)(redf + kPWarps);                // [kPWarps] sums
    float2* found = (float2*)(reds + kPWarps);                     // [32] the first peaks found: value, position
    int* verified = (int*)(found + 32);
    int* ncol = verified + 1;
    uint16_t* cols_s = (uint16_t*)(verified + 4);                  // [ntask][32] columns to look at
    float* lv_s = hrows;                                           // peak lists: after the row buffers are dead
    int* lp_s = (int*)(hrows + kPWarps * kMaxBands);

    // Radon row u of a pattern's means, NP pairs of neighbouring rho per lane from rho ia (even) on (a
    // means row repeats the last rho to its end); beyond 0 / 180 degrees the row 180 degrees away, rho
    // flipped
    auto load = [&](const float* rad, int ia, int u, Pair* x) {
        if (u >= 0 && u < a.nTheta) {
            const Pair* row = (const Pair*)(rad + u * a.rowp + ia) + lane;
#pragma unroll
            for (int k = 0; k < NP; ++k) x[k] = __ldg(row + 32 * k);
        } else {
            const float* row = rad + (u < 0 ? u + a.nTheta : u - a.nTheta) * a.rowp;
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const int i = a.nRho - 1 - ia - 2 * (lane + 32 * k);
                x[k] = pack2(__ldg(row + max(i, 0)), __ldg(row + max(i - 1, 0)));
            }
        }
    };
    const int item = blockIdx.x;
    const int pat = item / a.nslab, slab = item - pat * a.nslab;
    const int j0 = a.nTheta * slab / a.nslab, j1 = a.nTheta * (slab + 1) / a.nslab;
    const int CT = j1 - j0 + 2 * D1;
    if (tid == 0) verified[0] = verified[1] = 0;

    // ---- convolution, statistics and candidate peaks: a warp walks a strip of theta rows of one rho
    // segment.  The Radon rows under the theta taps, and a few rows to come, sit in a ring of registers;
    // a step goes once round it, so that no row is moved.
    float smin = INFINITY, gbest = 0.0f;
    long long ssum = 0;
    const int ubase = j0 - D1;                       // theta index of tile row 0
    for (int task = warp; task < ntask; task += kPWarps) {
        const int strip = task / a.nseg, seg = task - strip * a.nseg;
        const int r_beg = strip * a.strip_rows;
        const int r_end = min(r_beg + a.strip_rows, CT);
        float best = 0.0f;
        __syncwarp();                                // the row buffers' last reads
        if (r_beg >= CT) {                           // the slab has fewer strips than the widest
            bests[task * 32 + lane] = 0.0f;
            continue;
        }
        const int c0 = seg * a.SW;
        const int cols = min(a.FC - c0, a.SW);       // this segment's columns
        const int first = c0 - kOff - H0;            // rho of the row buffer's first entry
        const int ia = max(first, 0), lpad = ia - first, rest = cols + 2 * H0 - lpad - 64 * NP;
        const int oc = c0 + 4 * lane;                // this lane's first output column
        const bool live = 4 * lane < cols, last_lane = 4 * (lane + 1) >= cols;
        float* hw0 = hrows + warp * 2 * a.hb + lpad + 2 * lane;  // this lane's writes and reads in the row buffers
        float* hw1 = hw0 + a.hb;
        const float* hb0 = hrows + warp * 2 * a.hb + (live ? 4 * lane : 0);
        const float* hb1 = hb0 + a.hb;
        const float* rad = a.means + (size_t)pat * a.nRaysPad;
        Pair x[kRing][NP];
#pragma unroll
        for (int i = 0; i < kRing - 1; ++i) load(rad, ia, ubase + r_beg - H1 + i, x[i]);
        // statistics: weights of the four columns, 0 or infinity to leave a column out of the minimum;
        // the lane with the last rho's response adds the zero-extended rows
        float wgt[4], out_of[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = oc + k - kOff;
            wgt[k] = !live || i < 0 ? 0.0f : (i < a.nRho + H0 ? (i < a.stat_hi ? 1.0f : 0.0f) : (i == a.nRho + H0 ? a.stat_last : 0.0f));
            out_of[k] = wgt[k] > 0.0f ? 0.0f : INFINITY;
            wgt[k] *= a.stat_unit;
        }
        const bool tail = seg == a.nseg - 1 && a.nspecial > 0 && last_lane && live;
        const float tail_out = tail ? 0.0f : INFINITY, tail_sum = tail ? a.special_sum * a.stat_unit : 0.0f;
        // outside the Radon mask nothing is a candidate: values are cut off at -infinity there
        const uint8_t* mrow = a.mask + ((ptrdiff_t)ubase * a.FW + seg * 32 + lane);
        const unsigned mfix = live ? __ldg(a.mask + seg * 32 + lane) : 0u;
        float cut[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) cut[k] = (mfix >> k) & 1u ? INFINITY : -INFINITY;
        float v1[4], t1[4], t2[4];                   // the previous row and its 3-maxima, those of the row before it
#pragma unroll
        for (int k = 0; k < 4; ++k) v1[k] = -INFINITY, t1[k] = -INFINITY, t2[k] = -INFINITY;
        float* crow = conv + r_beg * PC + oc;
        const float* nrow = rad + (ubase + r_beg - H1 + kRing - 1) * a.rowp + ia + 2 * lane;  // the next row to load
        // kInner: a whole step of the slab's own rows, every row it loads between 0 and 180 degrees,
        // and the mask the same for every theta
        auto step = [&](int r, auto inner_tag) {
            constexpr bool kInner = decltype(inner_tag)::value;
#pragma unroll
            for (int j = 0; j < kRing; ++j) {
                if (!kInner && r + j >= r_end) break;
                const bool own = kInner || (r + j >= D1 && r + j < CT - D1);
                if (kInner) {
#pragma unroll
                    for (int k = 0; k < NP; ++k) x[(j + kRing - 1) % kRing][k] = __ldg((const Pair*)nrow + 32 * k);
                } else {
                    load(rad, ia, min(ubase + r + j - H1 + kRing - 1, j1 + D1 + H1 - 1), x[(j + kRing - 1) % kRing]);
                }
                nrow += a.rowp;
                Pair h[NP];
                float* hw = (j & 1) ? hw1 : hw0;
#pragma unroll
                for (int k = 0; k < NP; ++k) {
                    h[k] = mul2(a.kw[0], x[(j + K1 - 1) % kRing][k]);
#pragma unroll
                    for (int b = 1; b < K1; ++b) h[k] = fma2(a.kw[b], x[(j + K1 - 1 - b) % kRing][k], h[k]);
                    *((Pair*)hw + 32 * k) = h[k];
                }
                if (lpad > 0) {                      // rho padding: the first row repeats
                    const float e = __shfl_sync(0xffffffffu, unpack2(h[0]).x, 0);
                    if (lane < lpad) hw[-lpad - lane] = e;
                }
                if (rest > 0) {                      // ... and the last, past this lane's loads
                    const float e = __shfl_sync(0xffffffffu, unpack2(h[NP - 1]).y, 31);
                    if (lane < rest) hw[64 * NP - lane] = e;
                }
                __syncwarp();
                float q[4 * NQ], o[4];
                const float4* h4 = (const float4*)((j & 1) ? hb1 : hb0);
#pragma unroll
                for (int m = 0; m < NQ; ++m) {
                    const float4 t = h4[m];
                    q[4 * m] = t.x, q[4 * m + 1] = t.y, q[4 * m + 2] = t.z, q[4 * m + 3] = t.w;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    o[k] = a.ku[0] * q[k + 2 * H0];
#pragma unroll
                    for (int ka = 1; ka < K0; ++ka) o[k] = fmaf(a.ku[ka], q[k + 2 * H0 - ka], o[k]);
                }
                if (live) *(float4*)crow = make_float4(o[0], o[1], o[2], o[3]);
                crow += PC;
                if (own) {
                    const float e = q[3 + 2 * H0];   // the last lane's: the last rho's response
                    float rsum = e * tail_sum;
#pragma unroll
                    for (int k = 0; k < 4; ++k) rsum = fmaf(o[k], wgt[k], rsum);
#pragma unroll
                    for (int z = 0; z < H0; ++z) smin = fminf(smin, fmaf(e, a.special[z], tail_out));
                    smin = min3(smin, o[0] + out_of[0], o[1] + out_of[1]);
                    smin = min3(smin, o[2] + out_of[2], o[3] + out_of[3]);
                    ssum += __float2ll_rn(rsum);
                }
                float left = __shfl_up_sync(0xffffffffu, o[3], 1), right = __shfl_down_sync(0xffffffffu, o[0], 1);
                if (lane == 0) left = -INFINITY;
                if (last_lane) right = -INFINITY;
                const float t0[4] = {max3(left, o[0], o[1]), max3(o[0], o[1], o[2]), max3(o[1], o[2], o[3]), max3(o[2], o[3], right)};
                // candidates of the previous row: no smaller than their eight neighbours (one that
                // another warp holds passes)
                if ((kInner && j > 0) || (r + j - 1 >= D1 && r + j - 1 < CT - D1 && r + j > r_beg)) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (v1[k] >= max3(t2[k], t1[k], t0[k])) best = fmaxf(best, v1[k]);
                }
                unsigned m = 0u;
                if (!kInner) m = a.mask_fixed || !own || !live ? mfix : __ldg(mrow + (r + j) * a.FW);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    t2[k] = t1[k], t1[k] = t0[k];
                    v1[k] = fminf(o[k], kInner ? cut[k] : ((m >> k) & 1u ? INFINITY : -INFINITY));
                }
            }
        };
        for (int r = r_beg; r < r_end; r += kRing) {
            const int un = ubase + r - H1 + kRing - 1;  // the step's first row to load
            if (a.mask_fixed && r >= D1 && r + kRing <= min(r_end, CT - D1) && un >= 0 && un + kRing <= a.nTheta)
                step(r, std::true_type{});
            else
                step(r, std::false_type{});
            if (kRing & 1) __syncwarp();             // the next step starts with the buffer just read
        }
        if (r_end - 1 >= D1 && r_end - 1 < CT - D1) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (v1[k] >= fmaxf(t2[k], t1[k])) best = fmaxf(best, v1[k]);
        }
        bests[task * 32 + lane] = best;
        gbest = fmaxf(gbest, best);
    }
    for (int t = 16; t > 0; t >>= 1) {
        ssum += __shfl_xor_sync(0xffffffffu, ssum, t);
        smin = fminf(smin, __shfl_xor_sync(0xffffffffu, smin, t));
    }
    const unsigned wbest = __reduce_max_sync(0xffffffffu, __float_as_uint(gbest));
    if (lane == 0) gmax[warp] = __uint_as_float(wbest);
    if (lane == 0) { redf[warp] = smin; reds[warp] = ssum; }
    __syncthreads();

    // ---- peaks: only the candidates that can be among the nB best are held against the whole
    // window: those above a threshold that about `want` of the lanes' largest candidates reach.  When
    // fewer than nB of them are peaks the threshold is lowered.  (All candidates are positive, so
    // their bits are ordered as the values.)
    float hi = 0.0f;
#pragma unroll
    for (int w = 0; w < kPWarps; ++w) hi = fmaxf(hi, gmax[w]);
    constexpr int kWin = (2 * D1 + 1) * (2 * D0 + 1), kWinLoads = (kWin + 31) / 32;
    short wr[kWinLoads], wc[kWinLoads];  // this lane's window cells
#pragma unroll
    for (int e0 = 0; e0 < kWinLoads; ++e0) {
        const int e = min(e0 * 32 + lane, kWin - 1);
        wr[e0] = (short)(e / (2 * D0 + 1));
        wc[e0] = (short)(e - wr[e0] * (2 * D0 + 1) - D0);
    }
    int want = a.topk;
    unsigned top = 0xffffffffu;
    float lv = -INFINITY;
    int lp = -1;
    for (;;) {
        unsigned thr = 0u;
        if (want < kPThreads / 2) {
            float lo = 0.0f, up = hi;
            for (int it = 0; it < 12; ++it) {
                const float mid = 0.5f * (lo + up);
                const int c = __syncthreads_count(gbest >= mid && mid > 0.0f);
                if (c < want) {
                    up = mid;
                } else {
                    lo = mid;
                    if (2 * c <= 3 * want) break;
                }
            }
            thr = __float_as_uint(lo);
            hi = lo;
        }
        // the columns (a task's lane) that hold such candidates, dealt over the warps
        for (int task = warp; task < ntask; task += kPWarps) {
            const unsigned bb = __float_as_uint(bests[task * 32 + lane]);
            if (bb != 0u && bb >= thr) cols_s[atomicAdd(ncol, 1)] = (uint16_t)(task * 32 + lane);
        }
        __syncthreads();
        const int ncols = *ncol;
        for (int e = warp; e < ncols; e += kPWarps) {
            const int id = cols_s[e], task = id >> 5, sl = id & 31;
            const int strip = task / a.nseg, seg = task - strip * a.nseg, c = seg * a.SW + 4 * sl;
            const int r_lo = max(strip * a.strip_rows, D1), r_hi = min((strip + 1) * a.strip_rows, CT - D1);
            for (int rr = r_lo; rr < r_hi; rr += 32) {  // a row per lane
                const int r = rr + lane;
                unsigned m = 0u;
                if (r < r_hi) {
                    m = __ldg(a.mask + (ptrdiff_t)(ubase + r) * a.FW + seg * 32 + sl);
                    float n[3][6];
#pragma unroll
                    for (int y = 0; y < 3; ++y) {
                        const float* p = conv + (r + y - 1) * PC + c;
                        const float4 t = *(const float4*)p;
                        n[y][0] = p[-1], n[y][1] = t.x, n[y][2] = t.y, n[y][3] = t.z, n[y][4] = t.w, n[y][5] = p[4];
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float v = n[1][k + 1];
                        const float big = max3(max3(n[0][k], n[0][k + 1], n[0][k + 2]), fmaxf(n[1][k], n[1][k + 2]),
                                               max3(n[2][k], n[2][k + 1], n[2][k + 2]));
                        const unsigned key = __float_as_uint(v);
                        if (!(v >= big && v > 0.0f && key >= thr && key < top)) m &= ~(1u << k);
                    }
                }
                unsigned todo = __ballot_sync(0xffffffffu, m != 0u);
                while (todo) {
                    const int s = __ffs(todo) - 1;
                    todo &= todo - 1;
                    unsigned mm = __shfl_sync(0xffffffffu, m, s);
                    while (mm) {
                        const int k = __ffs(mm) - 1;
                        mm &= mm - 1;
                        const float* win = conv + (rr + s - D1) * PC;
                        const float cv = win[D1 * PC + c + k];
                        bool ok = true;
#pragma unroll
                        for (int e0 = 0; e0 < kWinLoads; ++e0)
                            ok = ok && !(win[wr[e0] * PC + min(max(c + k + wc[e0], 0), a.NC - 1)] > cv);
                        if (__all_sync(0xffffffffu, ok)) {
                            const int pos = (c + k - kOff) * a.nTheta + j0 + rr + s - D1;
                            list_add(cv, pos, lv, lp, nB, lane);
                            if (lane == 0) {
                                const int at = atomicAdd(verified, 1);
                                if (at < 32) found[at] = make_float2(cv, __int_as_float(pos));
                            }
                        }
                    }
                }
            }
        }
        if (lane < nB) {
            lv_s[warp * kMaxBands + lane] = lv;
            lp_s[warp * kMaxBands + lane] = lp;
        }
        __syncthreads();
        const int have = *verified;
        if (have >= nB || thr == 0u) break;
        __syncthreads();  // every thread has read the counts
        if (tid == 0) *ncol = 0;
        __syncthreads();
        top = thr;
        want *= 3;
    }

    if (warp == 0) {
        int pos = -1;
        const int nf = *verified;
        if (nf <= 32) {
            // rank of each peak among all; lane k then takes the k-th
            const float2 mine = lane < nf ? found[lane] : make_float2(0.0f, __int_as_float(-1));
            const int mp = __float_as_int(mine.y);
            int rank = 0;
            for (int l = 0; l < nf; ++l) {
                const float2 o = found[l];
                rank += ahead(o.x, __float_as_int(o.y), mine.x, mp) ? 1 : 0;
            }
            if (lane >= nf) rank = 32;
            for (int k = 0; k < nB && k < nf; ++k) {
                const int who = __ffs(__ballot_sync(0xffffffffu, rank == k)) - 1;
                const int p = __shfl_sync(0xffffffffu, mp, who);
                if (lane == k) pos = p;
            }
        } else {
            int from = 0, slot = 0;
            pos = merge_lists([&](int l, int s) { return lv_s[l * kMaxBands + s]; },
                              [&](int l, int s) { return lp_s[l * kMaxBands + s]; }, kPWarps, nB, lane, from, slot);
        }
        float* d = a.cap + (size_t)item * a.capf;
        if (lane < nB) {
            const bool has = pos >= 0;
            const int i = has ? pos / a.nTheta : 0, j = has ? pos - i * a.nTheta : j0;
            float* e = d + 4 + lane * kCapBand;
            e[1] = __int_as_float(pos);
            const float* n0 = conv + (j - j0 + D1 - 1) * PC + i + kOff - 1;
#pragma unroll
            for (int t = 0; t < 9; ++t) e[2 + t] = n0[(t % 3) * PC + t / 3];
            e[0] = n0[PC + 1];
        }
    } else if (warp == 1) {
        float mn = lane < kPWarps ? redf[lane] : INFINITY;
        long long sum = lane < kPWarps ? reds[lane] : 0;
#pragma unroll
        for (int t = kPWarps / 2; t > 0; t >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, t);
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, t));
        }
        float* d = a.cap + (size_t)item * a.capf;
        if (lane == 0) { d[0] = mn; d[2] = __int_as_float((int)sum); d[3] = __int_as_float((int)(sum >> 32)); }
    }
}

// ---- band fits (band_detect.py:691-809) with the record's float64 fields --------------------
__device__ __forceinline__ void fit_band(const PeakArgs& a, int64_t pat, int band, int pos, const float* blk, float mn,
                                         long long sum) {
    const bool has = pos >= 0;
    float nn[9];
#pragma unroll
    for (int t = 0; t < 9; ++t) nn[t] = has ? blk[t] : 0.0f;
    const int i = has ? pos / a.nTheta : 0, j = has ? pos - i * a.nTheta : 0;
    const float mean = (float)((double)sum * a.stat_scale);
    band_fit_block<float>(has, i + a.kc.p0, j + a.kc.p1, nn, mn, mean, a.kc, a.out, (a.out_offset + pat) * a.nB + band);
}

__device__ __forceinline__ long long cap_sum(const float* d) {
    return (long long)(unsigned)__float_as_int(d[2]) | ((long long)__float_as_int(d[3]) << 32);
}

// One slab per pattern: a thread per band.
__global__ void __launch_bounds__(256) k_strip_fit(const __grid_constant__ PeakArgs a, int64_t nbands) {
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (t >= nbands) return;
    const int64_t pat = t / a.nB;
    const int b = (int)(t - pat * a.nB);
    const float* d = a.cap + (size_t)pat * a.capf;
    const float* e = d + 4 + b * kCapBand;
    fit_band(a, pat, b, __float_as_int(e[1]), e + 2, d[0], cap_sum(d));
}

// Several: one warp per pattern merges its slabs' peaks (at most 32 slabs).
__global__ void __launch_bounds__(128) k_strip_merge(const __grid_constant__ PeakArgs a, int64_t n) {
    const int lane = threadIdx.x & 31;
    const int64_t pat = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (pat >= n) return;
    const float* base = a.cap + (size_t)pat * a.nslab * a.capf;
    int from = 0, slot = 0;
    const int pos = merge_lists([&](int l, int s) { return base[(size_t)l * a.capf + 4 + s * kCapBand]; },
                                [&](int l, int s) { return __float_as_int(base[(size_t)l * a.capf + 4 + s * kCapBand + 1]); },
                                a.nslab, a.nB, lane, from, slot);
    float mn = INFINITY;
    long long sum = 0;
    if (lane < a.nslab) {
        const float* d = base + (size_t)lane * a.capf;
        mn = d[0];
        sum = cap_sum(d);
    }
#pragma unroll
    for (int t = 16; t > 0; t >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, t);
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, t));
    }
    if (lane < a.nB) fit_band(a, pat, lane, pos, base + (size_t)from * a.capf + 4 + slot * kCapBand + 2, mn, sum);
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
template <int K0, int K1>
void* peaks_np(int np) {
    return np == 1 ? (void*)k_strip_peaks<K0, K1, 1> : (void*)k_strip_peaks<K0, K1, 2>;
}

void* peaks_kernel(int k0, int k1, int np) {
    if (k0 == 5 && k1 == 5) return peaks_np<5, 5>(np);
    if (k0 == 7 && k1 == 7) return peaks_np<7, 7>(np);
    if (k0 == 9 && k1 == 9) return peaks_np<9, 9>(np);
    if (k0 == 5 && k1 == 7) return peaks_np<5, 7>(np);
    if (k0 == 7 && k1 == 5) return peaks_np<7, 5>(np);
    return nullptr;
}

void* radon_kernel(int sb, int dtype) {
    if (dtype == EBSD_U8) return sb == 4 ? (void*)k_strip_radon<4, false> : (void*)k_strip_radon<2, false>;
    return sb == 4 ? (void*)k_strip_radon<4, true> : (void*)k_strip_radon<2, true>;
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Theta strips of a slab: about one task per warp, two where a row has many
// segments.
void peaks_strips(const StripGeom& g, int ctmax, int* nstrip, int* strip_rows) {
    const int want = std::max(1, (kPWarps + g.nseg - 1) / g.nseg * (g.nseg > 2 ? 2 : 1));
    *strip_rows = (ctmax + want - 1) / want;
    *nstrip = (ctmax + *strip_rows - 1) / *strip_rows;
}

int peaks_smem(const StripGeom& g, int nTheta, int K1, int nslab, int* ctmax) {
    const int own = (nTheta + nslab - 1) / nslab;
    *ctmax = own + 2 * K1;
    int nstrip = 0, rows = 0;
    peaks_strips(g, *ctmax, &nstrip, &rows);
    return *ctmax * g.PC * 4 + kPWarps * 2 * g.hb * 4 + nstrip * g.nseg * (128 + 64) + 32 * 4 + kPWarps * 12 + 32 * 8 + 16;
}

int radon_smem(const StripGeom& g, int sb) {
    return 2 * (sb * kWords * g.P * 16 + 16) + 2 * sb * 4 * std::max(g.PV[0], g.PV[1]) * 8;
}

// A ray of one theta as strip words: for every four-column strip with pixels the table entry
// (word, first row) whose cells are the ray's pixels there, cells the ray lacks being off the
// image or in no ray at all.  False when some strip fits no word.
bool ray_words(const int* v, int U, int V, const std::vector<char>& used_uv, std::vector<uint32_t>& out) {
    out.clear();
    for (int s = 0; 4 * s < U; ++s) {
        int cell[4], firstk = -1;
        for (int k = 0; k < 4; ++k) {
            cell[k] = 4 * s + k < U ? v[4 * s + k] : -1;
            if (cell[k] >= 0 && firstk < 0) firstk = k;
        }
        if (firstk < 0) continue;
        bool ok = false;
        for (int w = 0; w < kWords && !ok; ++w) {
            const int off[4] = {0, w >> 2, (w >> 2) + ((w >> 1) & 1), (w >> 2) + ((w >> 1) & 1) + (w & 1)};
            const int base = cell[firstk] - off[firstk];
            ok = base >= -kApron;
            for (int k = 0; k < 4 && ok; ++k) {
                const int u = 4 * s + k, at = base + off[k];
                if (cell[k] >= 0) ok = cell[k] == at;
                else if (u < U && at >= 0 && at < V) ok = !used_uv[(size_t)u * V + at];
            }
            if (ok) out.push_back((uint32_t)s | ((uint32_t)w << 16) | ((uint32_t)(base + kApron) << 20));
        }
        if (!ok) return false;
    }
    return true;
}

template <typename T>
int to_device(T** dst, const std::vector<T>& v) {
    EBSD_CUDA_TRY(cudaMalloc((void**)dst, std::max<size_t>(1, v.size()) * sizeof(T)));
    EBSD_CUDA_TRY(cudaMemcpy(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return EBSD_OK;
}

}  // namespace

// Plan-time tables; leaves p->st.ok at 0 for plans these kernels do not take: a LoG that is not
// separable or of another size, windows other than the standard ones, rays that are not digital
// lines, or images beyond the table's 16-bit offsets.
int strip_prepare(ebsd_plan_s* p, const ebsd_plan_desc* d) {
    p->st = StripGeom{};
    StripGeom g;
    const int K0 = p->k0, K1 = p->k1, H0 = K0 / 2, nT = p->nTheta, nR = p->nRho, L = d->lut_len;
    const int big = std::max(p->H, p->W);
    if (!p->sep || !peaks_kernel(K0, K1, 1) || p->pk0 != 2 * K0 + 1 || p->pk1 != 2 * K1 + 1) return EBSD_OK;
    if (p->bg_mode != 0 || nR < 8 || nT < 2 * K1 + 1 || p->p0 < K0 + K0 / 2 || p->p1 < K1 + K1 / 2) return EBSD_OK;
    if (p->maxCount > 257 || nT < K1 + K1 / 2) return EBSD_OK;
    int dev_smem = 0, sm_smem = 0, ct = 0;
    cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, p->device);
    cudaDeviceGetAttribute(&sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, p->device);
    cudaDeviceGetAttribute(&g.sms, cudaDevAttrMultiProcessorCount, p->device);
    const int U[2] = {p->W, p->H}, V[2] = {p->H, p->W};
    // a table row's bank is its first-pixel row modulo 8: the pitch is a multiple of 8 entries
    g.P = (big + kApron + 7) & ~7;
    for (int ax = 0; ax < 2; ++ax) g.V[ax] = V[ax], g.PV[ax] = (V[ax] + 2 * kApron + 3) & ~3;
    // strips per phase: the table's byte offsets stay in 16 bits, two tables fit on chip and a block's
    // threads cover its rows
    for (int sb = 4; sb >= 2 && !g.SB; sb /= 2)
        if (sb * kWords * g.P * 16 + 16 <= 65535 && radon_smem(g, sb) <= dev_smem && sb * (big + kApron) <= kRThreads) g.SB = sb;
    if (!g.SB) return EBSD_OK;
    const unsigned zero_off = g.SB * kWords * g.P * 16;

    // ---- tile geometry of the peak kernel
    g.NC = nR + 2 * H0 + 3;
    // (a pitch of an odd number of float4 keeps a column of them free of bank conflicts)
    g.FC = (g.NC + 3) & ~3;
    // rho segments of a row: at most 32 lanes of four outputs, and two loads of two per lane for the
    // interior responses under them
    for (g.nseg = 1; g.nseg <= 16; ++g.nseg) {
        g.SW = ((g.FC + g.nseg - 1) / g.nseg + 3) & ~3;
        g.np = 1;
        for (int s = 0; s * g.SW < g.FC; ++s) {
            const int first = s * g.SW - (H0 + 2) - H0, cols = std::min(g.SW, g.FC - s * g.SW);
            g.np = std::max(g.np, (std::min(cols + 2 * H0 - std::max(0, -first), nR - std::max(0, first)) + 63) / 64);
        }
        if (g.SW <= 128 && g.np <= 2 && (g.nseg - 1) * g.SW < g.FC) break;
    }
    if (g.nseg > 16) return EBSD_OK;
    // row buffer: the padding before the first rho and np pairs of responses per lane, and what the last
    // lane's float4 reads reach (the warps' peak lists reuse the buffers: kMaxBands values and
    // positions each)
    g.hb = std::max(g.SW + 4 * ((4 + 2 * H0 + 3) / 4), (2 * H0 + 2 + 64 * g.np + 2 * H0 + 4 + 3) & ~3);
    g.hb = std::max(g.hb, kMaxBands);
    g.FW = 32 * g.nseg;
    g.PC = (g.FC / 4) | 1;
    g.PC *= 4;
    // a row of means holds every load of its segments
    int reach = nR;
    for (int s = 0; s * g.SW < g.FC; ++s) reach = std::max(reach, std::max(s * g.SW - (H0 + 2) - H0, 0) + 64 * g.np);
    g.gpt = (reach + 31) / 32;
    g.nRaysPad = nT * g.gpt * 32;
    for (int ns = 1; ns <= 32 && !g.nslab; ++ns) {
        const int b = peaks_smem(g, nT, K1, ns, &ct);
        // the fewest slabs whose tiles leave room for two blocks per SM
        if (b <= dev_smem && 2 * (b + 1024) <= sm_smem && nT / ns >= 8) g.nslab = ns;
    }
    if (!g.nslab) return EBSD_OK;

    // ---- pixels in use, rays as strip words
    std::vector<uint8_t> used(p->nPx, 0);
    for (size_t k = 0; k < (size_t)nR * nT * L; ++k)
        if (d->lut[k] >= 0 && d->lut[k] < p->nPx) used[d->lut[k]] = 1;
    std::vector<char> uv[4];  // by octant: [u][v'], v' counted from either end
    for (int o = 0; o < 4; ++o) {
        const int ax = o >> 1;
        uv[o].resize((size_t)U[ax] * V[ax]);
        for (int u = 0; u < U[ax]; ++u)
            for (int v = 0; v < V[ax]; ++v) {
                const int vv = (o & 1) ? V[ax] - 1 - v : v;
                uv[o][(size_t)u * V[ax] + v] = (char)used[ax == 0 ? vv * p->W + u : u * p->W + vv];
            }
    }
    const int nRays = g.gpt * 32;
    std::vector<std::vector<uint32_t>> words((size_t)nT * nRays);
    std::vector<int> oct(nT, 0);
    std::vector<float4> cr((size_t)g.nRaysPad), task_cr;
    std::vector<int> order((size_t)nT * 32);  // per theta: the ray of a group each lane takes
    std::vector<int> line((size_t)big);
    for (int j = 0; j < nT; ++j) {
        bool fits = false;
        for (int o = 0; o < 4 && !fits; ++o) {
            const int ax = o >> 1;
            fits = true;
            for (int i = 0; i < nR && fits; ++i) {
                const int64_t* ray = d->lut + ((size_t)i * nT + j) * L;
                std::fill(line.begin(), line.end(), -1);
                for (int k = 0; k < L && ray[k] >= 0 && ray[k] < p->nPx && fits; ++k) {
                    const int y = (int)(ray[k] / p->W), x = (int)(ray[k] - (int64_t)y * p->W);
                    const int u = ax == 0 ? x : y, v = ax == 0 ? y : x;
                    if (line[u] >= 0) fits = false;
                    line[u] = (o & 1) ? V[ax] - 1 - v : v;
                }
                if (fits) fits = ray_words(line.data(), U[ax], V[ax], uv[o], words[(size_t)j * nRays + i]);
            }
            if (fits) oct[j] = o;
        }
        if (!fits) return EBSD_OK;
        for (int i = nR; i < nRays; ++i) words[(size_t)j * nRays + i] = words[(size_t)j * nRays + nR - 1];
        // Neighbouring rays' rows are `step` apart.  Eight lanes read the table at once without
        // conflict when their rows differ modulo 8: the group's rays are sorted by row modulo 8 and
        // dealt over the four eighths-of-a-warp in turn.
        {
            const int ax = oct[j] >> 1;
            int lo = -1, hi = -1;
            uint32_t rlo = 0, rhi = 0;
            for (int i = 0; i < nR; ++i)
                for (uint32_t w : words[(size_t)j * nRays + i])
                    if ((int)(w & 0xFFFFu) == (U[ax] / 2) / 4) {
                        if (lo < 0) lo = i, rlo = w >> 20;
                        hi = i, rhi = w >> 20;
                    }
            const double step = hi > lo ? ((double)rhi - (double)rlo) / (hi - lo) : 1.0;
            int by[32];
            double key[32];
            for (int l = 0; l < 32; ++l) by[l] = l, key[l] = std::fmod(step * l + 8192.0, 8.0);
            std::stable_sort(by, by + 32, [&](int x, int y) { return key[x] < key[y]; });
            for (int l = 0; l < 32; ++l) order[(size_t)j * 32 + (l & 3) * 8 + (l >> 2)] = by[l];
        }
        for (int t = 0; t < nRays; ++t) {  // (past the last rho a row repeats it)
            const int i = (t & ~31) + order[(size_t)j * 32 + (t & 31)];
            int c = 0;
            const int64_t* ray = d->lut + ((size_t)std::min(i, nR - 1) * nT + j) * L;
            while (c < L && ray[c] >= 0 && ray[c] < p->nPx) ++c;
            float4 q = make_float4(c ? (float)c : 1.0f, c ? 1.0f / (float)c : 1.0f, c ? 0.0f : -1.0f, 0.0f);
            const uint32_t at = (uint32_t)(j * nRays + i) * 4u;
            std::memcpy(&q.w, &at, sizeof(at));
            cr[(size_t)j * nRays + t] = q;
        }
    }

    // ---- tasks: an octant's 32-ray groups dealt over blocks, warps and slots, longest first
    std::vector<StripTask> tasks;
    std::vector<uint16_t> lut;
    std::vector<uint32_t> act;
    for (int o = 0; o < 4; ++o) {
        struct Grp {
            int id, work;
        };
        std::vector<Grp> grps;
        for (int j = 0; j < nT; ++j)
            if (oct[j] == o)
                for (int b = 0; b < g.gpt; ++b) {
                    uint64_t phases[2] = {0, 0};
                    for (int l = 0; l < 32; ++l)
                        for (uint32_t w : words[(size_t)j * nRays + 32 * b + l]) {
                            const int ph = (int)(w & 0xFFFFu) / g.SB;
                            phases[ph >> 6] |= 1ull << (ph & 63);
                        }
                    grps.push_back(Grp{j * g.gpt + b, __builtin_popcountll(phases[0]) + __builtin_popcountll(phases[1])});
                }
        if (grps.empty()) continue;
        std::stable_sort(grps.begin(), grps.end(), [](const Grp& x, const Grp& y) { return x.work > y.work; });
        const int nt = ((int)grps.size() + kTaskGroups - 1) / kTaskGroups;
        const int ax = o >> 1, nph = ((U[ax] + 3) / 4 + g.SB - 1) / g.SB;
        for (int t = 0; t < nt; ++t) {
            const size_t base = lut.size();
            StripTask tk{o, nph, (int)(base / 8), (int)act.size(), (int)task_cr.size()};
            lut.resize(base + (size_t)nph * kSlots * kRThreads * g.SB, (uint16_t)zero_off);
            act.resize(act.size() + (size_t)nph * kRWarps, 0u);
            float4 none = make_float4(1.0f, 1.0f, 0.0f, 0.0f);
            std::memset(&none.w, 0xff, 4);
            task_cr.resize(task_cr.size() + (size_t)kSlots * kRThreads, none);
            int at = 0;
            for (size_t k = t; k < grps.size(); k += nt, ++at) {
                // boustrophedon over the warps, so that every warp gets long and short groups
                const int slot = at / kRWarps, w = (slot & 1) ? kRWarps - 1 - at % kRWarps : at % kRWarps;
                const int j = grps[k].id / g.gpt, b = grps[k].id % g.gpt;
                for (int l = 0; l < 32; ++l) task_cr[tk.cr + (size_t)slot * kRThreads + w * 32 + l] = cr[(size_t)grps[k].id * 32 + l];
                for (int l = 0; l < 32; ++l)
                    for (uint32_t wd : words[(size_t)j * nRays + 32 * b + order[(size_t)j * 32 + l]]) {
                        const int s = (int)(wd & 0xFFFFu), ph = s / g.SB, ks = s % g.SB;
                        const int word = (int)(wd >> 16) & 7, row = (int)(wd >> 20);
                        act[tk.act + ph * kRWarps + w] |= 1u << slot;
                        lut[base + (((size_t)ph * (kSlots / 2) + slot / 2) * kRThreads + w * 32 + l) * 2 * g.SB + (slot % 2) * g.SB + ks] =
                            (uint16_t)(((ks * kWords + word) * g.P + row) * 16);
                    }
            }
            tasks.push_back(tk);
        }
    }
    g.ntask = (int)tasks.size();
    if (!g.ntask) return EBSD_OK;
    for (int ax = 0; ax < 2; ++ax) {
        g.U[ax] = ((U[ax] + 4 * g.SB - 1) / (4 * g.SB)) * 4 * g.SB;
    }
    g.axis1 = (size_t)g.U[0] * g.PV[0];
    g.unit_elems = (g.axis1 + (size_t)g.U[1] * g.PV[1] + 31) & ~(size_t)31;

    // ---- Radon mask
    // (the candidates' layout: a byte per lane and segment, a bit per output)
    std::vector<uint32_t> mask((size_t)nT * g.FW / 4, 0u);
    for (int i = 0; i < nR; ++i)
        for (int j = 0; j < nT; ++j)
            if (d->rdnmask[(size_t)i * nT + j]) {
                const int c = i + H0 + 2, seg = c / g.SW, byte = j * g.FW + seg * 32 + (c - seg * g.SW) / 4;
                mask[byte >> 2] |= 1u << (8 * (byte & 3) + (c - seg * g.SW) % 4);
            }

    g.mask_fixed = 1;
    for (size_t k = g.FW / 4; k < mask.size(); ++k) g.mask_fixed &= mask[k] == mask[k - g.FW / 4];

    int rc = EBSD_OK;
    if (rc == EBSD_OK) rc = to_device((StripTask**)&p->d_st_tasks, tasks);
    if (rc == EBSD_OK) rc = to_device(&p->d_st_lut, lut);
    if (rc == EBSD_OK) rc = to_device(&p->d_st_act, act);
    // uint16 sums, then uint8 sums (which the kernel reads off a float's mantissa: 2^23 more)
    const size_t half = task_cr.size();
    for (size_t k = 0; k < half; ++k) {
        float4 q = task_cr[k];
        q.z -= 8388608.0f;
        task_cr.push_back(q);
    }
    g.ncr = (int64_t)half;
    if (rc == EBSD_OK) rc = to_device((float4**)&p->d_st_cr, task_cr);
    if (rc == EBSD_OK) rc = to_device(&p->d_st_mask, mask);
    if (rc == EBSD_OK) rc = to_device(&p->d_st_used, used);
    if (rc != EBSD_OK) {
        strip_release(p);
        return rc;
    }
    // patterns per pass over the workspace: about 224 MB of Radon means, whole waves of blocks
    const int64_t want = ((int64_t)224 << 20) / ((int64_t)g.nRaysPad * 4);
    const int64_t wave = 2 * g.sms;
    g.chunk = want >= wave ? want / wave * wave : std::max<int64_t>(8, want & ~(int64_t)7);
    g.capf = (4 + p->nB * kCapBand + 3) & ~3;
    g.ok = 1;
    p->st = g;
    return EBSD_OK;
}

// The scratch of a captured call belongs to the graph that the capture builds: its replays run whenever they
// are launched, beside other graphs and direct calls of the plan.  The graph holds a user object whose
// destructor, when the graph and its executables are gone, marks the buffer free for a later capture.
// The plan frees the buffers with its tables.
struct StripCaptures {
    struct Slot {
        StripScratch mem;
        bool held = false;
        unsigned long long id = 0;      // the capture and the stream: calls captured one after the other on
        cudaStream_t stream = nullptr;  // one stream share the buffer
    };
    std::mutex m;                       // never held over a call of the runtime
    std::vector<std::unique_ptr<Slot>> slots;
};

namespace {

struct CaptureHold {
    std::shared_ptr<StripCaptures> pool;
    StripCaptures::Slot* slot;
};

void CUDART_CB capture_gone(void* arg) {
    CaptureHold* h = (CaptureHold*)arg;
    {
        std::lock_guard<std::mutex> lk(h->pool->m);
        h->slot->held = false;
        h->slot->id = 0;
    }
    delete h;
}

void captures_release(ebsd_plan_s* p) {
    if (!p->st_captures) return;
    for (auto& s : p->st_captures->slots) {  // (the plan's lock guards the list and the buffers)
        cudaFree(s->mem.ptr);
        s->mem = StripScratch{};
    }
    p->st_captures.reset();
}

// This thread's allocations neither fail in nor end a capture that runs in the process: its own, on
// whatever stream, or another thread's in global mode.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

}  // namespace

void strip_release(ebsd_plan_s* p) {
    cudaFree(p->d_st_tasks);
    cudaFree(p->d_st_lut);
    cudaFree(p->d_st_act);
    cudaFree(p->d_st_cr);
    cudaFree(p->d_st_mask);
    cudaFree(p->d_st_used);
    p->d_st_tasks = nullptr;
    p->d_st_lut = nullptr;
    p->d_st_act = nullptr;
    p->d_st_cr = nullptr;
    p->d_st_mask = nullptr;
    p->d_st_used = nullptr;
    cudaFree(p->st_ws.ptr);
    p->st_ws = StripScratch{};
    captures_release(p);
    if (p->st_event) cudaEventDestroy(p->st_event);
    p->st_event = nullptr;
    p->st = StripGeom{};
}

// Integer patterns of every plan with tables, except uint8 patterns under a 9-tap theta smoothing that
// the eight-pattern one-tile kernel (fused.cu) takes: there the peak kernel's register ring spills, and
// 30,011 patterns of 60x60 took 5.4 ms here against 4.85 ms (80x80, too large for that tile: 8.2 ms for
// 20,000 against 11.6 in theta slabs; with five taps 60x60 is faster here as well).
// Nor are they served here while the caller pins a tile shape.
bool strip_serves(const ebsd_plan_s* p, int method, int dtype) {
    if (!p->st.ok || method != EBSD_FUSED_F32 || p->tile_pinned) return false;
    if (dtype == EBSD_U8) return !(p->k1 >= 9 && p->fg.ok_f32 && p->fg.quad);
    return dtype == EBSD_U16;
}

namespace {

struct StripLayout {
    size_t elems, means, cap, total;
};

// of a scratch that holds n patterns
StripLayout strip_layout(const StripGeom& g, int64_t n) {
    StripLayout l;
    l.elems = 0;
    // uint16 patterns go four to a unit, uint8 eight
    l.means = align256(((size_t)n + 3) / 4 * g.unit_elems * 8);
    l.cap = l.means + align256((size_t)n * g.nRaysPad * 4);
    const size_t blocks = std::max<size_t>((size_t)n * g.nslab, (size_t)8 * g.sms);
    l.total = l.cap + align256(blocks * g.capf * 4);
    return l;
}

std::mutex g_strip_mtx;
struct StripAttr {
    const void* fn;
    int device, smem;
};
std::vector<StripAttr> g_strip_attr;

int strip_attr(const void* fn, int device, int smem) {
    std::lock_guard<std::mutex> lk(g_strip_mtx);
    for (StripAttr& s : g_strip_attr)
        if (s.fn == fn && s.device == device) {
            if (smem > s.smem) {
                EBSD_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
                s.smem = smem;
            }
            return EBSD_OK;
        }
    EBSD_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    g_strip_attr.push_back(StripAttr{fn, device, smem});
    return EBSD_OK;
}

}  // namespace

namespace {

// Patterns of a scratch for calls of n: powers of two up to a whole pass (0.3 GB at 80x80), so that a plan
// of small calls stays small and calls of growing size allocate a few times at most.
int64_t scratch_cap(const StripGeom& g, int64_t n) {
    int64_t cap = 64;
    while (cap < n && cap < g.chunk) cap *= 2;
    return std::min(cap, g.chunk);
}

int scratch_alloc(const StripGeom& g, int64_t cap, StripScratch* out) {
    void* ptr = nullptr;
    const cudaError_t e = cudaMalloc(&ptr, strip_layout(g, cap).total);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? EBSD_E_NOMEM : EBSD_E_LAUNCH;
    }
    *out = StripScratch{ptr, cap};
    return EBSD_OK;
}

// Scratch for n patterns of a call on `st`, which is being captured into `graph`.
bool capture_scratch(ebsd_plan_s* p, cudaStream_t st, unsigned long long id, cudaGraph_t graph, int64_t n, StripScratch* got) {
    if (!p->st_captures) p->st_captures = std::make_shared<StripCaptures>();
    StripCaptures& c = *p->st_captures;
    const int64_t cap = scratch_cap(p->st, n);
    StripCaptures::Slot *slot = nullptr, *small = nullptr;
    {
        std::lock_guard<std::mutex> lk(c.m);
        for (auto& s : c.slots) {
            const bool fits = s->mem.cap >= cap;
            if (s->held && s->id == id && s->stream == st && fits) {
                *got = s->mem;
                return true;
            }
            if (s->held) continue;
            if (!fits) small = s.get();
            else if (!slot || s->mem.cap < slot->mem.cap) slot = s.get();
        }
        if (!slot) slot = small;  // a buffer that no graph holds makes room for a larger one
        if (!slot) {
            c.slots.emplace_back(new StripCaptures::Slot());
            slot = c.slots.back().get();
        }
        slot->held = true;
    }
    auto give_back = [&] {
        std::lock_guard<std::mutex> lk(c.m);
        slot->held = false;
        return false;
    };
    const RelaxedCapture relaxed;
    if (slot->mem.cap < cap) {
        cudaFree(slot->mem.ptr);
        slot->mem = StripScratch{};
        if (scratch_alloc(p->st, cap, &slot->mem) != EBSD_OK) return give_back();
    }
    CaptureHold* hold = new (std::nothrow) CaptureHold{p->st_captures, slot};
    if (!hold) return give_back();
    cudaUserObject_t obj = nullptr;
    if (cudaUserObjectCreate(&obj, hold, capture_gone, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
        cudaGetLastError();
        delete hold;
        return give_back();
    }
    if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        cudaGetLastError();
        cudaUserObjectRelease(obj, 1);  // capture_gone gives it back
        return false;
    }
    std::lock_guard<std::mutex> lk(c.m);
    slot->id = id;
    slot->stream = st;
    *got = slot->mem;
    return true;
}

}  // namespace

// Whether the plan's own scratch is there for calls of n patterns.
bool strip_has(const ebsd_plan_s* p, int64_t n) { return p->st_ws.ptr && p->st_ws.cap >= scratch_cap(p->st, n); }

// The plan's own scratch, for calls of up to n patterns, or of any number in passes.
int strip_reserve(ebsd_plan_s* p, int64_t n) {
    if (!p->st.ok) return EBSD_OK;
    if (strip_has(p, n)) return EBSD_OK;
    const RelaxedCapture relaxed;
    cudaFree(p->st_ws.ptr);  // (waits for the calls in flight that use it)
    p->st_ws = StripScratch{};
    return scratch_alloc(p->st, scratch_cap(p->st, n), &p->st_ws);
}

// Whether a call of n patterns on `st` has scratch (*got), allocated now if need be: the plan's own, or the
// graph's if the call is being captured.  Where memory is short the single-kernel paths serve the call.
bool strip_ready(ebsd_plan_s* p, cudaStream_t st, int64_t n, StripScratch* got) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    cudaGraph_t graph = nullptr;
    if (cudaStreamGetCaptureInfo(st, &cap, &id, &graph, nullptr, nullptr, nullptr) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (cap == cudaStreamCaptureStatusActive) {
        try {
            return capture_scratch(p, st, id, graph, n, got);
        } catch (const std::bad_alloc&) {
            return false;
        }
    }
    if (cap != cudaStreamCaptureStatusNone || strip_reserve(p, n) != EBSD_OK) return false;
    *got = p->st_ws;
    return true;
}

int strip_run_chunk(ebsd_plan_s* p, const StripScratch& scratch, int dtype, const void* d_pats, int64_t n, const ebsd_bands* out,
                    int64_t out_offset, cudaStream_t st, int64_t* launches) {
    if (n <= 0) return EBSD_OK;
    const StripGeom& g = p->st;
    const StripLayout lay = strip_layout(g, scratch.cap);
    char* ws = (char*)scratch.ptr;
    const int K0 = p->k0, H0 = K0 / 2, nR = p->nRho;
    const int per = dtype == EBSD_U8 ? 8 : 4;
    void* rfn = radon_kernel(g.SB, dtype);
    void* pfn = peaks_kernel(p->k0, p->k1, g.np);
    const int rsmem = radon_smem(g, g.SB);
    int rc = strip_attr(rfn, p->device, rsmem);
    if (rc != EBSD_OK) return rc;

    RadonArgs ra;
    ra.elems = (const uint2*)(ws + lay.elems);
    ra.unit_elems = g.unit_elems;
    ra.axis1 = g.axis1;
    for (int ax = 0; ax < 2; ++ax) ra.V[ax] = g.V[ax], ra.PV[ax] = g.PV[ax];
    ra.tasks = (const StripTask*)p->d_st_tasks;
    ra.ntask = g.ntask;
    ra.lut = (const uint4*)p->d_st_lut;
    ra.act = p->d_st_act;
    ra.cr = (const float4*)p->d_st_cr + (dtype == EBSD_U8 ? g.ncr : 0);
    ra.means = (float*)(ws + lay.means);
    ra.nRaysPad = g.nRaysPad;
    ra.P = g.P;

    PeakArgs pa;
    std::memset(&pa, 0, sizeof(pa));
    pa.means = ra.means;
    pa.nRaysPad = g.nRaysPad;
    pa.rowp = g.gpt * 32;
    pa.nRho = nR;
    pa.nTheta = p->nTheta;
    pa.nB = p->nB;
    pa.NC = g.NC;
    pa.PC = g.PC;
    pa.nseg = g.nseg;
    pa.SW = g.SW;
    pa.hb = g.hb;
    pa.FW = g.FW;
    pa.FC = g.FC;
    // statistics slice (band_detect.py:627-630): padded rows [p0, min(R, Tp - p0)); rho nRho + H0
    // and beyond repeat one value until the zero extension below the padded array comes in reach
    const int statR = std::min(p->R, p->Tp - p->p0) - p->p0;
    pa.stat_hi = std::min(statR, nR + H0);
    pa.stat_last = (float)std::max(0, std::min(statR, nR + p->p0 - H0) - (nR + H0));
    double ssum = 0.0;
    for (int z = 0; z < H0 && nR + p->p0 - H0 + z < statR; ++z) {
        float v = 0.0f;  // row R - H0 + z of the padded array: taps a < H0 - ... reach zero rows
        for (int ka = 0; ka < K0; ++ka)
            if (z - ka < 0) v = std::fma(p->h_ku[ka], 1.0f, v);
        pa.special[pa.nspecial++] = v;
        ssum += v;
    }
    for (int z = pa.nspecial; z < 4; ++z) pa.special[z] = pa.special[0];
    pa.special_sum = (float)ssum;
    const double unit = stat_unit(p, dtype, statR);
    pa.stat_unit = (float)unit;
    pa.stat_scale = 1.0 / (unit * statR * p->nTheta);
    pa.topk = p->nB + 6;
    for (int k = 0; k < 9; ++k) {
        pa.ku[k] = k < p->k0 ? p->h_ku[k] : 0.0f;
        uint32_t bits = 0;
        if (k < p->k1) std::memcpy(&bits, &p->h_kw[k], 4);
        pa.kw[k] = (Pair)bits << 32 | bits;
    }
    pa.mask = (const uint8_t*)p->d_st_mask;
    pa.mask_fixed = g.mask_fixed;
    pa.kc = LabelConsts{p->p0, p->p1, p->nTheta, p->nRho, p->nB, p->d_theta, p->d_rho};
    pa.out = *out;
    pa.cap = (float*)(ws + lay.cap);
    pa.capf = g.capf;

    // the plan's own scratch passes from stream to stream in call order (a graph's is ordered by the graph).
    // The wait is issued whatever the stream: a handle may be another stream's by now, or name one per thread.
    const bool live = scratch.ptr == p->st_ws.ptr;
    if (live && p->st_event) EBSD_CUDA_TRY(cudaStreamWaitEvent(st, p->st_event, 0));

    const size_t px = (size_t)p->nPx * elem_size(dtype);
    for (int64_t s = 0; s < n; s += scratch.cap) {
        const int64_t m = std::min<int64_t>(scratch.cap, n - s);
        const unsigned units = (unsigned)((m + per - 1) / per);
        const void* in = (const char*)d_pats + (size_t)s * px;
        // tiles over both copies: x up to max(U0, W + apron) and y likewise, from -kApron
        const dim3 pg((unsigned)((std::max(g.U[0], p->W + kApron) + kApron + 31) / 32),
                      (unsigned)((std::max(g.U[1], p->H + kApron) + kApron + 31) / 32), units);
        if (dtype == EBSD_U8)
            k_strip_pack<uint8_t><<<pg, 256, 0, st>>>((const uint8_t*)in, m, p->H, p->W, p->d_st_used, (uint2*)(ws + lay.elems),
                                                      g.unit_elems, g.axis1, g.PV[0], g.PV[1], g.U[0], g.U[1]);
        else
            k_strip_pack<uint16_t><<<pg, 256, 0, st>>>((const uint16_t*)in, m, p->H, p->W, p->d_st_used, (uint2*)(ws + lay.elems),
                                                       g.unit_elems, g.axis1, g.PV[0], g.PV[1], g.U[0], g.U[1]);
        // calls with few units deal each task's slots over several blocks
        ra.parts = 1;
        while (ra.parts < kSlots && (int64_t)units * g.ntask * ra.parts * 2 <= g.sms) ra.parts *= 2;
        ra.parts = std::min(ra.parts, kSlots);
        ra.n = m;
        ra.nitem = (int)units * g.ntask * ra.parts;
        void* rargs[] = {&ra};
        EBSD_CUDA_TRY(cudaLaunchKernel(rfn, dim3((unsigned)std::min(ra.nitem, g.sms)), dim3(kRThreads), rargs, (size_t)rsmem, st));
        // ... and each pattern's theta range over more slabs
        int ns = g.nslab;
        while (m * (ns + 1) <= 2 * g.sms && ns < 12 && p->nTheta / (ns + 1) >= 15) ++ns;
        pa.nslab = ns;
        const int psmem = peaks_smem(g, p->nTheta, p->k1, ns, &pa.CTmax);
        peaks_strips(g, pa.CTmax, &pa.nstrip, &pa.strip_rows);
        if ((rc = strip_attr(pfn, p->device, psmem)) != EBSD_OK) return rc;
        pa.out_offset = out_offset + s;
        void* pargs[] = {&pa};
        EBSD_CUDA_TRY(cudaLaunchKernel(pfn, dim3((unsigned)(m * ns)), dim3(kPThreads), pargs, (size_t)psmem, st));
        if (ns > 1) k_strip_merge<<<(unsigned)((m + 3) / 4), 128, 0, st>>>(pa, m);
        else k_strip_fit<<<(unsigned)((m * p->nB + 255) / 256), 256, 0, st>>>(pa, m * p->nB);
        *launches += 4;
    }
    if (live) {
        if (!p->st_event) EBSD_CUDA_TRY(cudaEventCreateWithFlags(&p->st_event, cudaEventDisableTiming));
        EBSD_CUDA_TRY(cudaEventRecord(p->st_event, st));
    }
    return launch_status();
}

}  // namespace ebsd
