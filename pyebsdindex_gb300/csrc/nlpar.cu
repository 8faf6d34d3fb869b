// NLPAR (non-local pattern averaging) on the device: the noise estimate and the weighted
// neighbour average that run in front of band detection.
//
//   k_nlpar_sigma    NLPAR.sigma_numba, nlpar_cpu.py:753-796 (nn = 1): min over the clipped
//                    3x3 scan neighbourhood of SSD / (2 n), then sqrt
//   k_nlpar_weights  NLPAR.nlpar_nb, nlpar_cpu.py:866-927: normalised pair distance to each
//                    pattern of the (2 sr + 1)^2 window (shifted inward at the scan edges),
//                    weight exp(-max(d - dthresh, 0) / lam^2), centre weight 1, normalised
//   k_nlpar_average  nlpar_cpu.py:929-934: weighted sum over the window for every pixel
//   *_tiled          the same two for 32 neighbouring scan pixels per block, with the patterns
//                    their windows touch staged in shared memory (used for sr <= 3)
//
// The float32 arithmetic keeps the reference's order: squared differences accumulate
// sequentially over the masked-pixel list, window weights are summed and applied in window
// order, and every add/mul is an explicitly rounded intrinsic (no contracted FMAs).
#include "ebsd_internal.cuh"

#include <algorithm>
#include <type_traits>

namespace ebsd {
namespace {

__device__ __forceinline__ void window(int i, int sr, int n, int& start, int& end) {
    int a = i - sr > 0 ? i - sr : 0;
    int b = i + sr - (n - 1) > 0 ? i + sr - (n - 1) : 0;
    start = a - b;
    int c = i + sr < n - 1 ? i + sr : n - 1;
    int e = sr - i > 0 ? sr - i : 0;
    end = c + e + 1;
}

// Sequential float32 SSD over the masked pixels where both values are below mxval.
__device__ __forceinline__ void pair_ssd(const float* __restrict__ a, const float* __restrict__ b,
                                         const int32_t* __restrict__ ind, int nind, float mxval,
                                         float n_init, float& d2, float& n2) {
    float d = 0.0f, n = n_init;
    for (int q = 0; q < nind; ++q) {
        int k = __ldg(ind + q);
        float x = __ldg(a + k), y = __ldg(b + k);
        if (y < mxval && x < mxval) {
            n = __fadd_rn(n, 1.0f);
            float t = __fsub_rn(x, y);
            d = __fadd_rn(d, __fmul_rn(t, t));
        }
    }
    d2 = d;
    n2 = n;
}

// One warp per 4 scan pixels, 8 lanes per pixel (one neighbour each), min over the lanes.
__global__ void k_nlpar_sigma(const float* __restrict__ data, int nrows, int ncols, int npx,
                              const int32_t* __restrict__ ind, int nind, float mxval,
                              float* __restrict__ sigma) {
    int gt = blockIdx.x * blockDim.x + threadIdx.x;
    int pix = gt >> 3, slot = gt & 7;
    int npix = nrows * ncols;
    float s0 = 1e24f;
    if (pix < npix) {
        int j = pix / ncols, i = pix - (pix / ncols) * ncols;
        int k = slot < 4 ? slot : slot + 1;  // skip the centre of the 3x3 block
        int jn = j + k / 3 - 1, inn = i + k % 3 - 1;
        if (jn >= 0 && jn < nrows && inn >= 0 && inn < ncols) {
            float d2, n2;
            pair_ssd(data + (int64_t)pix * npx, data + (int64_t)(inn + ncols * jn) * npx, ind, nind, mxval,
                     1.0e-12f, d2, n2);
            if (d2 >= 1.e-3f) s0 = __fdiv_rn(d2, __fmul_rn(n2, 2.0f));
        }
    }
    for (int o = 4; o > 0; o >>= 1) s0 = fminf(s0, __shfl_down_sync(0xffffffffu, s0, o, 8));
    if (slot == 0 && pix < npix) sigma[pix] = sqrtf(s0);
}

// One block per scan pixel, one thread per window slot.
__global__ void k_nlpar_weights(const float* __restrict__ data, int nrows, int ncols, int npx,
                                const int32_t* __restrict__ ind, int nind, float mxval,
                                const float* __restrict__ sigma, float lam2, float dthresh, int sr,
                                float* __restrict__ wout, const float* __restrict__ coff = nullptr) {
    extern __shared__ float w_s[];
    __shared__ float tot_s;
    int pix = blockIdx.x;
    int j = pix / ncols, i = pix - (pix / ncols) * ncols;
    int xs, xe, ys, ye;
    window(i, sr, ncols, xs, xe);
    window(j, sr, nrows, ys, ye);
    int wx = xe - xs, winsz = (2 * sr + 1) * (2 * sr + 1);
    int c = threadIdx.x;
    if (c < winsz) {
        int jn = ys + c / wx, inn = xs + c % wx;
        int nb = inn + ncols * jn;
        float w;
        if (nb == pix) {
            w = -1.0e6f;
        } else {
            float s0 = sigma[pix], s1 = sigma[nb];
            s0 = __fmul_rn(s0, s0);
            s1 = __fmul_rn(s1, s1);
            float d2, n2;
            pair_ssd(data + (int64_t)pix * npx, data + (int64_t)nb * npx, ind, nind, mxval, 0.0f, d2, n2);
            float ss = __fadd_rn(s0, s1);
            d2 = __fsub_rn(d2, __fmul_rn(n2, ss));
            float dnorm = __fmul_rn(ss, sqrtf(__fmul_rn(2.0f, n2)));
            w = dnorm > 1.e-8f ? __fdiv_rn(d2, dnorm) : __fmul_rn(1e6f, n2);
        }
        w = fmaxf(__fsub_rn(w, dthresh), 0.0f);
        w = expf(__fmul_rn(__fmul_rn(-1.0f, w), lam2));
        if (coff && nb == pix) w = __fadd_rn(w, coff[pix]);  // diff_offset's centre addition
        w_s[c] = w;
    }
    __syncthreads();
    if (c == 0) {
        float t = 0.0f;
        for (int k = 0; k < winsz; ++k) t = __fadd_rn(t, w_s[k]);
        tot_s = t;
    }
    __syncthreads();
    if (c < winsz) wout[(int64_t)pix * winsz + c] = __fdiv_rn(w_s[c], tot_s);
}

__device__ __forceinline__ float wadd(float acc, float x, float w) { return __fadd_rn(acc, __fmul_rn(x, w)); }
__device__ __forceinline__ double wadd(double acc, double x, double w) { return __dadd_rn(acc, __dmul_rn(x, w)); }

// The averaged value as stored: float as is; an unsigned integer type as the reference's pattern
// writer stores it (pat_flt2int with method 'clip', ebsd_pattern.py:118-182: clipped to the
// type's range, then truncated toward zero by astype).
template <typename O> __device__ __forceinline__ O store_as(float v);
template <> __device__ __forceinline__ float store_as<float>(float v) { return v; }
template <> __device__ __forceinline__ double store_as<double>(float v) { return (double)v; }
template <> __device__ __forceinline__ uint8_t store_as<uint8_t>(float v) {
    return (uint8_t)fminf(fmaxf(v, 0.0f), 255.0f);
}
template <> __device__ __forceinline__ uint16_t store_as<uint16_t>(float v) {
    return (uint16_t)fminf(fmaxf(v, 0.0f), 65535.0f);
}

// out[pix][k] = sum over the window, in window order, of data[nb][k] * w[pix][c].
template <typename T>
__global__ void k_nlpar_average(const T* __restrict__ data, int nrows, int ncols, int npx,
                                const T* __restrict__ w, int sr, T* __restrict__ out) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    int pix = blockIdx.y;
    if (k >= npx) return;
    int j = pix / ncols, i = pix - (pix / ncols) * ncols;
    int xs, xe, ys, ye;
    window(i, sr, ncols, xs, xe);
    window(j, sr, nrows, ys, ye);
    int winsz = (2 * sr + 1) * (2 * sr + 1);
    const T* wp = w + (int64_t)pix * winsz;
    T acc = (T)0;
    int c = 0;
    for (int jn = ys; jn < ye; ++jn)
        for (int inn = xs; inn < xe; ++inn, ++c)
            acc = wadd(acc, __ldg(data + (int64_t)(inn + ncols * jn) * npx + k), __ldg(wp + c));
    out[(int64_t)pix * npx + k] = acc;
}

// The same, stored as O.
template <typename O>
__global__ void k_nlpar_average_to(const float* __restrict__ data, int nrows, int ncols, int npx,
                                   const float* __restrict__ w, int sr, O* __restrict__ out) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    int pix = blockIdx.y;
    if (k >= npx) return;
    int j = pix / ncols, i = pix - (pix / ncols) * ncols;
    int xs, xe, ys, ye;
    window(i, sr, ncols, xs, xe);
    window(j, sr, nrows, ys, ye);
    int winsz = (2 * sr + 1) * (2 * sr + 1);
    const float* wp = w + (int64_t)pix * winsz;
    float acc = 0.0f;
    int c = 0;
    for (int jn = ys; jn < ye; ++jn)
        for (int inn = xs; inn < xe; ++inn, ++c)
            acc = wadd(acc, __ldg(data + (int64_t)(inn + ncols * jn) * npx + k), __ldg(wp + c));
    out[(int64_t)pix * npx + k] = store_as<O>(acc);
}

// ---- tiled kernels: one block per 32 neighbouring scan pixels of one scan row ------------
// The block stages, for a chunk of pixels, the values of every pattern its windows touch
// (2 sr + 1 rows x up to 32 + 4 sr columns of the scan) in shared memory, so that each pattern
// is read from memory once per block instead of once per (pixel, window slot); the per-pair
// and per-output arithmetic is the untiled kernels', in the same order.
constexpr int kTileX = 32;  // scan pixels per block
constexpr int kChunk = 32;  // pixel values per staged pattern per step
constexpr int kSP = kChunk + 1;  // staged row pitch (odd: lanes on different patterns, no conflicts)
constexpr int kTy = 16;     // threadIdx.y extent (blockDim = 32 x 16)

// Scan rows whose windows are shifted inward (rows within sr of the top or bottom edge), and
// columns likewise: their windows reach past +-sr.
__device__ __forceinline__ bool edge_row(int y, int sr, int nrows) { return y < sr || y >= nrows - sr; }
__device__ __forceinline__ bool edge_col(int x, int sr, int ncols) { return x < sr || x >= ncols - sr; }

// Distance weights of NLPAR.nlpar_nb (nlpar_cpu.py:866-927) for window slots c = ty + 16 j.
template <int MP>
__global__ void __launch_bounds__(kTileX * kTy) k_nlpar_weights_tiled(
        const float* __restrict__ data, int nrows, int ncols, int npx, const int32_t* __restrict__ ind,
        int nind, float mxval, const float* __restrict__ sigma, float lam2, float dthresh, int sr,
        float* __restrict__ wout, const float* __restrict__ coff) {
    extern __shared__ float sm[];
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kTileX + tx;
    const int y = blockIdx.y, x0 = blockIdx.x * kTileX;
    const int wn = 2 * sr + 1, winsz = wn * wn;
    int ys, ye;
    window(y, sr, nrows, ys, ye);
    const int cx0 = x0 - 2 * sr > 0 ? x0 - 2 * sr : 0;
    const int cx1 = x0 + kTileX + 2 * sr < ncols ? x0 + kTileX + 2 * sr : ncols;
    const int ncx = cx1 - cx0, nstage = wn * ncx;
    float* S = sm;                    // [nstage][kSP]
    float* W = sm + nstage * kSP;     // [kTileX][winsz], then [kTileX] totals
    float* T = W + kTileX * winsz;
    const int x = x0 + tx;
    const bool px_ok = x < ncols;
    int xs, xe;
    window(px_ok ? x : ncols - 1, sr, ncols, xs, xe);
    const int pix = y * ncols + (px_ok ? x : ncols - 1);
    const int cslot = (y - ys) * ncx + ((px_ok ? x : ncols - 1) - cx0);
    float d[MP], n[MP];
    int nbs[MP];
#pragma unroll
    for (int j = 0; j < MP; ++j) {
        const int c = ty + kTy * j;
        d[j] = 0.0f;
        n[j] = 0.0f;
        nbs[j] = c < winsz ? (c / wn) * ncx + (xs + c % wn - cx0) : cslot;
    }
    for (int q0 = 0; q0 < nind; q0 += kChunk) {
        const int qn = nind - q0 < kChunk ? nind - q0 : kChunk;
        const int k = tx < qn ? __ldg(ind + q0 + tx) : 0;
        __syncthreads();  // the previous chunk has been consumed
        for (int st = ty; st < nstage; st += kTy) {
            const int r = st / ncx, cc = st - r * ncx;
            const int64_t pat = (int64_t)(ys + r) * ncols + (cx0 + cc);
            S[st * kSP + tx] = tx < qn ? __ldg(data + pat * npx + k) : 0.0f;
        }
        __syncthreads();
        for (int qq = 0; qq < qn; ++qq) {
            const float xv = S[cslot * kSP + qq];
#pragma unroll
            for (int j = 0; j < MP; ++j) {
                const float yv = S[nbs[j] * kSP + qq];
                if (yv < mxval && xv < mxval) {  // pair_ssd's order: count, difference, square
                    n[j] = __fadd_rn(n[j], 1.0f);
                    const float t = __fsub_rn(xv, yv);
                    d[j] = __fadd_rn(d[j], __fmul_rn(t, t));
                }
            }
        }
    }
    // weights (k_nlpar_weights' arithmetic), then the window-order normalisation
#pragma unroll
    for (int j = 0; j < MP; ++j) {
        const int c = ty + kTy * j;
        if (c < winsz && px_ok) {
            const int jn = ys + c / wn, inn = xs + c % wn;
            const int nb = inn + ncols * jn;
            float w;
            if (nb == pix) {
                w = -1.0e6f;
            } else {
                float s0 = sigma[pix], s1 = sigma[nb];
                s0 = __fmul_rn(s0, s0);
                s1 = __fmul_rn(s1, s1);
                const float ss = __fadd_rn(s0, s1);
                const float d2 = __fsub_rn(d[j], __fmul_rn(n[j], ss));
                const float dnorm = __fmul_rn(ss, sqrtf(__fmul_rn(2.0f, n[j])));
                w = dnorm > 1.e-8f ? __fdiv_rn(d2, dnorm) : __fmul_rn(1e6f, n[j]);
            }
            w = fmaxf(__fsub_rn(w, dthresh), 0.0f);
            w = expf(__fmul_rn(__fmul_rn(-1.0f, w), lam2));
            if (coff && nb == pix) w = __fadd_rn(w, coff[pix]);  // diff_offset's centre addition
            W[tx * winsz + c] = w;
        }
    }
    __syncthreads();
    if (ty == 0 && px_ok) {
        float t = 0.0f;
        for (int c = 0; c < winsz; ++c) t = __fadd_rn(t, W[tx * winsz + c]);
        T[tx] = t;
    }
    __syncthreads();
    for (int i = tid; i < kTileX * winsz; i += kTileX * kTy) {
        const int px = i / winsz, c = i - px * winsz;
        if (x0 + px < ncols) wout[(int64_t)(y * ncols + x0 + px) * winsz + c] = __fdiv_rn(W[px * winsz + c], T[px]);
    }
}

// Weighted window sum (k_nlpar_average's order) for 32 scan pixels x 32 pattern pixels per step,
// stored as O (float, or clipped and truncated to uint8 / uint16 -- the detection input).
// SR > 0 fixes the search radius at compile time (unrolled window loops); 0 reads sr.
template <typename T, typename O, int SR>
__global__ void __launch_bounds__(kTileX * kTy) k_nlpar_average_tiled(
        const T* __restrict__ data, int nrows, int ncols, int npx, const T* __restrict__ w, int sr_arg,
        O* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smraw[];
    T* sm = (T*)smraw;
    const int sr = SR > 0 ? SR : sr_arg;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kTileX + tx;
    const int y = blockIdx.y, x0 = blockIdx.x * kTileX;
    const int wn = 2 * sr + 1, winsz = wn * wn;
    int ys, ye;
    window(y, sr, nrows, ys, ye);
    const int cx0 = x0 - 2 * sr > 0 ? x0 - 2 * sr : 0;
    const int cx1 = x0 + kTileX + 2 * sr < ncols ? x0 + kTileX + 2 * sr : ncols;
    const int ncx = cx1 - cx0;
    T* S = sm;                      // [wn rows][ncx][kSP]
    // [kTileX][WP]: each pixel's weights at a 16-byte aligned row of WP = winsz rounded up to 4,
    // read four at a time (one broadcast load for four window slots)
    const int WP = (winsz + 3) & ~3;
    T* Wt = sm + ((wn * ncx * kSP + 3) & ~3);
    const int npix_tile = ncols - x0 < kTileX ? ncols - x0 : kTileX;
    for (int i = tid; i < npix_tile * winsz; i += kTileX * kTy)
        Wt[(i / winsz) * WP + i % winsz] = w[(int64_t)(y * ncols + x0) * winsz + i];
    // this thread's scan pixels: the neighbours px = 2 ty + m (kTileX = 2 kTy), and their
    // windows' first staged column
    constexpr int kPx = kTileX / kTy;
    int xsc[kPx];
#pragma unroll
    for (int m = 0; m < kPx; ++m) {
        const int px = kPx * ty + m;
        int xs, xe;
        window(px < npix_tile ? x0 + px : x0, sr, ncols, xs, xe);
        xsc[m] = xs - cx0;
    }
    // neighbouring windows one column apart share all but one column of staged values
    const bool shared_cols = SR > 0 && kPx == 2 && kPx * ty + 1 < npix_tile && xsc[1] == xsc[0] + 1;
    for (int k0 = 0; k0 < npx; k0 += kChunk) {
        const int kn = npx - k0 < kChunk ? npx - k0 : kChunk;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < (SR > 0 ? 2 * SR + 1 : 1); ++r) {
            const int rr0 = SR > 0 ? r : 0, rr1 = SR > 0 ? r + 1 : wn;
            for (int rr = rr0; rr < rr1; ++rr) {
                const int64_t prow = (int64_t)(ys + rr) * ncols + cx0;
                for (int cc = ty; cc < ncx; cc += kTy)
                    S[(rr * ncx + cc) * kSP + tx] = tx < kn ? data[(prow + cc) * npx + k0 + tx] : (T)0;
            }
        }
        __syncthreads();
        if (tx >= kn) continue;
        if (SR > 0 && shared_cols) {
            // both pixels at once: each staged value loaded once for the two sums
            constexpr int WN = 2 * SR + 1, WS = WN * WN;
            const T* s0 = S + xsc[0] * kSP + tx;
            const T* wpa = Wt + (kPx * ty) * WP;
            const T* wpb = wpa + WP;
            T acc0 = (T)0, acc1 = (T)0;
#pragma unroll
            for (int c4 = 0; c4 < WS; c4 += 4) {
                T wa[4], wb[4];
                if (sizeof(T) == 4) {
                    const float4 a4 = *(const float4*)(wpa + c4), b4 = *(const float4*)(wpb + c4);
                    wa[0] = a4.x; wa[1] = a4.y; wa[2] = a4.z; wa[3] = a4.w;
                    wb[0] = b4.x; wb[1] = b4.y; wb[2] = b4.z; wb[3] = b4.w;
                } else {
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        wa[t] = c4 + t < WS ? wpa[c4 + t] : (T)0;
                        wb[t] = c4 + t < WS ? wpb[c4 + t] : (T)0;
                    }
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int c = c4 + t;
                    if (c < WS) {
                        const int r = c / WN, cc = c % WN;
                        acc0 = wadd(acc0, s0[(r * ncx + cc) * kSP], wa[t]);
                        acc1 = wadd(acc1, s0[(r * ncx + cc + 1) * kSP], wb[t]);
                    }
                }
            }
            const int64_t o = (int64_t)(y * ncols + x0 + kPx * ty) * npx + k0 + tx;
            out[o] = store_as<O>(acc0);
            out[o + npx] = store_as<O>(acc1);
            continue;
        }
#pragma unroll
        for (int m = 0; m < kPx; ++m) {
            const int px = kPx * ty + m;
            if (px < npix_tile) {
                const T* wp = Wt + px * WP;
                T acc = (T)0;
                int c = 0;
                for (int r = 0; r < wn; ++r) {
                    const T* srow = S + (r * ncx + xsc[m]) * kSP + tx;
                    for (int cc = 0; cc < wn; ++cc, ++c) acc = wadd(acc, srow[cc * kSP], wp[c]);
                }
                out[(int64_t)(y * ncols + x0 + px) * npx + k0 + tx] = store_as<O>(acc);
            }
        }
    }
}

template <typename T, typename O>
void launch_average_tiled(dim3 grid, dim3 block, size_t smem, cudaStream_t st, const T* data, int nrows, int ncols,
                          int npx, const T* w, int sr, O* out) {
    switch (sr) {
        case 1: k_nlpar_average_tiled<T, O, 1><<<grid, block, smem, st>>>(data, nrows, ncols, npx, w, sr, out); break;
        case 2: k_nlpar_average_tiled<T, O, 2><<<grid, block, smem, st>>>(data, nrows, ncols, npx, w, sr, out); break;
        case 3: k_nlpar_average_tiled<T, O, 3><<<grid, block, smem, st>>>(data, nrows, ncols, npx, w, sr, out); break;
        default: k_nlpar_average_tiled<T, O, 0><<<grid, block, smem, st>>>(data, nrows, ncols, npx, w, sr, out);
    }
}

typedef unsigned long long Pair2;              // two floats in a 64-bit register
__device__ __forceinline__ Pair2 p2_pack(float a, float b) {
    Pair2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 p2_unpack(Pair2 p) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(p));
    return d;
}
__device__ __forceinline__ Pair2 p2_add(Pair2 a, Pair2 b) {
    Pair2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// a * b, rounded by itself: the assembler contracts mul.f32x2 with an add that follows it into one
// multiply-add, so the product is a multiply-add of a zero that it cannot see (z, a run-time value)
__device__ __forceinline__ Pair2 p2_mul(Pair2 a, Pair2 b, Pair2 z) {
    Pair2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(z));
    return d;
}
// a - b: b's product with -1 is exact, so the sum is rounded once
__device__ __forceinline__ Pair2 p2_sub(Pair2 a, Pair2 b, Pair2 minus_one) {
    Pair2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(b), "l"(minus_one), "l"(a));
    return d;
}

// Weighted window sum, register-blocked along the scan row (search radius SR fixed).  A block
// takes RP neighbouring scan pixels of two rows and 4 * kRbThreads pattern values; each thread
// holds the 2 RP pixels' sums for four consecutive pattern values and streams the window rows'
// RP + 2 SR columns once: a loaded value feeds every pixel whose window holds it, and a broadcast
// weight feeds the four values, two at a time (packed products and sums, each rounded as its own).
// What bounds it is L2: with one row a block the 98 loads of 16 bytes per 8 pixels came to 9.7 TB/s
// (128x160 scan of 80x80, radius 3: 0.66 ms packed, 0.80 ms with scalar products).  Each sum adds its window slots in window order
// (rows, then columns) as fadd(acc, fmul(value, weight)) from zero -- the order and rounding of
// k_nlpar_average -- so the result equals the tiled kernel's bit for bit.  Needs npx % 4 == 0
// and 16-byte aligned data.
constexpr int kRbThreads = 128;
constexpr int kRbPix = 8;

template <typename O> __device__ __forceinline__ void store4(O* dst, const float* v);
template <> __device__ __forceinline__ void store4<float>(float* dst, const float* v) {
    *(float4*)dst = make_float4(v[0], v[1], v[2], v[3]);
}
template <> __device__ __forceinline__ void store4<uint8_t>(uint8_t* dst, const float* v) {
    *(uint32_t*)dst = (uint32_t)store_as<uint8_t>(v[0]) | ((uint32_t)store_as<uint8_t>(v[1]) << 8) |
                      ((uint32_t)store_as<uint8_t>(v[2]) << 16) | ((uint32_t)store_as<uint8_t>(v[3]) << 24);
}
template <> __device__ __forceinline__ void store4<uint16_t>(uint16_t* dst, const float* v) {
    *(uint2*)dst = make_uint2((uint32_t)store_as<uint16_t>(v[0]) | ((uint32_t)store_as<uint16_t>(v[1]) << 16),
                              (uint32_t)store_as<uint16_t>(v[2]) | ((uint32_t)store_as<uint16_t>(v[3]) << 16));
}

template <typename O, int SR>
__global__ void __launch_bounds__(kRbThreads) k_nlpar_average_rb(const float* __restrict__ data, int nrows, int ncols,
                                                                  int npx, const float* __restrict__ w,
                                                                  O* __restrict__ out, float zero) {
    constexpr int WN = 2 * SR + 1, WS = WN * WN, RP = kRbPix, NC = RP + 2 * SR;
    __shared__ Pair2 ws[2][RP * WS];  // each weight twice: one multiplies two pattern values at a time
    const Pair2 z = p2_pack(zero, zero);
    const int y = 2 * blockIdx.z, p0 = blockIdx.y * RP;
    const int np = ncols - p0 < RP ? ncols - p0 : RP, ny = nrows - y < 2 ? nrows - y : 2;
    for (int i = threadIdx.x; i < ny * np * WS; i += kRbThreads) {
        const int k = i / (np * WS), c = i - k * np * WS;
        const float v = w[((int64_t)(y + k) * ncols + p0) * WS + c];
        ws[k][c] = p2_pack(v, v);
    }
    __syncthreads();
    const int k = (blockIdx.x * kRbThreads + threadIdx.x) * 4;
    if (k >= npx) return;
    int ys, ye, ys1;
    window(y + ny - 1, SR, nrows, ys1, ye);  // the second row's window (one row: its own)
    const int y_last = ye;
    window(y, SR, nrows, ys, ye);
    const int sh = ys1 - ys;                 // 0 at the scan's top and bottom, else 1
    Pair2 acc[2][RP][2];
#pragma unroll
    for (int m = 0; m < RP; ++m) acc[0][m][0] = acc[0][m][1] = acc[1][m][0] = acc[1][m][1] = 0ull;
    const bool centred = p0 >= SR && p0 + RP + SR <= ncols;
    int xs[RP];
#pragma unroll
    for (int m = 0; m < RP; ++m) {
        int xe;
        window(m < np ? p0 + m : p0 + np - 1, SR, ncols, xs[m], xe);
    }
    // window row i of both pixel rows' union: slot row i of the first, i - sh of the second
    auto row = [&](int i, auto first, auto second) {
        constexpr bool kA = decltype(first)::value, kB = decltype(second)::value;
        const Pair2 *wa = ws[0] + i * WN, *wb = ws[1] + (i - sh) * WN;
        if (centred) {
            // every window of the block is centred: column j of the strip is slot j - m of pixel m
            const float* src = data + ((int64_t)(ys + i) * ncols + (p0 - SR)) * npx + k;
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const ulonglong2 v = __ldg((const ulonglong2*)(src + (int64_t)j * npx));
#pragma unroll
                for (int m = 0; m < RP; ++m) {
                    if (j - m < 0 || j - m >= WN) continue;
                    if (kA) {
                        const Pair2 wv = wa[m * WS + (j - m)];
                        acc[0][m][0] = p2_add(acc[0][m][0], p2_mul(v.x, wv, z));
                        acc[0][m][1] = p2_add(acc[0][m][1], p2_mul(v.y, wv, z));
                    }
                    if (kB) {
                        const Pair2 wv = wb[m * WS + (j - m)];
                        acc[1][m][0] = p2_add(acc[1][m][0], p2_mul(v.x, wv, z));
                        acc[1][m][1] = p2_add(acc[1][m][1], p2_mul(v.y, wv, z));
                    }
                }
            }
        } else {
            // windows shifted inward at the scan's left / right edge (starts do not decrease with m)
            const float* src = data + (int64_t)(ys + i) * ncols * npx + k;
            for (int c = xs[0]; c <= xs[RP - 1] + 2 * SR; ++c) {
                const ulonglong2 v = __ldg((const ulonglong2*)(src + (int64_t)c * npx));
#pragma unroll
                for (int m = 0; m < RP; ++m) {
                    const int d = c - xs[m];
                    if (m >= np || d < 0 || d >= WN) continue;
                    if (kA) {
                        const Pair2 wv = wa[m * WS + d];
                        acc[0][m][0] = p2_add(acc[0][m][0], p2_mul(v.x, wv, z));
                        acc[0][m][1] = p2_add(acc[0][m][1], p2_mul(v.y, wv, z));
                    }
                    if (kB) {
                        const Pair2 wv = wb[m * WS + d];
                        acc[1][m][0] = p2_add(acc[1][m][0], p2_mul(v.x, wv, z));
                        acc[1][m][1] = p2_add(acc[1][m][1], p2_mul(v.y, wv, z));
                    }
                }
            }
        }
    };
    for (int i = 0; ys + i < y_last; ++i) {
        const bool a = i < WN, b = ny == 2 && i >= sh;
        if (a && b) row(i, std::true_type(), std::true_type());
        else if (a) row(i, std::true_type(), std::false_type());
        else row(i, std::false_type(), std::true_type());
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int m = 0; m < RP; ++m)
            if (m < np && h < ny) {
                const float2 a = p2_unpack(acc[h][m][0]), b = p2_unpack(acc[h][m][1]);
                const float v[4] = {a.x, a.y, b.x, b.y};
                store4<O>(out + ((int64_t)(y + h) * ncols + p0 + m) * npx + k, v);
            }
}

// The weighted window sum of the pair path: the register-blocked kernel where it applies
// (radius 1-3, npx a multiple of 4, 16-byte aligned buffers), else the tiled kernel.
template <typename O>
void launch_average(dim3 tgrid, dim3 tblock, size_t tsmem, cudaStream_t st, const float* data, int nrows, int ncols,
                    int npx, const float* w, int sr, O* out) {
    const bool rb = sr >= 1 && sr <= 3 && npx % 4 == 0 && (uintptr_t)data % 16 == 0 && (uintptr_t)out % 16 == 0 &&
                    nrows <= 65535 && (ncols + kRbPix - 1) / kRbPix <= 65535;  // grid y / z limits
    if (!rb) {
        launch_average_tiled<float, O>(tgrid, tblock, tsmem, st, data, nrows, ncols, npx, w, sr, out);
        return;
    }
    const dim3 grid((unsigned)((npx / 4 + kRbThreads - 1) / kRbThreads), (unsigned)((ncols + kRbPix - 1) / kRbPix),
                    (unsigned)((nrows + 1) / 2));
    switch (sr) {
        case 1: k_nlpar_average_rb<O, 1><<<grid, kRbThreads, 0, st>>>(data, nrows, ncols, npx, w, out, 0.0f); break;
        case 2: k_nlpar_average_rb<O, 2><<<grid, kRbThreads, 0, st>>>(data, nrows, ncols, npx, w, out, 0.0f); break;
        default: k_nlpar_average_rb<O, 3><<<grid, kRbThreads, 0, st>>>(data, nrows, ncols, npx, w, out, 0.0f); break;
    }
}

// ---- pair kernels: each unordered pair's distance computed once ---------------------------
// The squared difference of a pair is symmetric bit for bit ((a - b)^2 == (b - a)^2 in float,
// and the saturation test is symmetric), so pixel p's distance to neighbour q is the same
// float sum whichever of the two computes it.  k_nlpar_pairs computes, for every scan pixel,
// the sums of the nF = sr (2 sr + 1) + sr "forward" offsets (dy, dx) -- dy > 0, or dy == 0 and
// dx > 0, |dy|, |dx| <= sr -- in the reference's pixel order; a pixel's window slot at offset
// -o reads the sum its neighbour computed for o.  Slots beyond +-sr, which only the windows
// shifted inward at the scan edges have, are summed directly from memory.  With kSig the
// kernel also sums the four forward 3x3 neighbours under sigma_numba's saturation level, from
// which k_nlpar_sigma_pairs takes the noise sigma without another pass over the patterns.
__device__ __forceinline__ int fwd_count(int sr) { return sr * (2 * sr + 1) + sr; }
__device__ __forceinline__ int fwd_index(int dy, int dx, int sr) {
    return dy == 0 ? dx - 1 : sr + (dy - 1) * (2 * sr + 1) + (dx + sr);
}

constexpr int kPairThreads = 256;
__device__ __forceinline__ void stage4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// ---- edge pixels: windows shifted inward, reaching past +-sr ----------------------------------
// Edge pixels are those of the sr top and bottom rows, and the sr left and right columns of the
// other rows; index: top rows, bottom rows, then per middle row its 2 sr edge columns.  Their
// raw window sums (SSD, count per slot, in the reference's pixel order) come from the pair sums and
// from edge_sums, and k_nlpar_weights_edge turns them into normalised weights, one block per edge
// pixel.
__device__ __forceinline__ int64_t edge_index(int y, int x, int sr, int nrows, int ncols) {
    if (y < sr) return (int64_t)y * ncols + x;
    if (y >= nrows - sr) return (int64_t)(sr + y - (nrows - sr)) * ncols + x;
    return (int64_t)2 * sr * ncols + (int64_t)(y - sr) * 2 * sr + (x < sr ? x : sr + x - (ncols - sr));
}

// The slots of an edge pixel's window that lie beyond +-sr (the pair sums hold the others).  A block
// takes two lines of the scan -- an edge line and a partner line more than sr away -- and 32 positions
// along them, one per lane; warp s sums window slot s along the line.  First the row pairs (edge row y,
// row y2 of its window; positions are columns, every column's window along x), then the column pairs
// (edge column x, column x2 of its window; positions are rows, and only slots within +-sr rows: the
// row pairs have the others).  Pixels stream through two buffers as in k_nlpar_pairs.
constexpr int kEdgePitch = kChunk + 1;

// Part of the pair kernel's launch: these blocks are few and long, and run beside the others.
__device__ void edge_sums(float* sm, int block, const float* __restrict__ data, int nrows, int ncols, int npx,
                          const int32_t* __restrict__ ind, int nind, float mxval, int sr, int row_blocks,
                          float2* __restrict__ raw) {
    const int lane = threadIdx.x & 31, s = threadIdx.x >> 5, wn = 2 * sr + 1, winsz = wn * wn, nw = blockDim.x >> 5;
    const bool cols = block >= row_blocks;
    const int b = cols ? block - row_blocks : block;
    const int nalong = cols ? nrows : ncols, nacross = cols ? ncols : nrows;
    const int nblk = (nalong + 31) / 32, line = b / nblk, p0 = (b - line * nblk) * 32;
    // line pair: side, then (edge line k = 0 .. sr - 1, one of its sr - k partners)
    const int per = sr * (sr + 1) / 2, side = line / per;
    int k = 0, t = line - side * per;
    while (t >= sr - k) t -= sr - k++;
    const int l1 = side ? nacross - 1 - k : k, l2 = side ? nacross - 1 - (k + sr + 1 + t) : k + sr + 1 + t;
    // staged: 32 positions of the edge line, then the partner's positions under their windows
    const int a0 = max(p0 - 2 * sr, 0), a1 = min(p0 + 32 + 2 * sr, nalong);
    const int n1 = min(32, nalong - p0), nst = n1 + a1 - a0;
    const int bufn = (32 + 32 + 4 * sr) * kEdgePitch;
    auto pattern = [&](int along, int across) { return data + ((int64_t)(cols ? along : across) * ncols + (cols ? across : along)) * npx; };
    auto stage = [&](int q0, float* buf) {
        const int q = q0 + lane;
        if (q < nind) {
            const int px = __ldg(ind + q);
            for (int i = s; i < nst; i += nw)
                stage4(buf + i * kEdgePitch + lane, (i < n1 ? pattern(p0 + i, l1) : pattern(a0 + i - n1, l2)) + px);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int p = p0 + lane;
    int ws, we;
    window(p < nalong ? p : nalong - 1, sr, nalong, ws, we);
    const int p2 = ws + (s < wn ? s : 0);  // the slot's position along the partner line
    const bool ok = s < wn && p < nalong && (!cols || (p2 - p <= sr && p - p2 <= sr));
    const int self = ok ? lane * kEdgePitch : 0, other = ok ? (n1 + p2 - a0) * kEdgePitch : 0;
    float d = 0.0f, n = 0.0f;
    stage(0, sm);
    for (int q0 = 0, it = 0; q0 < nind; q0 += kChunk, ++it) {
        const float* cur = sm + (it & 1) * bufn;
        const int qn = min(kChunk, nind - q0);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (q0 + kChunk < nind) stage(q0 + kChunk, sm + ((it + 1) & 1) * bufn);
        if (s >= wn) continue;
#pragma unroll 8
        for (int qq = 0; qq < qn; ++qq) {
            const float xv = cur[self + qq], yv = cur[other + qq];
            const float u = __fsub_rn(xv, yv), uu = __fmul_rn(u, u);
            if (yv < mxval && xv < mxval) {  // pair_ssd's order: count, difference, square
                n = __fadd_rn(n, 1.0f);
                d = __fadd_rn(d, uu);
            }
        }
    }
    if (!ok) return;
    const int y = cols ? p : l1, x = cols ? l1 : p, y2 = cols ? p2 : l2, x2 = cols ? l2 : p2;
    int ys, ye, xs, xe;
    window(y, sr, nrows, ys, ye);
    window(x, sr, ncols, xs, xe);
    raw[edge_index(y, x, sr, nrows, ncols) * winsz + (y2 - ys) * wn + (x2 - xs)] = make_float2(d, n);
}

// Register-blocked: a block takes 2 * kPairLanes neighbouring scan pixels of one row; warp dy sums
// the offsets into row y + dy, each lane two neighbouring pixels x, x + 1 against every dx -- the
// 2 SR + 2 values of row y + dy under both windows are loaded once as pairs and feed 2 SR + 1 packed
// (two-pixel) differences, squares and sums, each rounded as its own.  The patterns' next kChunk
// pixels stream into a second buffer (cp.async) while the current ones are summed, stored with the scan
// columns along the fast axis.  A pattern pixel with no value at or above a saturation level (nor a NaN)
// in the block's columns is summed without the per-term tests and counted whole; the others add zero
// for a term that does not count (3 of 10,000 values saturated, 60x61 scan of 60x60, radius 2, with the
// weights: 340 us; none 228; whole chunks term by term, branching: 1169 and 218; a sum per pair and slot,
// which saturation does not slow: 1087).  Measured, 128x160 scan of 80x80, radius 3: 1.35
// ms with one pair per thread and step (11 instructions a term, staging exposed), 0.84 ms now; bound by
// the summing warps' dependent packed operations: the offsets' differences, squares and sums are issued
// kind by kind and eight pixels unrolled (offset by offset, four pixels: 0.87; a third staging buffer,
// one block fewer an SM: 7 % more).
constexpr int kPairLanes = 30;                 // 60 pixels and 2 SR halo columns
constexpr int kPairPitch = 66;                 // staged columns (2 modulo 32: a column's 32 pixels in 16 banks)

// (Radius 3: the three blocks an SM that shared memory allows; left to itself the compiler spills with sigma.)
template <int SR, bool kSig>
__global__ void __launch_bounds__(kPairThreads, SR == 3 ? 3 : 0) k_nlpar_pairs(
        const float* __restrict__ data, int nrows, int ncols, int npx, const int32_t* __restrict__ ind,
        int nind, float mxval, float mxsig, float zero, float2* __restrict__ pairs, float2* __restrict__ sigp,
        int edge_rows, int edge_all, float2* __restrict__ raw) {
    extern __shared__ __align__(16) float sm[];
    constexpr int WN = 2 * SR + 1, kRowF = kChunk * kPairPitch, kBufF = (SR + 1) * kRowF, nF = SR * WN + SR;
    const int lane = threadIdx.x & 31, dy = threadIdx.x >> 5;
    if ((int)blockIdx.x < edge_all) {
        edge_sums(sm, blockIdx.x, data, nrows, ncols, npx, ind, nind, mxval, SR, edge_rows, raw);
        return;
    }
    __shared__ unsigned bad_s[2];                                 // the pixels of the buffers' chunks with a saturated value or a NaN
    const int nxb = (ncols + 2 * kPairLanes - 1) / (2 * kPairLanes);
    const int y = ((int)blockIdx.x - edge_all) / nxb, x0 = ((int)blockIdx.x - edge_all - y * nxb) * 2 * kPairLanes;
    const int nr = min(SR + 1, nrows - y);                        // rows y .. y + nr - 1 exist
    const int c_lo = max(SR - x0, 0), c_hi = min(kPairPitch, ncols - x0 + SR);  // staged columns that exist
    const float lim = kSig ? fminf(mxval, mxsig) : mxval;
    const Pair2 m1 = p2_pack(-1.0f, -1.0f), z = p2_pack(zero, zero);
    for (int i = threadIdx.x; i < 2 * kBufF; i += kPairThreads) sm[i] = 0.0f;  // columns and rows off the scan stay zero
    __syncthreads();
    // the warps past SR stage a chunk, wait for it and look it over while the others sum the one before
    constexpr int kHelpers = kPairThreads / 32 - SR - 1;
    const int helper = dy - SR - 1;
    auto stage = [&](int q0, int b) {
        float* buf = sm + b * kBufF;
        const int q = q0 + lane, qn = min(kChunk, nind - q0);
        if (helper == 0 && lane == 0) bad_s[b] = 0u;
        if (q < nind) {
            const float* src = data + ((int64_t)y * ncols + x0 - SR) * npx + __ldg(ind + q);
            float* dst = buf + lane * kPairPitch;
            const int64_t step = (int64_t)kHelpers * npx;
            for (int r = 0; r < nr; ++r) {
                const float* p = src + ((int64_t)r * ncols + c_lo + helper) * npx;
                float* t = dst + r * kRowF;
#pragma unroll 4
                for (int c = c_lo + helper; c < c_hi; c += kHelpers, p += step) stage4(t + c, p);
            }
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_all;" ::: "memory");
        __syncwarp();  // the aligned barrier takes whole warps; lanes past the chunk's end skipped the copies
        asm volatile("bar.sync 1, %0;" ::"n"(kHelpers * 32) : "memory");
        bool bad = false;
        for (int r = 0; r < nr; ++r) {
            const float2* row = (const float2*)(buf + r * kRowF);
#pragma unroll 4
            for (int i = helper * 32 + lane; i < qn * (kPairPitch / 2); i += kHelpers * 32) {
                const float2 v = row[i];
                bad |= !(v.x < lim) | !(v.y < lim);
            }
        }
        if (bad) {  // which pixels: rarely needed, so looked for in a pass of its own
            unsigned mask = 0u;
            for (int r = 0; r < nr; ++r) {
                const float2* row = (const float2*)(buf + r * kRowF);
#pragma unroll 1
                for (int i = helper * 32 + lane; i < qn * (kPairPitch / 2); i += kHelpers * 32) {
                    const float2 v = row[i];
                    if (!(v.x < lim) | !(v.y < lim)) mask |= 1u << (i / (kPairPitch / 2));
                }
            }
            atomicOr(&bad_s[b], mask);
        }
    };
    const bool mine = lane < kPairLanes && dy < nr && helper < 0;
    const int cl = mine ? 2 * lane : 0;                           // first staged column under pixel x = x0 + 2 lane
    Pair2 d[WN], ds[3];
    float n0 = 0.0f;                                              // terms of the chunks counted whole
    float na[WN], nb[WN], nsa[3], nsb[3];
#pragma unroll
    for (int e = 0; e < WN; ++e) d[e] = 0ull, na[e] = 0.0f, nb[e] = 0.0f;
#pragma unroll
    for (int e = 0; e < 3; ++e) ds[e] = 0ull, nsa[e] = 0.0f, nsb[e] = 0.0f;
    // sigma's forward neighbours: dx 1 in the same row; dx -1, 0, 1 in the next
    const bool near1 = kSig && dy == 1, near0 = kSig && dy == 0;
    // one pattern pixel; checked: a term counts if both its values lie below the level, else every term
    auto terms = [&](const float* q, int dyv, auto tag, auto checked) {
        constexpr int kKind = decltype(tag)::value;        // 0: the same row (dx > 0), 1: the next, 2: others
        constexpr bool kCheck = decltype(checked)::value;
        const float* pa = q + cl + SR;
        const Pair2 a = (SR & 1) ? p2_pack(pa[0], pa[1]) : *(const Pair2*)pa;
        const float* pb = q + dyv * kRowF + cl;
        Pair2 v[SR + 1];
#pragma unroll
        for (int k = 0; k <= SR; ++k)
            if (kKind != 0 || 2 * k + 1 > SR) v[k] = *(const Pair2*)(pb + 2 * k);
        constexpr int e0 = kKind == 0 ? SR + 1 : 0;
        Pair2 t[WN];
#pragma unroll
        for (int e = e0; e < WN; ++e) {
            const Pair2 b = (e & 1) ? p2_pack(p2_unpack(v[e / 2]).y, p2_unpack(v[e / 2 + 1]).x) : v[e / 2];
            t[e] = p2_sub(a, b, m1);
        }
#pragma unroll
        for (int e = e0; e < WN; ++e) t[e] = p2_mul(t[e], t[e], z);
        if (kCheck) {
            // a sum of squares plus zero is the sum, so a term that does not count adds zero
            const float2 av = p2_unpack(a);
            auto value = [&](int c) { return (c & 1) ? p2_unpack(v[c / 2]).y : p2_unpack(v[c / 2]).x; };
#pragma unroll
            for (int e = e0; e < WN; ++e) {
                const float2 u = p2_unpack(t[e]);
                const bool oka = av.x < mxval && value(e) < mxval, okb = av.y < mxval && value(e + 1) < mxval;
                d[e] = p2_add(d[e], p2_pack(oka ? u.x : 0.0f, okb ? u.y : 0.0f));
                na[e] += oka ? 1.0f : 0.0f;
                nb[e] += okb ? 1.0f : 0.0f;
                const int g = kKind == 0 ? 0 : e - SR + 1;  // sigma's sums
                if (kSig && (kKind == 0 ? e == SR + 1 : kKind == 1 && g >= 0 && g <= 2)) {
                    const bool sa = av.x < mxsig && value(e) < mxsig, sb = av.y < mxsig && value(e + 1) < mxsig;
                    ds[g] = p2_add(ds[g], p2_pack(sa ? u.x : 0.0f, sb ? u.y : 0.0f));
                    nsa[g] += sa ? 1.0f : 0.0f;
                    nsb[g] += sb ? 1.0f : 0.0f;
                }
            }
            return;
        }
#pragma unroll
        for (int e = e0; e < WN; ++e) {
            d[e] = p2_add(d[e], t[e]);
            if (kSig && kKind == 0 && e == SR + 1) ds[0] = p2_add(ds[0], t[e]);
            if (kSig && kKind == 1 && e >= SR - 1 && e <= SR + 1) ds[e - SR + 1] = p2_add(ds[e - SR + 1], t[e]);
        }
    };
    // a chunk of qn pixels, every term counted; and one with the pixels of the mask `bad` term by term
    auto whole = [&](const float* cur, int qn, int dyv, auto tag) {
#pragma unroll 8
        for (int qq = 0; qq < qn; ++qq) terms(cur + qq * kPairPitch, dyv, tag, std::false_type());
    };
    auto mixed = [&](const float* cur, int qn, unsigned bad, int dyv, auto tag) {
#pragma unroll 1
        for (int qq = 0; qq < qn; ++qq) {
            if ((bad >> qq) & 1u) terms(cur + qq * kPairPitch, dyv, tag, std::true_type());
            else terms(cur + qq * kPairPitch, dyv, tag, std::false_type());
        }
    };
    if (helper >= 0) stage(0, 0);
    __syncthreads();
    for (int q0 = 0, it = 0; q0 < nind; q0 += kChunk, ++it) {
        const float* cur = sm + (it & 1) * kBufF;
        const int qn = min(kChunk, nind - q0);
        if (helper >= 0) {
            if (q0 + kChunk < nind) stage(q0 + kChunk, (it + 1) & 1);
        } else if (mine) {
            const unsigned bad = bad_s[it & 1];
            if (bad == 0u) {
                if (dy == 0) whole(cur, qn, 0, std::integral_constant<int, 0>());
                else if (dy == 1) whole(cur, qn, 1, std::integral_constant<int, 1>());
                else whole(cur, qn, dy, std::integral_constant<int, 2>());
            } else if (dy == 0) {
                mixed(cur, qn, bad, 0, std::integral_constant<int, 0>());
            } else if (dy == 1) {
                mixed(cur, qn, bad, 1, std::integral_constant<int, 1>());
            } else {
                mixed(cur, qn, bad, dy, std::integral_constant<int, 2>());
            }
            n0 += (float)(qn - __popc(bad));               // (the counts are exact integers either way)
        }
        __syncthreads();  // the next chunk is in place, this one's buffer free
    }
    if (!mine) return;
    const int x = x0 + 2 * lane;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (x + h >= ncols) continue;
        const int64_t pix = (int64_t)y * ncols + x + h;
#pragma unroll
        for (int e = 0; e < WN; ++e) {
            const int dx = e - SR;
            if ((dy == 0 && dx <= 0) || x + h + dx < 0 || x + h + dx >= ncols) continue;
            const float2 s = p2_unpack(d[e]);
            pairs[pix * nF + (dy == 0 ? dx - 1 : SR + (dy - 1) * WN + e)] = make_float2(h ? s.y : s.x, n0 + (h ? nb[e] : na[e]));
            const int g = dx + 1;
            if (kSig && ((near1 && g >= 0 && g <= 2) || (near0 && g == 2))) {
#pragma unroll
                for (int z = 0; z < 3; ++z) {
                    if (z != (near0 ? 0 : g)) continue;
                    const float2 w = p2_unpack(ds[z]);
                    sigp[pix * 4 + (near0 ? 0 : 1 + g)] = make_float2(h ? w.y : w.x, n0 + (h ? nsb[z] : nsa[z]));
                }
            }
        }
    }
}

// sigma_numba (nn = 1) from the pair sums: min over the clipped 3x3 neighbourhood of
// SSD / (2 n) for SSD >= 1e-3 (the count starts at 1e-12, which the first add absorbs).
__global__ void k_nlpar_sigma_pairs(const float2* __restrict__ sigp, int nrows, int ncols, float* __restrict__ sigma) {
    const int64_t pix = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= (int64_t)nrows * ncols) return;
    const int j = (int)(pix / ncols), i = (int)(pix - (int64_t)j * ncols);
    // forward 3x3 offsets in sigp order, and their mirrors
    const int fdy[4] = {0, 1, 1, 1}, fdx[4] = {1, -1, 0, 1};
    float s0 = 1e24f;
    for (int k = 0; k < 8; ++k) {
        const int kk = k & 3;
        const int dy = k < 4 ? fdy[kk] : -fdy[kk], dx = k < 4 ? fdx[kk] : -fdx[kk];
        const int jn = j + dy, inn = i + dx;
        if (jn < 0 || jn >= nrows || inn < 0 || inn >= ncols) continue;
        const float2 e = k < 4 ? sigp[pix * 4 + kk] : sigp[((int64_t)jn * ncols + inn) * 4 + kk];
        const float n2 = e.y > 0.0f ? e.y : 1.0e-12f;
        if (e.x >= 1.e-3f) s0 = fminf(s0, __fdiv_rn(e.x, __fmul_rn(n2, 2.0f)));
    }
    sigma[pix] = sqrtf(s0);
}

// The window weights of k_nlpar_weights_tiled from the pair sums (slots c = ty + 16 j), for the
// pixels whose windows are centred; the edge pixels take k_nlpar_weights_edge.
template <int MP>
__global__ void __launch_bounds__(kTileX * kTy) k_nlpar_weights_pairs(
        int nrows, int ncols, const float2* __restrict__ pairs, const float* __restrict__ sigma, float lam2,
        float dthresh, int sr, float* __restrict__ wout, const float* __restrict__ coff) {
    __shared__ float W[kTileX * 49];
    __shared__ float T[kTileX];
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kTileX + tx;
    const int y = blockIdx.y, x0 = blockIdx.x * kTileX;
    if (edge_row(y, sr, nrows)) return;
    const int wn = 2 * sr + 1, winsz = wn * wn, nF = fwd_count(sr);
    int ys, ye;
    window(y, sr, nrows, ys, ye);
    const int x = x0 + tx;
    const bool px_ok = x < ncols && !edge_col(x, sr, ncols);
    int xs, xe;
    window(x < ncols ? x : ncols - 1, sr, ncols, xs, xe);
    const int64_t pix = (int64_t)y * ncols + (x < ncols ? x : ncols - 1);
#pragma unroll
    for (int j = 0; j < MP; ++j) {
        const int c = ty + kTy * j;
        if (c < winsz && px_ok) {
            const int jn = ys + c / wn, inn = xs + c % wn;
            const int64_t nb = (int64_t)jn * ncols + inn;
            const int dy = jn - y, dx = inn - x;
            float w;
            if (nb == pix) {
                w = -1.0e6f;
            } else {
                // (the windows here are centred: every slot lies within +-sr)
                const float2 e = (dy > 0 || (dy == 0 && dx > 0)) ? pairs[pix * nF + fwd_index(dy, dx, sr)]
                                                                : pairs[nb * nF + fwd_index(-dy, -dx, sr)];
                const float n2 = e.y;
                float d2 = e.x;
                float s0 = sigma[pix], s1 = sigma[nb];
                s0 = __fmul_rn(s0, s0);
                s1 = __fmul_rn(s1, s1);
                const float ss = __fadd_rn(s0, s1);
                d2 = __fsub_rn(d2, __fmul_rn(n2, ss));
                const float dnorm = __fmul_rn(ss, sqrtf(__fmul_rn(2.0f, n2)));
                w = dnorm > 1.e-8f ? __fdiv_rn(d2, dnorm) : __fmul_rn(1e6f, n2);
            }
            w = fmaxf(__fsub_rn(w, dthresh), 0.0f);
            w = expf(__fmul_rn(__fmul_rn(-1.0f, w), lam2));
            if (coff && nb == pix) w = __fadd_rn(w, coff[pix]);  // diff_offset's centre addition
            W[tx * winsz + c] = w;
        }
    }
    __syncthreads();
    if (ty == 0 && px_ok) {
        float t = 0.0f;
        for (int c = 0; c < winsz; ++c) t = __fadd_rn(t, W[tx * winsz + c]);
        T[tx] = t;
    }
    __syncthreads();
    for (int i = tid; i < kTileX * winsz; i += kTileX * kTy) {
        const int px = i / winsz, c = i - px * winsz;
        if (x0 + px < ncols && !edge_col(x0 + px, sr, ncols))
            wout[((int64_t)y * ncols + x0 + px) * winsz + c] = __fdiv_rn(W[px * winsz + c], T[px]);
    }
}

int edge_blocks(int sr, int nalong) { return sr * (sr + 1) * ((nalong + 31) / 32); }

// Normalised window weights of the edge pixels from their raw sums: one block (64 threads) per
// edge pixel, the arithmetic of k_nlpar_weights_tiled.
__global__ void k_nlpar_weights_edge(const float2* __restrict__ raw, const float2* __restrict__ pairs, int nrows, int ncols, int sr,
                                     const float* __restrict__ sigma, float lam2, float dthresh,
                                     float* __restrict__ wout, const float* __restrict__ coff) {
    __shared__ float W[64];
    __shared__ float T;
    const int wn = 2 * sr + 1, winsz = wn * wn;
    const int64_t b = blockIdx.x;
    // edge index -> pixel
    int y, x;
    const int64_t top = (int64_t)sr * ncols;
    if (b < 2 * top) {
        const int64_t r = b / ncols;
        y = (int)(r < sr ? r : nrows - 2 * sr + r);
        x = (int)(b - r * ncols);
    } else {
        const int64_t m = b - 2 * top;
        y = sr + (int)(m / (2 * sr));
        const int e = (int)(m - (int64_t)(y - sr) * 2 * sr);
        x = e < sr ? e : ncols - 2 * sr + e;
    }
    int ys, ye, xs, xe;
    window(y, sr, nrows, ys, ye);
    window(x, sr, ncols, xs, xe);
    const int64_t pix = (int64_t)y * ncols + x;
    const int c = threadIdx.x;
    if (c < winsz) {
        const int64_t nb = (int64_t)(ys + c / wn) * ncols + (xs + c % wn);
        float w;
        if (nb == pix) {
            w = -1.0e6f;
        } else {
            const int dy = ys + c / wn - y, dx = xs + c % wn - x, nF = fwd_count(sr);
            const float2 e2 = dy < -sr || dy > sr || dx < -sr || dx > sr ? raw[b * winsz + c]
                              : (dy > 0 || (dy == 0 && dx > 0)) ? pairs[pix * nF + fwd_index(dy, dx, sr)]
                                                               : pairs[nb * nF + fwd_index(-dy, -dx, sr)];
            float s0 = sigma[pix], s1 = sigma[nb];
            s0 = __fmul_rn(s0, s0);
            s1 = __fmul_rn(s1, s1);
            const float ss = __fadd_rn(s0, s1);
            const float d2 = __fsub_rn(e2.x, __fmul_rn(e2.y, ss));
            const float dnorm = __fmul_rn(ss, sqrtf(__fmul_rn(2.0f, e2.y)));
            w = dnorm > 1.e-8f ? __fdiv_rn(d2, dnorm) : __fmul_rn(1e6f, e2.y);
        }
        w = fmaxf(__fsub_rn(w, dthresh), 0.0f);
        w = expf(__fmul_rn(__fmul_rn(-1.0f, w), lam2));
        if (coff && nb == pix) w = __fadd_rn(w, coff[pix]);  // diff_offset's centre addition
        W[c] = w;
    }
    __syncthreads();
    if (c == 0) {
        float t = 0.0f;
        for (int k = 0; k < winsz; ++k) t = __fadd_rn(t, W[k]);
        T = t;
    }
    __syncthreads();
    if (c < winsz) wout[pix * winsz + c] = __fdiv_rn(W[c], T);
}

size_t pairs_smem(int sr) {
    return std::max((size_t)2 * (sr + 1) * kChunk * kPairPitch, (size_t)2 * (64 + 4 * sr) * kEdgePitch) * sizeof(float);
}

// The pair sums of the scan, with sigma's own when asked, and the edge pixels' other window sums.
int launch_pairs(cudaStream_t st, const float* data, int nrows, int ncols, int npx, const int32_t* ind, int nind,
                 float datamax, int saturation_protect, int sr, bool with_sigma, float2* pairs, float2* sigp, float2* raw) {
    const float mxval = saturation_protect ? datamax * 0.999f : datamax + 1.0f;
    const float mxsig = saturation_protect ? datamax * 0.9961f : datamax + 1.0f;
    const int edge_rows = edge_blocks(sr, ncols), edge_all = edge_rows + edge_blocks(sr, nrows);
    const int64_t pgrid = edge_all + (int64_t)((ncols + 2 * kPairLanes - 1) / (2 * kPairLanes)) * nrows;
    if (pgrid > 0x7fffffff) return EBSD_E_UNSUPPORTED;
    typedef void (*PairsFn)(const float*, int, int, int, const int32_t*, int, float, float, float, float2*, float2*, int, int,
                            float2*);
    PairsFn fn = with_sigma ? (sr == 1 ? k_nlpar_pairs<1, true> : sr == 2 ? k_nlpar_pairs<2, true> : k_nlpar_pairs<3, true>)
                            : (sr == 1 ? k_nlpar_pairs<1, false> : sr == 2 ? k_nlpar_pairs<2, false> : k_nlpar_pairs<3, false>);
    const size_t psm = pairs_smem(sr);
    EBSD_CUDA_TRY(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psm));
    fn<<<(unsigned)pgrid, (unsigned)kPairThreads, psm, st>>>(data, nrows, ncols, npx, ind, nind, mxval, mxsig, 0.0f, pairs,
                                                             sigp, edge_rows, edge_all, raw);
    return launch_status();
}

// ---- the weights with the pieces of their derivative, from the pair sums ----------------------
// 1024 pixels of 14400 values, radius 2: k_sigma_arg and k_nlpar_weights_d, which sum every pair once
// for each of its pixels and slots with a serial, uncoalesced pair_ssd, took 1010 + 1165 us; the pair
// kernel (648, its 32 blocks' serial chains) and these two (6 + 6) take their place at radius 1-3.
// sigma^2 with the neighbour that attains the minimum and its pair count: k_sigma_arg's scan of the
// eight neighbours in raster order, the sums read instead of made.
__global__ void k_nlpar_sigma_arg_pairs(const float2* __restrict__ sigp, int nrows, int ncols, float* __restrict__ sig2,
                                        int* __restrict__ arg, float* __restrict__ nsig) {
    const int64_t pix = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= (int64_t)nrows * ncols) return;
    const int j = (int)(pix / ncols), i = (int)(pix - (int64_t)j * ncols);
    float best = 1e24f, bn = 0.0f;
    int ba = -1;
    for (int kk = 0; kk < 9; ++kk) {
        const int dy = kk / 3 - 1, dx = kk % 3 - 1, jn = j + dy, inn = i + dx;
        if (kk == 4 || jn < 0 || jn >= nrows || inn < 0 || inn >= ncols) continue;
        const int64_t nb = (int64_t)jn * ncols + inn;
        // forward neighbours: dx 1 in the same row; dx -1, 0, 1 in the next
        const float2 e = kk > 4 ? sigp[pix * 4 + (kk == 5 ? 0 : 2 + dx)] : sigp[nb * 4 + (kk == 3 ? 0 : 2 - dx)];
        const float n2 = __fadd_rn(e.y, 1.0e-12f);
        if (!(e.x >= 1.e-3f)) continue;
        const float v = __fdiv_rn(e.x, __fmul_rn(n2, 2.0f));
        if (v < best) { best = v; ba = (int)nb; bn = n2; }
    }
    const float sg = sqrtf(best);
    sig2[pix] = __fmul_rn(sg, sg);
    arg[pix] = ba;
    nsig[pix] = bn;
}

// k_nlpar_weights_d's arithmetic, one block (64 threads) per scan pixel, a thread per window slot.
__global__ void k_nlpar_weights_d_pairs(const float2* __restrict__ pairs, const float2* __restrict__ raw, int nrows,
                                        int ncols, int sr, const float* __restrict__ sig2, float lam2, float dthresh,
                                        float* __restrict__ wout, float* __restrict__ mout, float* __restrict__ dsout,
                                        float* __restrict__ dgout) {
    __shared__ float W[64];
    __shared__ float T;
    const int wn = 2 * sr + 1, winsz = wn * wn, nF = fwd_count(sr), c = threadIdx.x;
    const int64_t pix = blockIdx.x;
    const int y = (int)(pix / ncols), x = (int)(pix - (int64_t)y * ncols);
    int ys, ye, xs, xe;
    window(y, sr, nrows, ys, ye);
    window(x, sr, ncols, xs, xe);
    float m = 0.0f, dS = 0.0f, dg = 0.0f;
    if (c < winsz) {
        const int dy = ys + c / wn - y, dx = xs + c % wn - x;
        const int64_t nb = pix + (int64_t)dy * ncols + dx;
        float w = -1.0e6f;
        if (nb != pix) {
            const float2 e = dy < -sr || dy > sr || dx < -sr || dx > sr ? raw[edge_index(y, x, sr, nrows, ncols) * winsz + c]
                             : (dy > 0 || (dy == 0 && dx > 0)) ? pairs[pix * nF + fwd_index(dy, dx, sr)]
                                                              : pairs[nb * nF + fwd_index(-dy, -dx, sr)];
            const float ss = __fadd_rn(sig2[pix], sig2[nb]);
            const float d2 = __fsub_rn(e.x, __fmul_rn(e.y, ss));
            const float dnorm = __fmul_rn(ss, sqrtf(__fmul_rn(2.0f, e.y)));
            if (dnorm > 1.e-8f) {
                w = __fdiv_rn(d2, dnorm);
                dS = 1.0f / dnorm;
                dg = -e.x / (ss * dnorm);
            } else {
                w = __fmul_rn(1e6f, e.y);
            }
        }
        m = fmaxf(__fsub_rn(w, dthresh), 0.0f);
        if (!(w - dthresh > 0.0f)) { dS = 0.0f; dg = 0.0f; }  // clamped: no derivative
        W[c] = expf(__fmul_rn(__fmul_rn(-1.0f, m), lam2));
    }
    __syncthreads();
    if (c == 0) {
        float t = 0.0f;
        for (int k = 0; k < winsz; ++k) t = __fadd_rn(t, W[k]);
        T = t;
    }
    __syncthreads();
    if (c < winsz) {
        const int64_t o = pix * winsz + c;
        wout[o] = __fdiv_rn(W[c], T);
        mout[o] = m;
        dsout[o] = dS;
        dgout[o] = dg;
    }
}

size_t tiled_smem(int sr, int ncols, size_t elem, bool weights) {
    const int wn = 2 * sr + 1;
    const int ncx = std::min(ncols, kTileX + 4 * sr);
    // staged rows (rounded up to 4 elements), then the pixels' weights at rows of winsz
    // rounded up to 4
    size_t b = (((size_t)wn * ncx * kSP + 3) & ~(size_t)3) * elem + (size_t)kTileX * ((wn * wn + 3) & ~3) * elem;
    if (weights) b += kTileX * sizeof(float);
    return b;
}


// ---- lambda optimisation (NLPAR.opt_lambda_cpu, nlpar_cpu.py:94-155) -------------------
// calcsigma_cpu (nlpar_cpu.py:157-264) runs sigma_numba per scan tile with nn and the tile's
// start/count arrays as uint64, so `j - nn` wraps for the tile's first row and first column:
// those pixels get an empty window (sigma sqrt(1e24), no distances).  Every other pixel gets
// its clipped 3x3 window in row-major slot order (centre: count = pattern length, distance 0);
// the distances are normalised with the tile's own sigma (nlpar_cpu.py:805-817), then merged
// into the scan: sigma = min over tiles, a slot's distance and count replaced where the tile's
// count is positive.

__device__ __forceinline__ uint32_t fmax_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fmax_unkey(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// largest value of the tile's patterns (np.max(data) of the tile)
__global__ void k_tile_max(const float* __restrict__ data, int ncols, int npx, int r0, int c0, int tr, int tc,
                           uint32_t* __restrict__ key) {
    const int64_t total = (int64_t)tr * tc * npx;
    float m = -INFINITY;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t pix = t / npx;
        const int q = (int)(t - pix * npx);
        const int j = (int)(pix / tc), i = (int)(pix - (int64_t)j * tc);
        m = fmaxf(m, __ldg(data + ((int64_t)(r0 + j) * ncols + (c0 + i)) * npx + q));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(key, fmax_key(m));
}

// raw distances and counts per slot, and the tile sigma; 8 lanes per pixel (the neighbours)
__global__ void k_tile_dist(const float* __restrict__ data, int ncols, int npx, int r0, int c0, int tr, int tc,
                            const int32_t* __restrict__ ind, int nind, int satp, const uint32_t* __restrict__ key,
                            float* __restrict__ sig_t, float* __restrict__ d2_t, float* __restrict__ n2_t) {
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int pix = gt >> 3, lane8 = gt & 7;
    const float m = fmax_unkey(*key);
    const float mxval = satp ? __fmul_rn(m, 0.9961f) : __fadd_rn(m, 1.0f);
    float s0 = 1e24f;
    if (pix < tr * tc) {
        const int j = pix / tc, i = pix - (pix / tc) * tc;
        if (j >= 1 && i >= 1) {  // the first row and column of a tile have empty windows
            const int cstart = i - 1, cend = min(i + 1, tc - 1) + 1, width = cend - cstart;
            const int k = lane8 < 4 ? lane8 : lane8 + 1;
            const int jn = j + k / 3 - 1, inn = i + k % 3 - 1;
            if (lane8 == 0) {
                const int cslot = width + 1;  // (j - rstart) * width + (i - cstart)
                n2_t[(int64_t)pix * 9 + cslot] = (float)npx;
                d2_t[(int64_t)pix * 9 + cslot] = 0.0f;
            }
            if (jn < tr && inn < tc) {
                const int slot = (jn - (j - 1)) * width + (inn - cstart);
                float d2, n2;
                pair_ssd(data + ((int64_t)(r0 + j) * ncols + (c0 + i)) * npx,
                         data + ((int64_t)(r0 + jn) * ncols + (c0 + inn)) * npx, ind, nind, mxval, 1.0e-12f, d2, n2);
                n2_t[(int64_t)pix * 9 + slot] = n2;
                d2_t[(int64_t)pix * 9 + slot] = d2;
                if (d2 >= 1.e-3f) s0 = __fdiv_rn(d2, __fmul_rn(n2, 2.0f));
            }
        }
    }
    for (int o = 4; o > 0; o >>= 1) s0 = fminf(s0, __shfl_down_sync(0xffffffffu, s0, o, 8));
    if (lane8 == 0 && pix < tr * tc) sig_t[pix] = __fsqrt_rn(s0);
}

// normalise with the tile sigma and merge into the scan arrays (one thread per pixel and slot)
__global__ void k_tile_merge(int ncols, int r0, int c0, int tr, int tc, const float* __restrict__ sig_t,
                             const float* __restrict__ d2_t, const float* __restrict__ n2_t,
                             float* __restrict__ sigma, float* __restrict__ d2, float* __restrict__ n2) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)tr * tc * 9) return;
    const int pix = (int)(t / 9), q = (int)(t - (int64_t)pix * 9);
    const int j = pix / tc, i = pix - (pix / tc) * tc;
    const int64_t g = (int64_t)(r0 + j) * ncols + (c0 + i);
    if (q == 0) sigma[g] = fminf(sigma[g], sig_t[pix]);
    const float n = n2_t[t];
    if (n > 0.0f) {
        const int cstart = i - 1, cend = min(i + 1, tc - 1) + 1, width = cend - cstart;
        const int jj = j - 1 + q / width, ii = cstart + q % width;
        const float sa = sig_t[pix], sb = sig_t[jj * tc + ii];
        const float s12 = __fadd_rn(__fmul_rn(sa, sa), __fmul_rn(sb, sb));
        float v = __fsub_rn(d2_t[t], __fmul_rn(n, s12));
        v = __fdiv_rn(v, __fmul_rn(s12, __fsqrt_rn(__fmul_rn(2.0f, n))));
        d2[g * 9 + q] = v;
        n2[g * 9 + q] = n;
    }
}

// the objective mean |tw - 1 / (sum_q exp(-max(d2, dthresh) / lam^2) + 1e-12)| over the pixels
// (rows and columns stepped by `stride`), float64; per-block sums, then one block in order
constexpr int kLamBlocks = 256;

__global__ void k_lam_partial(const float* __restrict__ d2, int nrows, int ncols, int stride, float dthresh,
                              double lam2, double tw, double* __restrict__ part) {
    __shared__ double red[256];
    const int sr = (nrows + stride - 1) / stride, sc = (ncols + stride - 1) / stride;
    const int64_t total = (int64_t)sr * sc;
    double acc = 0.0;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int a = (int)(t / sc), b = (int)(t - (int64_t)a * sc);
        const float* v = d2 + ((int64_t)(a * stride) * ncols + b * stride) * 9;
        double e[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const float m = fmaxf(v[q], dthresh);  // np.maximum (no NaN in the distances)
            e[q] = exp(__ddiv_rn((double)(-m), lam2));
        }
        // numpy's pairwise order for nine terms
        double w = __dadd_rn(__dadd_rn(__dadd_rn(e[0], e[1]), __dadd_rn(e[2], e[3])),
                             __dadd_rn(__dadd_rn(e[4], e[5]), __dadd_rn(e[6], e[7])));
        w = __dadd_rn(__dadd_rn(w, e[8]), 1e-12);
        acc = __dadd_rn(acc, fabs(__dsub_rn(tw, __ddiv_rn(1.0, w))));
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] = __dadd_rn(red[threadIdx.x], red[threadIdx.x + o]);
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void k_lam_final(const double* __restrict__ part, int nparts, double count, double* __restrict__ out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double s = 0.0;
        for (int b = 0; b < nparts; ++b) s = __dadd_rn(s, part[b]);
        *out = __ddiv_rn(s, count);
    }
}

}  // namespace
}  // namespace ebsd

using namespace ebsd;

extern "C" {

int ebsd_nlpar_sigma(const float* d_data, int32_t nrows, int32_t ncols, int32_t npx, const int32_t* d_indices,
                     int32_t nind, float datamax, int saturation_protect, float* d_sigma, void* stream) {
    if (!d_data || !d_indices || !d_sigma || nrows <= 0 || ncols <= 0 || npx <= 0 || nind < 0 || nind > npx)
        return EBSD_E_ARG;
    float mxval = saturation_protect ? datamax * 0.9961f : datamax + 1.0f;
    int64_t threads = (int64_t)nrows * ncols * 8;
    k_nlpar_sigma<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        d_data, nrows, ncols, npx, d_indices, nind, mxval, d_sigma);
    return launch_status();
}

int ebsd_nlpar_sigma_tile(const float* d_data, int32_t nrows, int32_t ncols, int32_t npx, int32_t r0, int32_t r1,
                          int32_t c0, int32_t c1, const int32_t* d_indices, int32_t nind, int saturation_protect,
                          float* d_sigma, float* d_d2, float* d_n2, float* d_work, void* stream) {
    if (!d_data || !d_indices || !d_sigma || !d_d2 || !d_n2 || !d_work || nrows <= 0 || ncols <= 0 || npx <= 0 ||
        nind < 0 || nind > npx)
        return EBSD_E_ARG;
    if (r0 < 0 || c0 < 0 || r1 > nrows || c1 > ncols || r1 <= r0 || c1 <= c0) return EBSD_E_ARG;
    const int tr = r1 - r0, tc = c1 - c0;
    const int64_t tp = (int64_t)tr * tc;
    cudaStream_t st = (cudaStream_t)stream;
    float* sig_t = d_work;
    float* d2_t = sig_t + tp;
    float* n2_t = d2_t + tp * 9;
    uint32_t* key = (uint32_t*)(n2_t + tp * 9);
    EBSD_CUDA_TRY(cudaMemsetAsync(d2_t, 0, (size_t)tp * 18 * sizeof(float) + sizeof(uint32_t), st));
    const int64_t elems = tp * npx;
    const int mb = (int)std::min<int64_t>((elems + 255) / 256, 152 * 8);
    k_tile_max<<<mb, 256, 0, st>>>(d_data, ncols, npx, r0, c0, tr, tc, key);
    int rc = launch_status();
    if (rc != EBSD_OK) return rc;
    const int64_t th = tp * 8;
    k_tile_dist<<<(unsigned)((th + 255) / 256), 256, 0, st>>>(d_data, ncols, npx, r0, c0, tr, tc, d_indices, nind,
                                                             saturation_protect, key, sig_t, d2_t, n2_t);
    rc = launch_status();
    if (rc != EBSD_OK) return rc;
    const int64_t tm = tp * 9;
    k_tile_merge<<<(unsigned)((tm + 255) / 256), 256, 0, st>>>(ncols, r0, c0, tr, tc, sig_t, d2_t, n2_t, d_sigma,
                                                              d_d2, d_n2);
    return launch_status();
}

int ebsd_nlpar_lambda_metric(const float* d_d2, int32_t nrows, int32_t ncols, int32_t stride, float dthresh,
                             double lam, double tw, double* d_work, double* d_out, void* stream) {
    if (!d_d2 || !d_work || !d_out || nrows <= 0 || ncols <= 0 || stride < 1) return EBSD_E_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t sr = (nrows + stride - 1) / stride, sc = (ncols + stride - 1) / stride;
    k_lam_partial<<<kLamBlocks, 256, 0, st>>>(d_d2, nrows, ncols, stride, dthresh, lam * lam, tw, d_work);
    int rc = launch_status();
    if (rc != EBSD_OK) return rc;
    k_lam_final<<<1, 32, 0, st>>>(d_work, kLamBlocks, (double)(sr * sc), d_out);
    return launch_status();
}

int ebsd_nlpar(const float* d_data, int32_t nrows, int32_t ncols, int32_t npx, const int32_t* d_indices,
               int32_t nind, float datamax, float lam, int32_t sr, float dthresh, const float* d_sigma,
               int saturation_protect, float* d_work, float* d_out, void* stream) {
    return ebsd_nlpar_out(d_data, nrows, ncols, npx, d_indices, nind, datamax, lam, sr, dthresh, d_sigma,
                          saturation_protect, d_work, EBSD_F32, d_out, nullptr, stream);
}

int ebsd_nlpar_out(const float* d_data, int32_t nrows, int32_t ncols, int32_t npx, const int32_t* d_indices,
                   int32_t nind, float datamax, float lam, int32_t sr, float dthresh, const float* d_sigma,
                   int saturation_protect, float* d_work, int out_dtype, void* d_out,
                   const float* d_centre_offset, void* stream) {
    if (out_dtype != EBSD_F32 && out_dtype != EBSD_U8 && out_dtype != EBSD_U16) return EBSD_E_DTYPE;
    if (!d_data || !d_indices || !d_sigma || !d_work || !d_out || nrows <= 0 || ncols <= 0 || npx <= 0 ||
        nind < 0 || nind > npx || sr < 0 || sr > 10 || !(lam > 0.0f))
        return EBSD_E_ARG;
    if (2 * sr + 1 > nrows || 2 * sr + 1 > ncols) return EBSD_E_ARG;  // window must fit the scan
    float mxval = saturation_protect ? datamax * 0.999f : datamax + 1.0f;
    float lam2 = 1.0f / (lam * lam);
    int winsz = (2 * sr + 1) * (2 * sr + 1);
    int bs = ((winsz + 31) / 32) * 32;
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 tgrid((unsigned)((ncols + kTileX - 1) / kTileX), (unsigned)nrows), tblock(kTileX, kTy);
    const size_t wsm = tiled_smem(sr, ncols, sizeof(float), true), asm_ = tiled_smem(sr, ncols, sizeof(float), false);
    if (sr <= 3 && wsm <= 48 * 1024 && asm_ <= 48 * 1024) {
        k_nlpar_weights_tiled<4><<<tgrid, tblock, wsm, st>>>(d_data, nrows, ncols, npx, d_indices, nind, mxval,
                                                             d_sigma, lam2, dthresh, sr, d_work, d_centre_offset);
        int rc = launch_status();
        if (rc != EBSD_OK) return rc;
        if (out_dtype == EBSD_U8)
            launch_average_tiled<float, uint8_t>(tgrid, tblock, asm_, st, d_data, nrows, ncols, npx, d_work, sr,
                                                 (uint8_t*)d_out);
        else if (out_dtype == EBSD_U16)
            launch_average_tiled<float, uint16_t>(tgrid, tblock, asm_, st, d_data, nrows, ncols, npx, d_work, sr,
                                                  (uint16_t*)d_out);
        else
            launch_average_tiled<float, float>(tgrid, tblock, asm_, st, d_data, nrows, ncols, npx, d_work, sr,
                                               (float*)d_out);
        return launch_status();
    }
    k_nlpar_weights<<<(unsigned)(nrows * ncols), bs, winsz * sizeof(float), st>>>(
        d_data, nrows, ncols, npx, d_indices, nind, mxval, d_sigma, lam2, dthresh, sr, d_work, d_centre_offset);
    int rc = launch_status();
    if (rc != EBSD_OK) return rc;
    dim3 grid((unsigned)((npx + 255) / 256), (unsigned)(nrows * ncols));
    if (out_dtype == EBSD_U8)
        k_nlpar_average_to<uint8_t><<<grid, 256, 0, st>>>(d_data, nrows, ncols, npx, d_work, sr, (uint8_t*)d_out);
    else if (out_dtype == EBSD_U16)
        k_nlpar_average_to<uint16_t><<<grid, 256, 0, st>>>(d_data, nrows, ncols, npx, d_work, sr, (uint16_t*)d_out);
    else
        k_nlpar_average<float><<<grid, 256, 0, st>>>(d_data, nrows, ncols, npx, d_work, sr, (float*)d_out);
    return launch_status();
}

int ebsd_nlpar_pairs_out(const float* d_data, int32_t nrows, int32_t ncols, int32_t npx, const int32_t* d_indices,
                         int32_t nind, float datamax, float lam, int32_t sr, float dthresh, float* d_sigma,
                         int compute_sigma, int saturation_protect, float* d_work, int out_dtype, void* d_out,
                         const float* d_centre_offset, void* stream) {
    if (out_dtype != EBSD_F32 && out_dtype != EBSD_U8 && out_dtype != EBSD_U16) return EBSD_E_DTYPE;
    if (!d_data || !d_indices || !d_sigma || !d_work || !d_out || nrows <= 0 || ncols <= 0 || npx <= 0 ||
        nind < 0 || nind > npx || sr < 1 || sr > 3 || !(lam > 0.0f))
        return EBSD_E_ARG;
    if (2 * sr + 1 > nrows || 2 * sr + 1 > ncols) return EBSD_E_ARG;  // window must fit the scan
    const size_t asm_ = tiled_smem(sr, ncols, sizeof(float), false);
    if (asm_ > 48 * 1024) return EBSD_E_UNSUPPORTED;
    const float lam2 = 1.0f / (lam * lam);
    const int64_t npix = (int64_t)nrows * ncols;
    const int winsz = (2 * sr + 1) * (2 * sr + 1), nF = sr * (2 * sr + 1) + sr;
    float* w = d_work;
    // the pair sums start at the next even float after the weights (8-byte aligned float2;
    // d_work itself is at least 8-byte aligned)
    if ((uintptr_t)d_work % 8 != 0) return EBSD_E_ARG;
    float2* pairs = (float2*)(d_work + ((npix * winsz + 1) & ~(int64_t)1));
    float2* sigp = pairs + npix * nF;
    cudaStream_t st = (cudaStream_t)stream;
    float2* raw = sigp + npix * 4;  // the edge pixels' window sums that are no pair sums
    int rc = launch_pairs(st, d_data, nrows, ncols, npx, d_indices, nind, datamax, saturation_protect, sr, compute_sigma != 0,
                          pairs, sigp, raw);
    if (rc != EBSD_OK) return rc;
    if (compute_sigma) {
        k_nlpar_sigma_pairs<<<(unsigned)((npix + 255) / 256), 256, 0, st>>>(sigp, nrows, ncols, d_sigma);
        if ((rc = launch_status()) != EBSD_OK) return rc;
    }
    const dim3 tgrid((unsigned)((ncols + kTileX - 1) / kTileX), (unsigned)nrows), tblock(kTileX, kTy);
    k_nlpar_weights_pairs<4><<<tgrid, tblock, 0, st>>>(nrows, ncols, pairs, d_sigma, lam2, dthresh, sr, w,
                                                       d_centre_offset);
    if ((rc = launch_status()) != EBSD_OK) return rc;
    {
        // edge pixels: their weights
        const int nri = nrows - 2 * sr;
        const int64_t nedge = (int64_t)2 * sr * ncols + (int64_t)nri * 2 * sr;
        k_nlpar_weights_edge<<<(unsigned)nedge, 64, 0, st>>>(raw, pairs, nrows, ncols, sr, d_sigma, lam2, dthresh, w,
                                                             d_centre_offset);
        if ((rc = launch_status()) != EBSD_OK) return rc;
    }
    if (out_dtype == EBSD_U8)
        launch_average<uint8_t>(tgrid, tblock, asm_, st, d_data, nrows, ncols, npx, w, sr, (uint8_t*)d_out);
    else if (out_dtype == EBSD_U16)
        launch_average<uint16_t>(tgrid, tblock, asm_, st, d_data, nrows, ncols, npx, w, sr, (uint16_t*)d_out);
    else
        launch_average<float>(tgrid, tblock, asm_, st, d_data, nrows, ncols, npx, w, sr, (float*)d_out);
    return launch_status();
}

int64_t ebsd_nlpar_sigma_weights_d_work(int32_t nrows, int32_t ncols, int32_t sr) {
    if (nrows <= 0 || ncols <= 0 || sr < 1 || sr > 3 || 2 * sr + 1 > nrows || 2 * sr + 1 > ncols) return 0;
    const int64_t npix = (int64_t)nrows * ncols, nedge = (int64_t)2 * sr * (ncols + nrows - 2 * sr);
    return 2 * (npix * (sr * (2 * sr + 1) + sr + 4) + nedge * (2 * sr + 1) * (2 * sr + 1));
}

int ebsd_nlpar_sigma_weights_d(const float* d_data, int32_t nrows, int32_t ncols, int32_t npx, const int32_t* d_indices,
                               int32_t nind, float datamax, float lam, int32_t sr, float dthresh, int compute_sigma,
                               int saturation_protect, float* d_work, float* d_sig2, int32_t* d_arg, float* d_nsig,
                               float* d_w, float* d_m, float* d_dS, float* d_dsig, void* stream) {
    if (!d_data || !d_indices || !d_work || (uintptr_t)d_work % 8 != 0 || !d_sig2 || !d_w || !d_m || !d_dS || !d_dsig ||
        (compute_sigma && (!d_arg || !d_nsig)) || nrows <= 0 || ncols <= 0 || npx <= 0 || nind < 0 || nind > npx || sr < 1 ||
        sr > 3 || !(lam > 0.0f) || 2 * sr + 1 > nrows || 2 * sr + 1 > ncols)
        return EBSD_E_ARG;
    const int64_t npix = (int64_t)nrows * ncols;
    if (npix > 0x7fffffff) return EBSD_E_ARG;
    float2* pairs = (float2*)d_work;
    float2* sigp = pairs + npix * (sr * (2 * sr + 1) + sr);
    float2* raw = sigp + npix * 4;
    cudaStream_t st = (cudaStream_t)stream;
    int rc = launch_pairs(st, d_data, nrows, ncols, npx, d_indices, nind, datamax, saturation_protect, sr, compute_sigma != 0,
                          pairs, sigp, raw);
    if (rc != EBSD_OK) return rc;
    if (compute_sigma) {
        k_nlpar_sigma_arg_pairs<<<(unsigned)((npix + 255) / 256), 256, 0, st>>>(sigp, nrows, ncols, d_sig2, d_arg, d_nsig);
        if ((rc = launch_status()) != EBSD_OK) return rc;
    }
    k_nlpar_weights_d_pairs<<<(unsigned)npix, 64, 0, st>>>(pairs, raw, nrows, ncols, sr, d_sig2, 1.0f / (lam * lam), dthresh,
                                                           d_w, d_m, d_dS, d_dsig);
    return launch_status();
}

int ebsd_nlpar_apply(const float* d_x, int32_t nrows, int32_t ncols, int32_t npx, const float* d_w, int32_t sr,
                     float* d_out, void* stream) {
    if (!d_x || !d_w || !d_out || nrows <= 0 || ncols <= 0 || npx <= 0 || sr < 0 || sr > 10 || 2 * sr + 1 > nrows ||
        2 * sr + 1 > ncols)
        return EBSD_E_ARG;
    const size_t asm_ = tiled_smem(sr, ncols, sizeof(float), false);
    if (asm_ <= 48 * 1024) {
        const dim3 tgrid((unsigned)((ncols + kTileX - 1) / kTileX), (unsigned)nrows), tblock(kTileX, kTy);
        launch_average<float>(tgrid, tblock, asm_, (cudaStream_t)stream, d_x, nrows, ncols, npx, d_w, sr, d_out);
        return launch_status();
    }
    dim3 grid((unsigned)((npx + 255) / 256), (unsigned)(nrows * ncols));
    k_nlpar_average<float><<<grid, 256, 0, (cudaStream_t)stream>>>(d_x, nrows, ncols, npx, d_w, sr, d_out);
    return launch_status();
}

int ebsd_nlpar_apply64(const double* d_x, int32_t nrows, int32_t ncols, int32_t npx, const double* d_w, int32_t sr,
                       double* d_out, void* stream) {
    if (!d_x || !d_w || !d_out || nrows <= 0 || ncols <= 0 || npx <= 0 || sr < 0 || sr > 10 || 2 * sr + 1 > nrows ||
        2 * sr + 1 > ncols)
        return EBSD_E_ARG;
    dim3 grid((unsigned)((npx + 255) / 256), (unsigned)(nrows * ncols));
    k_nlpar_average<double><<<grid, 256, 0, (cudaStream_t)stream>>>(d_x, nrows, ncols, npx, d_w, sr, d_out);
    return launch_status();
}

}  // extern "C"
