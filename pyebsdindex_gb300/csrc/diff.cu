// Adjoint kernels for the differentiable band-sharpness path.
//
// Linear stages are sparse operators held on the device in CSR form; each is applied by a
// gather (one thread per output row per pattern), so the adjoint needs no atomics:
//   Radon          R[ray][px] = 1/count(ray) for the ray's pixels  (radon_fast.py:281-310)
//   Radon adjoint  R^T: per pixel, the rays through it -- back-projection through the
//                  transposed lookup table
//   LoG            M = conv(kernel) o pad (band_detect.py:573-606) restricted to the interior;
//                  its transpose M^T is the correlation with the kernel folded back through
//                  the padding map
// NLPAR (nlpar_cpu.py:821-936) with weights W(lambda) held fixed in the patterns:
//   k_nlpar_weights2  normalised window weights w and exponent arguments m = max(d - dthresh, 0)
//   k_nlpar_apply_t   W^T g (gather over the windows that contain each scan pixel)
//   k_nlpar_lam_grad  dL/dlambda = sum_p sum_c dw_pc/dlambda (g_p . x_c),
//                     dw_pc/dlambda = w_pc (2 / lambda^3) (m_pc - sum_c' w_pc' m_pc')
#include "ebsd_internal.cuh"

#include <cstring>
#include <new>
#include <type_traits>

struct ebsd_linop_s {
    int device = 0;
    int64_t nrows = 0, ncols = 0, nnz = 0;
    int64_t* rowptr = nullptr;
    int32_t* col = nullptr;
    float* val = nullptr;
    double* val64 = nullptr;
    int2* ent = nullptr;     // (column, float value) of each nonzero
    int64_t width = 0;       // the rows' image width, or 0: where neighbouring rows lie
};

namespace ebsd {
namespace {

template <typename T>
__global__ void k_csr_gather(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                             const T* __restrict__ val, const T* __restrict__ x, T* __restrict__ y,
                             int64_t nrows, int64_t ncols) {
    int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t b = blockIdx.y;
    if (row >= nrows) return;
    const T* xb = x + b * ncols;
    T acc = (T)0;
    for (int64_t e = rowptr[row]; e < rowptr[row + 1]; ++e) acc = fma(val[e], xb[col[e]], acc);
    y[b * nrows + row] = acc;
}

// The same products with the patterns along the fast axis: x^T [ncols][ldx], y^T [nrows][ldy]
// hold pattern b in column b.  Each output adds its row's terms in CSR order with fused
// multiply-adds, as k_csr_gather, so the results are the same bit for bit.
//
// Rows that neighbour in the image they index (rays of near angle and offset, near pixels) meet
// the same columns at about the same place of their rows, so a block takes a tile of
// kCsrTileY x kCsrTileX rows of that image and its reads of x^T hit L1 instead of L2.  A warp takes a
// row and 32 NV patterns: a nonzero costs one 8-byte broadcast, and NV coalesced loads feed NV
// multiply-adds of independent chains, eight nonzeros in flight.  Bound by the L1's 128 bytes a cycle.
// 1024 patterns, 120x120 pixels, 180x180 rays: Radon 1260 us with a row a warp and 32 patterns, unrolled by
// four (16 TB/s, eight instructions a nonzero), 479 now; its adjoint 1235, 496 now; the LoG 450, 183 now.
// Two rows a warp, unrolled by two: 509, 566, 193, and half the warps where a batch is small (one
// pattern of 60x60: the adjoint 58 us, 21 now).
constexpr int kCsrTileY = 2, kCsrTileX = 4;

template <typename T> struct CsrEnt;
template <> struct CsrEnt<float> {
    const int2* e;
    __device__ __forceinline__ void get(int64_t i, int& c, float& v) const {
        const int2 t = __ldg(e + i);
        c = t.x;
        v = __int_as_float(t.y);
    }
};
template <> struct CsrEnt<double> {
    const int32_t* col;
    const double* val;
    __device__ __forceinline__ void get(int64_t i, int& c, double& v) const {
        c = __ldg(col + i);
        v = __ldg(val + i);
    }
};

template <typename T, int NV>
__global__ void __launch_bounds__(256) k_csr_gather_cols(const int64_t* __restrict__ rowptr, CsrEnt<T> ent,
                                                         const T* __restrict__ xT, int64_t ldx, T* __restrict__ yT,
                                                         int64_t ldy, int64_t nrows, int64_t width, int64_t n) {
    static_assert(kCsrTileY * kCsrTileX == 8, "eight warps a tile");
    const int64_t tx = (width + kCsrTileX - 1) / kCsrTileX, ty = blockIdx.x / tx;
    const int64_t gx = (blockIdx.x - ty * tx) * kCsrTileX + threadIdx.y % kCsrTileX;
    const int64_t gy = ty * kCsrTileY + threadIdx.y / kCsrTileX, row = gy * width + gx;
    if (gx >= width || row >= nrows) return;
    const int64_t b0 = (int64_t)blockIdx.y * (32 * NV) + threadIdx.x;
    const int64_t e0 = __ldg(rowptr + row);
    const int len = (int)(__ldg(rowptr + row + 1) - e0);
    // kWhole: every pattern of the block exists, so that a nonzero's loads differ by constants from
    // one address; else patterns past the last read column 0 and are not stored
    auto run = [&](auto whole) {
        constexpr bool kWhole = decltype(whole)::value;
        const T* xb = kWhole ? xT + b0 : xT;
        int64_t off[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) off[v] = kWhole ? 32 * v : (b0 + 32 * v < n ? b0 + 32 * v : 0);
        T acc[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] = (T)0;
#pragma unroll 8
        for (int t = 0; t < len; ++t) {
            int c;
            T a;
            ent.get(e0 + t, c, a);
            const T* xr = xb + (int64_t)c * ldx;
#pragma unroll
            for (int v = 0; v < NV; ++v) acc[v] = fma(a, __ldg(xr + off[v]), acc[v]);
        }
#pragma unroll
        for (int v = 0; v < NV; ++v)
            if (kWhole || b0 + 32 * v < n) yT[row * ldy + b0 + 32 * v] = acc[v];
    };
    if ((int64_t)(blockIdx.y + 1) * (32 * NV) <= n) run(std::true_type());
    else run(std::false_type());
}

// Patterns a warp: in float as many as the batch fills, up to 128 (1024 patterns of 120x120: 479 us with 128,
// 657 with 64, 1188 with 32; 64 of 60x60: 31, 16 and 25).  In double 32: the FP64 pipe bounds it, and wider
// warps only pad the batch (200 patterns of 60x60: 246 us, 279 with 64, 279 with 128).
template <typename T>
void launch_csr_cols(cudaStream_t st, const int64_t* rowptr, CsrEnt<T> ent, const T* xT, int64_t ldx, T* yT, int64_t ldy,
                     int64_t nrows, int64_t width, int64_t n) {
    const unsigned tiles = (unsigned)(((width + kCsrTileX - 1) / kCsrTileX) * ((nrows + width * kCsrTileY - 1) / (width * kCsrTileY)));
    auto go = [&](auto nv) {
        constexpr int NV = decltype(nv)::value;
        k_csr_gather_cols<T, NV><<<dim3(tiles, (unsigned)((n + 32 * NV - 1) / (32 * NV))), dim3(32, 8), 0, st>>>(
            rowptr, ent, xT, ldx, yT, ldy, nrows, width, n);
    };
    if (sizeof(T) == 8 || n <= 32) go(std::integral_constant<int, 1>());
    else if (n <= 64) go(std::integral_constant<int, sizeof(T) == 4 ? 2 : 1>());
    else go(std::integral_constant<int, sizeof(T) == 4 ? 4 : 1>());
}

__device__ __forceinline__ void window(int i, int sr, int n, int& start, int& end) {
    int a = i - sr > 0 ? i - sr : 0;
    int b = i + sr - (n - 1) > 0 ? i + sr - (n - 1) : 0;
    start = a - b;
    int c = i + sr < n - 1 ? i + sr : n - 1;
    int e = sr - i > 0 ? sr - i : 0;
    end = c + e + 1;
}

__device__ __forceinline__ void pair_ssd(const float* __restrict__ a, const float* __restrict__ b,
                                         const int32_t* __restrict__ ind, int nind, float mxval,
                                         float& d2, float& n2) {
    float d = 0.0f, n = 0.0f;
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

// Normalised weights w and exponent arguments m of every window slot (one block per pixel).
__global__ void k_nlpar_weights2(const float* __restrict__ data, int nrows, int ncols, int npx,
                                 const int32_t* __restrict__ ind, int nind, float mxval,
                                 const float* __restrict__ sigma, float lam2, float dthresh, int sr,
                                 float* __restrict__ wout, float* __restrict__ mout) {
    extern __shared__ float w_s[];
    __shared__ float tot_s;
    int pix = blockIdx.x;
    int j = pix / ncols, i = pix - (pix / ncols) * ncols;
    int xs, xe, ys, ye;
    window(i, sr, ncols, xs, xe);
    window(j, sr, nrows, ys, ye);
    int wx = xe - xs, winsz = (2 * sr + 1) * (2 * sr + 1);
    int c = threadIdx.x;
    float m = 0.0f;
    if (c < winsz) {
        int nb = (xs + c % wx) + ncols * (ys + c / wx);
        float w;
        if (nb == pix) {
            w = -1.0e6f;
        } else {
            float s0 = sigma[pix], s1 = sigma[nb];
            s0 = __fmul_rn(s0, s0);
            s1 = __fmul_rn(s1, s1);
            float d2, n2;
            pair_ssd(data + (int64_t)pix * npx, data + (int64_t)nb * npx, ind, nind, mxval, d2, n2);
            float ss = __fadd_rn(s0, s1);
            d2 = __fsub_rn(d2, __fmul_rn(n2, ss));
            float dnorm = __fmul_rn(ss, sqrtf(__fmul_rn(2.0f, n2)));
            w = dnorm > 1.e-8f ? __fdiv_rn(d2, dnorm) : __fmul_rn(1e6f, n2);
        }
        m = fmaxf(__fsub_rn(w, dthresh), 0.0f);
        w_s[c] = expf(__fmul_rn(__fmul_rn(-1.0f, m), lam2));
    }
    __syncthreads();
    if (c == 0) {
        float t = 0.0f;
        for (int k = 0; k < winsz; ++k) t = __fadd_rn(t, w_s[k]);
        tot_s = t;
    }
    __syncthreads();
    if (c < winsz) {
        wout[(int64_t)pix * winsz + c] = __fdiv_rn(w_s[c], tot_s);
        mout[(int64_t)pix * winsz + c] = m;
    }
}

// The list of the scan pixels p near q that `take(p, jp, ip)` accepts, in raster order, made by
// one warp: candidates within reach of q (|dj|, |di| <= reach, inside the grid), the accepted
// ones numbered by ballot from `base` on and handed to `put(index, p, jp, ip)`.  Returns the end.
template <typename Take, typename Put>
__device__ __forceinline__ int list_near(int q, int nrows, int ncols, int reach, int lane, int base, Take take, Put put) {
    const int jq = q / ncols, iq = q - (q / ncols) * ncols, w = 2 * reach + 1;
    for (int c0 = 0; c0 < w * w; c0 += 32) {
        const int c = c0 + lane, jp = jq + c / w - reach, ip = iq + c % w - reach;
        const int p = ip + ncols * jp;
        const bool ok = c < w * w && jp >= 0 && jp < nrows && ip >= 0 && ip < ncols && take(p, jp, ip);
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (ok) put(base + __popc(m & ((1u << lane) - 1u)), p, jp, ip);
        base += __popc(m);
    }
    return base;
}

// The window slot in which pixel (jp, ip) holds (jq, iq), or -1.
__device__ __forceinline__ int slot_of(int jp, int ip, int jq, int iq, int sr, int nrows, int ncols) {
    int xs, xe, ys, ye;
    window(ip, sr, ncols, xs, xe);
    window(jp, sr, nrows, ys, ye);
    return jq >= ys && jq < ye && iq >= xs && iq < xe ? (jq - ys) * (2 * sr + 1) + (iq - xs) : -1;
}

// out[q][k] = sum over scan pixels p whose window holds q of w[p][slot] * g[p][k].
// One scan pixel q per blockIdx.y: the windows that hold q (pixel p, slot c) are listed by the
// block's first warp in the scan order of the sum, then each thread adds w[p][c] g[p][k] over the
// list for four pattern values at once (four loads in flight a term: with one, their latency was
// the bound).  1024 pixels of 14400 values, radius 2: 364 us before, 115 now.
constexpr int kAtVals = 4;
template <typename T>
__global__ void __launch_bounds__(256) k_nlpar_apply_t(const T* __restrict__ g, int nrows, int ncols, int npx,
                                                       const T* __restrict__ w, int sr, T* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char atsm[];
    const int q = blockIdx.y;
    const int winsz = (2 * sr + 1) * (2 * sr + 1);
    const int maxt = (4 * sr + 1) * (4 * sr + 1);
    T* wt = (T*)atsm;                 // [maxt] weights
    int* pt = (int*)(wt + maxt);      // [maxt] pixels
    __shared__ int nterm;
    if (threadIdx.x < 32) {
        const int jq = q / ncols, iq = q - (q / ncols) * ncols;
        const int nt = list_near(
            q, nrows, ncols, 2 * sr, threadIdx.x, 0,
            [&](int, int jp, int ip) { return slot_of(jp, ip, jq, iq, sr, nrows, ncols) >= 0; },
            [&](int t, int p, int jp, int ip) {
                wt[t] = w[(int64_t)p * winsz + slot_of(jp, ip, jq, iq, sr, nrows, ncols)];
                pt[t] = p;
            });
        if (threadIdx.x == 0) nterm = nt;
    }
    __syncthreads();
    const int k0 = blockIdx.x * (blockDim.x * kAtVals) + threadIdx.x;
    if (k0 >= npx) return;
    const int nt = nterm;
    int64_t kk[kAtVals];
    T acc[kAtVals];
#pragma unroll
    for (int i = 0; i < kAtVals; ++i) {
        const int k = k0 + i * (int)blockDim.x;
        kk[i] = k < npx ? k : k0;
        acc[i] = (T)0;
    }
#pragma unroll 2
    for (int t = 0; t < nt; ++t) {
        const T* row = g + (int64_t)pt[t] * npx;
        const T c = wt[t];
#pragma unroll
        for (int i = 0; i < kAtVals; ++i) acc[i] = fma(c, __ldg(row + kk[i]), acc[i]);
    }
#pragma unroll
    for (int i = 0; i < kAtVals; ++i)
        if (k0 + i * (int)blockDim.x < npx) out[(int64_t)q * npx + kk[i]] = acc[i];
}

// Per scan pixel: sum_c dw_pc/dlambda * (g_p . x_c); block reduction over the pattern pixels.
template <typename T>
__global__ void k_nlpar_lam_grad(const T* __restrict__ g, const T* __restrict__ x, int nrows, int ncols, int npx,
                                 const float* __restrict__ w, const float* __restrict__ m, int sr, float lam,
                                 double* __restrict__ out) {
    __shared__ double red[32];
    int p = blockIdx.x;
    int jp = p / ncols, ip = p - (p / ncols) * ncols;
    int xs, xe, ys, ye;
    window(ip, sr, ncols, xs, xe);
    window(jp, sr, nrows, ys, ye);
    int wx = xe - xs, winsz = (2 * sr + 1) * (2 * sr + 1);
    const float* wp = w + (int64_t)p * winsz;
    const float* mp = m + (int64_t)p * winsz;
    double mbar = 0.0;
    for (int c = 0; c < winsz; ++c) mbar += (double)wp[c] * (double)mp[c];
    const double coef = 2.0 / ((double)lam * lam * lam);
    double acc = 0.0;
    const T* gp = g + (int64_t)p * npx;
    for (int k = threadIdx.x; k < npx; k += blockDim.x) {
        double gk = (double)gp[k], s = 0.0;
        for (int c = 0; c < winsz; ++c) {
            int nb = (xs + c % wx) + ncols * (ys + c / wx);
            s += (double)wp[c] * ((double)mp[c] - mbar) * (double)x[(int64_t)nb * npx + k];
        }
        acc += gk * s;
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        acc = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if (threadIdx.x == 0) out[p] = acc * coef;
    }
}

// ---- Gaussian background blur: one axis of a separable filter with reflect padding ----------
// Forward along `axis` (0: rows y, 1: columns x) of [n][H][W]:
//   out[o] = sum_{t=-r..r} taps[t + r] in[refl(o + t)],   refl(q) = -q (q < 0), 2(L-1) - q (q >= L)
// (torch's "reflect" padding followed by a correlation), and its adjoint
//   out[i] = sum_o sum_t taps[t + r] v[o] [refl(o + t) == i]
// as a gather: the direct terms o = i - t, the mirror of the low edge (o + t = -i, 1 <= i <= r)
// and of the high edge (o + t = 2(L-1) - i, L-1-r <= i <= L-2).  Requires r < L.  A thread per
// output: double values (the FP64 pipe bounds them however they are read), r < 3, longest lines.
template <typename T>
__global__ void k_blur1d(const T* __restrict__ in, T* __restrict__ out, int64_t total, int H, int W, int axis,
                         const T* __restrict__ taps, int r) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int64_t p = idx / ((int64_t)H * W);
    const int rem = (int)(idx - p * H * W), y = rem / W, x = rem - (rem / W) * W;
    const int L = axis == 0 ? H : W, o = axis == 0 ? y : x, stride = axis == 0 ? W : 1;
    const T* base = in + p * H * W + (axis == 0 ? x : y * W);
    T acc = (T)0;
    if (o >= r && o + r < L) {
        // the window lies inside the line: no reflection (the same taps in the same order)
        const T* b0 = base + (int64_t)(o - r) * stride;
        for (int t = 0; t <= 2 * r; ++t) acc = fma(__ldg(taps + t), __ldg(b0 + (int64_t)t * stride), acc);
    } else {
        for (int t = -r; t <= r; ++t) {
            int q = o + t;
            q = q < 0 ? -q : (q >= L ? 2 * (L - 1) - q : q);
            acc = fma(__ldg(taps + t + r), __ldg(base + (int64_t)q * stride), acc);
        }
    }
    out[idx] = acc;
}

template <typename T>
__global__ void k_blur1d_t(const T* __restrict__ v, T* __restrict__ out, int64_t total, int H, int W, int axis,
                           const T* __restrict__ taps, int r) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int64_t p = idx / ((int64_t)H * W);
    const int rem = (int)(idx - p * H * W), y = rem / W, x = rem - (rem / W) * W;
    const int L = axis == 0 ? H : W, i = axis == 0 ? y : x, stride = axis == 0 ? W : 1;
    const T* base = v + p * H * W + (axis == 0 ? x : y * W);
    T acc = (T)0;
    const int a0 = i - r > 0 ? i - r : 0, a1 = i + r < L - 1 ? i + r : L - 1;
    for (int o = a0; o <= a1; ++o) acc = fma(__ldg(taps + (i - o) + r), __ldg(base + (int64_t)o * stride), acc);
    if (i >= 1 && i <= r)
        for (int o = 0; o <= r - i; ++o) acc = fma(__ldg(taps + (-i - o) + r), __ldg(base + (int64_t)o * stride), acc);
    if (i <= L - 2 && i >= L - 1 - r)
        for (int o = 2 * (L - 1) - i - r; o <= L - 1; ++o)
            acc = fma(__ldg(taps + (2 * (L - 1) - i - o) + r), __ldg(base + (int64_t)o * stride), acc);
    out[idx] = acc;
}

// The same sums in the same order for float lines of moderate length (r >= 3): a block stages 32
// whole lines in shared memory, a warp takes kBlurR neighbouring outputs of the 32 lines (a lane
// per line, lines at a pitch of 33 floats: no bank conflicts along either axis), so each staged
// value read feeds kBlurR multiply-adds and sixteen taps come in four 16-byte broadcasts.
// Per output the positions ascend: the first and last kBlurR - 1 reach part of the outputs
// (triangles unrolled), those between reach all of them.  What bounds it is issue: of the ~12
// instructions a position costs 8 are the multiply-adds; the one-output-a-thread kernels above
// spend 21 a tap.  1024 120x120 patterns, r = 30, per pass: 643 / 452 us along y / x before,
// 74 / 88 now (the adjoint 384 / 526 before, 75 / 91 now).
constexpr int kBlurR = 8, kBlurWarps = 4, kBlurLines = 32, kBlurPitch = 33, kBlurPad = 20;

__host__ __device__ inline int blur_tap_off(int r) { return kBlurPad + ((4 - ((2 * r + 2 + kBlurPad) & 3)) & 3); }
__host__ __device__ inline int blur_tap_len(int r) { return (blur_tap_off(r) + 2 * r + 1 + kBlurPad + 3) & ~3; }
inline size_t blur_smem(int L, int axis, int r) {
    return ((size_t)L * kBlurPitch * (axis == 1 ? 2 : 1) + (size_t)blur_tap_len(r)) * sizeof(float);
}

// acc[j] += sum of taps[c0 + j - o + r] line[o] (kCorr false, the positions o inside the line) or
// of taps[o - c0 - j + r] line[refl(o)] (kCorr true), o ascending; tp holds the taps as the sum
// meets them (kCorr reversed), tp[t] with t = c0 + j - o + r falling as o rises.
template <bool kCorr, bool kRev>
__device__ __forceinline__ void blur_sum(float (&acc)[kBlurR], const float* __restrict__ line,
                                         const float* __restrict__ tp, int r, int c0, int L) {
    auto at = [&](int o, bool& ok) -> int {
        if (kCorr) {
            ok = true;
            o = o < 0 ? -o : o;
            return o >= L ? 2 * (L - 1) - o : o;
        }
        ok = (unsigned)o < (unsigned)L;
        return o;
    };
    const int base = c0 - r;
    if (kCorr || base + kBlurR - 2 >= 0) {
        float tq[kBlurR - 1];
#pragma unroll
        for (int i = 0; i < kBlurR - 1; ++i) tq[i] = tp[2 * r - i];
#pragma unroll
        for (int s = 0; s < kBlurR - 1; ++s) {
            bool ok;
            const int o = at(base + s, ok);
            if (ok) {
                const float v = line[o * kBlurPitch];
#pragma unroll
                for (int j = 0; j <= s; ++j) {
                    float& a = acc[kRev ? kBlurR - 1 - j : j];
                    a = fmaf(tq[s - j], v, a);
                }
            }
        }
    }
    const int m0 = base + kBlurR - 1, m1 = c0 + r;  // positions that reach all outputs: [m0, m1]
    for (int o0 = m0; o0 <= m1; o0 += kBlurR) {
        if (!kCorr && (o0 + kBlurR - 1 < 0 || o0 >= L)) continue;
        float t[2 * kBlurR];
        const float4* t4 = reinterpret_cast<const float4*>(tp + (c0 - o0 - (kBlurR - 1) + r));
#pragma unroll
        for (int i = 0; i < 2 * kBlurR / 4; ++i) {
            const float4 f = t4[i];
            t[4 * i] = f.x; t[4 * i + 1] = f.y; t[4 * i + 2] = f.z; t[4 * i + 3] = f.w;
        }
        if (o0 >= 0 && o0 + kBlurR <= L && o0 + kBlurR - 1 <= m1) {  // inside the line: one address
            const float* lp = line + o0 * kBlurPitch;
#pragma unroll
            for (int s = 0; s < kBlurR; ++s) {
                const float v = lp[s * kBlurPitch];
#pragma unroll
                for (int j = 0; j < kBlurR; ++j) {
                    float& a = acc[kRev ? kBlurR - 1 - j : j];
                    a = fmaf(t[kBlurR - 1 - s + j], v, a);
                }
            }
            continue;
        }
#pragma unroll
        for (int s = 0; s < kBlurR; ++s) {
            bool ok;
            const int o = at(o0 + s, ok);
            if (ok && o0 + s <= m1) {
                const float v = line[o * kBlurPitch];
#pragma unroll
                for (int j = 0; j < kBlurR; ++j) {
                    float& a = acc[kRev ? kBlurR - 1 - j : j];
                    a = fmaf(t[kBlurR - 1 - s + j], v, a);
                }
            }
        }
    }
    if (kCorr || m1 + 1 < L) {
        float tq[kBlurR - 1];
#pragma unroll
        for (int i = 0; i < kBlurR - 1; ++i) tq[i] = tp[i];
#pragma unroll
        for (int s = 0; s < kBlurR - 1; ++s) {
            bool ok;
            const int o = at(m1 + 1 + s, ok);
            if (ok) {
                const float v = line[o * kBlurPitch];
#pragma unroll
                for (int j = s + 1; j < kBlurR; ++j) {
                    float& a = acc[kRev ? kBlurR - 1 - j : j];
                    a = fmaf(tq[j - 1 - s], v, a);
                }
            }
        }
    }
}

template <int kAxis, bool kAdj>
__global__ void __launch_bounds__(32 * kBlurWarps) k_blur_lines(const float* __restrict__ in, float* __restrict__ out,
                                                                int64_t nlines, int H, int W,
                                                                const float* __restrict__ taps, int r) {
    extern __shared__ __align__(16) float blsm[];
    const int L = kAxis == 0 ? H : W, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tlen = blur_tap_len(r), toff = blur_tap_off(r);
    float* tile = blsm + tlen;
    float* otile = tile + L * kBlurPitch;   // along x only
    for (int i = threadIdx.x; i < tlen; i += 32 * kBlurWarps) {
        const int t = i - toff;
        blsm[i] = (unsigned)t <= 2u * r ? taps[kAdj ? t : 2 * r - t] : 0.0f;
    }
    const int64_t l0 = (int64_t)blockIdx.x * kBlurLines;
    const int nl = nlines - l0 < kBlurLines ? (int)(nlines - l0) : kBlurLines;
    int64_t cb = 0;   // along y: the lane's column
    if (kAxis == 0) {
        const int64_t l = l0 + (lane < nl ? lane : nl - 1), p = l / W;
        cb = p * H * W + (l - p * W);
        for (int q = warp; q < L; q += kBlurWarps) tile[q * kBlurPitch + lane] = __ldg(in + cb + (int64_t)q * W);
    } else {
        for (int row = warp; row < nl; row += kBlurWarps)
            for (int q = lane; q < L; q += 32) tile[q * kBlurPitch + row] = __ldg(in + (l0 + row) * L + q);
    }
    __syncthreads();
    const float* line = tile + (lane < nl ? lane : 0);
    const float* tp = blsm + toff;
    for (int g0 = warp * kBlurR; g0 < L; g0 += kBlurWarps * kBlurR) {
        // the last outputs of a ragged line: a group that ends with the line, some of them twice
        const int i0 = g0 + kBlurR <= L || L < kBlurR ? g0 : L - kBlurR;
        float acc[kBlurR];
#pragma unroll
        for (int j = 0; j < kBlurR; ++j) acc[j] = 0.0f;
        if (!kAdj) {
            if (L >= kBlurR) {
                blur_sum<true, false>(acc, line, tp, r, i0, L);
            } else {  // a line shorter than a group: output by output
                for (int j = 0; j < L - i0; ++j) {
                    float a = 0.0f;
                    for (int t = 0; t <= 2 * r; ++t) {
                        int o = i0 + j + t - r;
                        o = o < 0 ? -o : (o >= L ? 2 * (L - 1) - o : o);
                        a = fmaf(tp[2 * r - t], line[o * kBlurPitch], a);
                    }
#pragma unroll
                    for (int jj = 0; jj < kBlurR; ++jj) if (jj == j) acc[jj] = a;
                }
            }
        } else {
            blur_sum<false, false>(acc, line, tp, r, i0, L);
            if (i0 <= r) {  // the low edge's mirror images, output 0 not among them
                const float keep = acc[0];
                blur_sum<false, true>(acc, line, tp, r, -i0 - (kBlurR - 1), L);
                if (i0 == 0) acc[0] = keep;
            }
            if (i0 + kBlurR - 1 >= L - 1 - r) {  // the high edge's, without output L - 1
                float keep[kBlurR];
#pragma unroll
                for (int j = 0; j < kBlurR; ++j) keep[j] = acc[j];
                blur_sum<false, true>(acc, line, tp, r, 2 * (L - 1) - i0 - (kBlurR - 1), L);
#pragma unroll
                for (int j = 0; j < kBlurR; ++j) if (i0 + j == L - 1) acc[j] = keep[j];
            }
        }
#pragma unroll
        for (int j = 0; j < kBlurR; ++j) {
            if (i0 + j < L) {
                if (kAxis == 1) otile[(i0 + j) * kBlurPitch + lane] = acc[j];
                else if (lane < nl) out[cb + (int64_t)(i0 + j) * W] = acc[j];
            }
        }
    }
    if (kAxis == 1) {
        __syncthreads();
        for (int row = warp; row < nl; row += kBlurWarps)
            for (int q = lane; q < L; q += 32) out[(l0 + row) * L + q] = otile[q * kBlurPitch + row];
    }
}

// Whether the blocked kernel takes the call: three and more taps a side (the triangles need
// 2 r + 2 >= kBlurR), lines that leave two blocks an SM (<= 96 KB of shared memory), and blocks enough:
// with few of them each warp's chain of taps is all the time there is, and a thread per output fills
// the chip.  120x120, r = 30: 30 blocks 10.7 .. 14.4 us blocked, 8.3 .. 10.4 with a thread per output; 60
// blocks 11.5 .. 14.5 and 10.4 .. 16.5; 90 blocks 11.9 .. 14.4 and 14.4 .. 22.6.  Short filters need more:
// r = 3, 120 blocks 6.4 .. 10.3 and 8.0 .. 8.4, 180 blocks 7.2 .. 10.3 and 8.4 .. 10.4.
constexpr size_t kBlurSmemMax = 96 * 1024;
inline bool blur_blocked(int64_t n, int H, int W, int axis, int r) {
    const int64_t lines = axis == 0 ? n * W : n * H, blocks = (lines + kBlurLines - 1) / kBlurLines;
    return r >= (kBlurR - 2) / 2 && blur_smem(axis == 0 ? H : W, axis, r) <= kBlurSmemMax &&
           blocks >= (r < 12 ? 152 : 64) && blocks <= 0x7fffffff;
}

template <int kAxis, bool kAdj>
int launch_blur(const float* in, int64_t n, int H, int W, const float* taps, int r, float* out, cudaStream_t st) {
    const size_t sm = blur_smem(kAxis == 0 ? H : W, kAxis, r);
    if (sm > 48 * 1024 && cudaFuncSetAttribute(k_blur_lines<kAxis, kAdj>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kBlurSmemMax) != cudaSuccess)
        return launch_status();
    const int64_t lines = kAxis == 0 ? n * W : n * H;
    k_blur_lines<kAxis, kAdj><<<(unsigned)((lines + kBlurLines - 1) / kBlurLines), 32 * kBlurWarps, sm, st>>>(
        in, out, lines, H, W, taps, r);
    return launch_status();
}

// ---- soft-argmax band sharpness ------------------------------------------------------------
// Per pattern (one block): J_p = sum_i s_i c_i over the Radon-mask cells, s = softmax(c / tau),
// and dJ_p / dc_i = s_i (1 + (c_i - J_p) / tau) (zero off the mask).  Sums in float64.
//
// Float patterns take the exponentials in float of arguments formed in double, and round the
// gradient to float once.  What bounds the float kernel is the FP64 pipe, which issues a warp
// operation in sixteen cycles.  What can leave that pipe without a rounding has left it: the maximum is
// taken of the floats (a product with inv_tau > 0 keeps their order), a float widens by integer shifts, and
// the division by the exponentials' sum (1 <= sum <= ncm, a float over it far from underflow) is a
// product with its reciprocal and one correction, which gives the correctly rounded quotient
// (P. Markstein, IBM J. Res. Dev. 34(1), 1990).
// 1024 patterns of 180x180 cells: 1660 us before, 911 now, the same bits.  Arguments and gradient in pairs of
// floats took 473, but kept 45 bits of c / tau only, which shows in the gradient from c / tau = 2^24 on.

// (double)f by integer operations (a conversion instruction runs at the FP64 pipe's rate)
__device__ __forceinline__ double widen(float f) {
    const unsigned u = __float_as_uint(f), sign = u & 0x80000000u;
    unsigned m = u & 0x7fffffffu, bias = 0x38000000u;  // the exponent rebiased by 1023 - 127
    if (m - 0x00800000u >= 0x7f000000u) {
        if (m == 0) return __hiloint2double((int)sign, 0);
        if (m >= 0x7f800000u) {
            bias = 0x70000000u;                        // infinity, NaN
        } else {
            const int sh = __clz(m) - 8;               // subnormal: normalised
            m = (m << sh) & 0x7fffffu;
            bias = (unsigned)(897 - sh) << 20;
        }
    }
    return __hiloint2double((int)(sign | ((m >> 3) + bias)), (int)(m << 29));
}

__device__ __forceinline__ double wide(float f) { return widen(f); }
__device__ __forceinline__ double wide(double d) { return d; }

template <typename T>
__global__ void k_softargmax(const T* __restrict__ c, int64_t ncell, const int32_t* __restrict__ cells, int ncm,
                             double inv_tau, double* __restrict__ Jp, T* __restrict__ grad) {
    __shared__ double red[66];
    const int64_t p = blockIdx.x;
    const T* cp = c + p * ncell;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    T vx = (T)-INFINITY;
#pragma unroll 8
    for (int k = tid; k < ncm; k += blockDim.x) {
        const T v = cp[__ldg(cells + k)];
        vx = v > vx ? v : vx;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const T a = __shfl_down_sync(0xffffffffu, vx, o);
        vx = a > vx ? a : vx;
    }
    if (lane == 0) red[warp] = (double)vx;
    __syncthreads();
    if (tid == 0) {
        double m = red[0];
        for (int w = 1; w < nw; ++w) m = fmax(m, red[w]);
        red[64] = m * inv_tau;
    }
    __syncthreads();
    const double mx = red[64];
    auto expo = [&](double v) -> double {
        if (sizeof(T) == 4) return wide(expf((float)(v * inv_tau - mx)));
        return exp(v * inv_tau - mx);
    };
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
    for (int k = tid; k < ncm; k += blockDim.x) {
        const double v = wide(cp[__ldg(cells + k)]);
        const double e = expo(v);
        s0 += e;
        s1 += e * v;
    }
    for (int o = 16; o > 0; o >>= 1) {
        s0 += __shfl_down_sync(0xffffffffu, s0, o);
        s1 += __shfl_down_sync(0xffffffffu, s1, o);
    }
    __syncthreads();
    if (lane == 0) { red[warp] = s0; red[32 + warp] = s1; }
    __syncthreads();
    if (tid == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < nw; ++w) { a += red[w]; b += red[32 + w]; }
        red[64] = a;
        red[65] = b / a;
        Jp[p] = b / a;
    }
    __syncthreads();
    const double S0 = red[64], J = red[65], r = 1.0 / S0;
    T* gp = grad + p * ncell;
#pragma unroll 4
    for (int k = tid; k < ncm; k += blockDim.x) {
        const int cell = __ldg(cells + k);
        const double v = wide(cp[cell]), e = expo(v);
        double s = e / S0;
        if (sizeof(T) == 4) {                          // the same quotient, in a third of the division's operations
            const double q = e * r;
            s = fma(fma(-q, S0, e), r, q);
        }
        gp[cell] = (T)(s * (1.0 + (v - J) * inv_tau));
    }
}

// ---- NLPAR weights as functions of the patterns ----------------------------------------------
// sigma (nlpar_cpu.py:753-796, nn = 1) with the neighbour that attains the minimum and its pair
// count: sig2 = sigma^2 as the weights use it, arg = that neighbour (-1: none), nsig = its count.
__global__ void k_sigma_arg(const float* __restrict__ data, int nrows, int ncols, int npx,
                            const int32_t* __restrict__ ind, int nind, float mxval, float* __restrict__ sig2,
                            int* __restrict__ arg, float* __restrict__ nsig) {
    // eight lanes per scan pixel, one per neighbour of the 3x3 neighbourhood in raster order
    // (the centre skipped); each lane sums its pair in pair_ssd's order, then the pixel's first
    // lane takes the minimum in raster order (strict <, the first of equal values), as a
    // sequential scan of the eight pairs would
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int pix = t >> 3, slot = t & 7;
    const int npix = nrows * ncols;
    const int kk = slot < 4 ? slot : slot + 1;  // 3x3 index, the centre (4) skipped
    float s0 = 1e24f, n2 = 0.0f;
    int nb = -1;
    if (pix < npix) {
        const int j = pix / ncols, i = pix - (pix / ncols) * ncols;
        const int jn = j + kk / 3 - 1, inn = i + kk % 3 - 1;
        if (jn >= 0 && jn < nrows && inn >= 0 && inn < ncols) {
            nb = inn + ncols * jn;
            float d2;
            pair_ssd(data + (int64_t)pix * npx, data + (int64_t)nb * npx, ind, nind, mxval, d2, n2);
            n2 = __fadd_rn(n2, 1.0e-12f);
            if (d2 >= 1.e-3f) s0 = __fdiv_rn(d2, __fmul_rn(n2, 2.0f));
            else nb = -1;
        }
    }
    const int lane = threadIdx.x & 31, base = lane & ~7;
    float best = 1e24f, bn = 0.0f;
    int ba = -1;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float v = __shfl_sync(0xffffffffu, s0, base + k);
        const float vn = __shfl_sync(0xffffffffu, n2, base + k);
        const int vb = __shfl_sync(0xffffffffu, nb, base + k);
        if (vb >= 0 && v < best) { best = v; ba = vb; bn = vn; }
    }
    if (pix < npix && slot == 0) {
        const float sg = sqrtf(best);
        sig2[pix] = __fmul_rn(sg, sg);
        arg[pix] = ba;
        nsig[pix] = bn;
    }
}

// Window weights with the pieces of their derivative (one block per scan pixel, one thread per
// slot): w (normalised), m = max(d - dthresh, 0), and for the normalised distance
// d = (S - n s) / (s sqrt(2 n)) (s = sigma_p^2 + sigma_c^2): dS = dd/dS = 1 / (s sqrt(2 n)),
// ds = dd/ds = -S / (s^2 sqrt(2 n)); both 0 at the centre slot and where d is set to 1e6 n.
__global__ void k_nlpar_weights_d(const float* __restrict__ data, int nrows, int ncols, int npx,
                                  const int32_t* __restrict__ ind, int nind, float mxval,
                                  const float* __restrict__ sig2, float lam2, float dthresh, int sr,
                                  float* __restrict__ wout, float* __restrict__ mout, float* __restrict__ dsout,
                                  float* __restrict__ dgout) {
    extern __shared__ float w_s[];
    __shared__ float tot_s;
    const int pix = blockIdx.x;
    const int j = pix / ncols, i = pix - (pix / ncols) * ncols;
    int xs, xe, ys, ye;
    window(i, sr, ncols, xs, xe);
    window(j, sr, nrows, ys, ye);
    const int wx = xe - xs, winsz = (2 * sr + 1) * (2 * sr + 1);
    const int c = threadIdx.x;
    float m = 0.0f, dS = 0.0f, dg = 0.0f;
    if (c < winsz) {
        const int nb = (xs + c % wx) + ncols * (ys + c / wx);
        float w;
        if (nb == pix) {
            w = -1.0e6f;
        } else {
            float d2, n2;
            pair_ssd(data + (int64_t)pix * npx, data + (int64_t)nb * npx, ind, nind, mxval, d2, n2);
            const float ss = __fadd_rn(sig2[pix], sig2[nb]);
            const float S = d2;
            d2 = __fsub_rn(d2, __fmul_rn(n2, ss));
            const float dnorm = __fmul_rn(ss, sqrtf(__fmul_rn(2.0f, n2)));
            if (dnorm > 1.e-8f) {
                w = __fdiv_rn(d2, dnorm);
                dS = 1.0f / dnorm;
                dg = -S / (ss * dnorm);
            } else {
                w = __fmul_rn(1e6f, n2);
            }
        }
        m = fmaxf(__fsub_rn(w, dthresh), 0.0f);
        if (!(w - dthresh > 0.0f)) { dS = 0.0f; dg = 0.0f; }  // clamped: no derivative
        w_s[c] = expf(__fmul_rn(__fmul_rn(-1.0f, m), lam2));
    }
    __syncthreads();
    if (c == 0) {
        float t = 0.0f;
        for (int k = 0; k < winsz; ++k) t = __fadd_rn(t, w_s[k]);
        tot_s = t;
    }
    __syncthreads();
    if (c < winsz) {
        const int64_t o = (int64_t)pix * winsz + c;
        wout[o] = __fdiv_rn(w_s[c], tot_s);
        mout[o] = m;
        dsout[o] = dS;
        dgout[o] = dg;
    }
}

// G[p][c] = g_p . x_c over all pattern pixels (float64 sums); one block per scan pixel, one warp
// per kDotSlots window slots at a time: g_p is read once for them, and their sums are
// independent chains (with one slot a warp, the compensated sum's four dependent additions and
// the loads' latency were the bound).  1024 pixels of 14400 values, radius 2: 340 us before,
// 258 now (the loop unrolled by four: 319).
constexpr int kDotSlots = 4;
template <typename T>
__global__ void __launch_bounds__(256) k_nlpar_dots(const T* __restrict__ g, const T* __restrict__ x, int nrows,
                                                    int ncols, int npx, int sr, double* __restrict__ G) {
    const int p = blockIdx.x;
    const int jp = p / ncols, ip = p - (p / ncols) * ncols;
    int xs, xe, ys, ye;
    window(ip, sr, ncols, xs, xe);
    window(jp, sr, nrows, ys, ye);
    const int wx = xe - xs, winsz = (2 * sr + 1) * (2 * sr + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const T* gp = g + (int64_t)p * npx;
    for (int c0 = warp * kDotSlots; c0 < winsz; c0 += nw * kDotSlots) {
        const T* xc[kDotSlots];
        double acc[kDotSlots];
#pragma unroll
        for (int i = 0; i < kDotSlots; ++i) {
            const int c = c0 + i < winsz ? c0 + i : winsz - 1;
            xc[i] = x + (int64_t)((xs + c % wx) + ncols * (ys + c / wx)) * npx;
            acc[i] = 0.0;
        }
        if (sizeof(T) == 4) {
            // float patterns: each lane's products summed in float with Kahan's compensation
            // (off the slow FP64 pipe), the lanes' sums combined in double
            float sum[kDotSlots], comp[kDotSlots];
#pragma unroll
            for (int i = 0; i < kDotSlots; ++i) sum[i] = comp[i] = 0.0f;
#pragma unroll 2
            for (int k = lane; k < npx; k += 32) {
                const float gk = (float)__ldg(gp + k);
#pragma unroll
                for (int i = 0; i < kDotSlots; ++i) {
                    const float y = __fsub_rn(__fmul_rn(gk, (float)__ldg(xc[i] + k)), comp[i]);
                    const float t = __fadd_rn(sum[i], y);
                    comp[i] = __fsub_rn(__fsub_rn(t, sum[i]), y);
                    sum[i] = t;
                }
            }
#pragma unroll
            for (int i = 0; i < kDotSlots; ++i) acc[i] = (double)sum[i] - (double)comp[i];
        } else {
            for (int k = lane; k < npx; k += 32) {
                const double gk = (double)__ldg(gp + k);
#pragma unroll
                for (int i = 0; i < kDotSlots; ++i) acc[i] += gk * (double)__ldg(xc[i] + k);
            }
        }
#pragma unroll
        for (int i = 0; i < kDotSlots; ++i) {
            for (int o = 16; o > 0; o >>= 1) acc[i] += __shfl_down_sync(0xffffffffu, acc[i], o);
            if (lane == 0 && c0 + i < winsz) G[(int64_t)p * winsz + c0 + i] = acc[i];
        }
    }
}

// Per scan pixel p: Gbar = sum_c w_pc G_pc; dJ/dd_pc = -(w_pc / lam^2) (G_pc - Gbar) where the
// weight's exponent is not clamped; alpha = dJ/dd * dd/dS, beta = dJ/dd * dd/ds; and the lambda
// term sum_c w_pc (2 m_pc / lam^3) (G_pc - Gbar).
__global__ void k_nlpar_coef(const double* __restrict__ G, const float* __restrict__ w, const float* __restrict__ m,
                             const float* __restrict__ dS, const float* __restrict__ dg, int npix, int winsz,
                             double lam, double* __restrict__ alpha, double* __restrict__ beta,
                             double* __restrict__ glam) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    const int64_t o = (int64_t)p * winsz;
    double gbar = 0.0;
    for (int c = 0; c < winsz; ++c) gbar += (double)w[o + c] * G[o + c];
    const double il2 = 1.0 / (lam * lam), c3 = 2.0 / (lam * lam * lam);
    double gl = 0.0;
    for (int c = 0; c < winsz; ++c) {
        const double dg_ = G[o + c] - gbar;
        const double a = -(double)w[o + c] * il2 * dg_;
        alpha[o + c] = a * (double)dS[o + c];
        beta[o + c] = a * (double)dg[o + c];
        gl += (double)w[o + c] * c3 * (double)m[o + c] * dg_;
    }
    glam[p] = gl;
}

// gamma_q = dJ / d sigma_q^2 = sum of beta over the pairs that hold q (as window centre or as
// neighbour); s_pc = sigma_p^2 + sigma_c^2 enters both.
__global__ void k_nlpar_gamma(const double* __restrict__ beta, int nrows, int ncols, int sr,
                              double* __restrict__ gamma) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nrows * ncols) return;
    const int winsz = (2 * sr + 1) * (2 * sr + 1), wx = 2 * sr + 1;
    const int jq = q / ncols, iq = q - (q / ncols) * ncols;
    double acc = 0.0;
    for (int c = 0; c < winsz; ++c) acc += beta[(int64_t)q * winsz + c];
    const int j0 = jq - 2 * sr < 0 ? 0 : jq - 2 * sr, j1 = jq + 2 * sr > nrows - 1 ? nrows - 1 : jq + 2 * sr;
    const int i0 = iq - 2 * sr < 0 ? 0 : iq - 2 * sr, i1 = iq + 2 * sr > ncols - 1 ? ncols - 1 : iq + 2 * sr;
    for (int jp = j0; jp <= j1; ++jp) {
        int ys, ye;
        window(jp, sr, nrows, ys, ye);
        if (jq < ys || jq >= ye) continue;
        for (int ip = i0; ip <= i1; ++ip) {
            int xs, xe;
            window(ip, sr, ncols, xs, xe);
            if (iq < xs || iq >= xe) continue;
            const int p = ip + ncols * jp;
            if (p == q) continue;
            acc += beta[(int64_t)p * winsz + (jq - ys) * wx + (iq - xs)];
        }
    }
    gamma[q] = acc;
}

// dJ/dx_q[k] from the weights' dependence on the patterns: the pair SSDs of q's own window, of
// the windows that hold q, and the noise sigma's minimising pair (q's own, and those of the
// 3x3 neighbours whose minimum pairs with q).  Masked pixels only, each pair's saturation test.
// One scan pixel q per blockIdx.x, the threads over the pattern values k.  The block's first warp
// lists the pixels n that share a pair with q and their coefficients -- 2 alpha of the pair as q's
// slot plus 2 alpha as n's slot, added in double, then gamma / n of the sigma pairs -- and every
// value adds coef * (x_q - x_n) for the terms whose two values pass the saturation test of their
// kind (a value of q that fails it, or lies off the mask, compares with -infinity).  Float
// patterns accumulate in float (the coefficients rounded once), double in double.  A thread takes
// four values, so four loads are in flight a term: with one value a thread and a list of both
// orders of each pair made by one thread, latency was the bound.  1024 pixels of 14400 values,
// radius 2: 1520 us before, 211 now.
constexpr int kDxVals = 4, kDxThreads = 256;
template <typename T>
__global__ void __launch_bounds__(kDxThreads) k_nlpar_dx(const T* __restrict__ x, int nrows, int ncols, int npx, int sr,
                                                         const uint8_t* __restrict__ pmask, float mxw, float mxs,
                                                         const double* __restrict__ alpha,
                                                         const double* __restrict__ gamma, const int* __restrict__ arg,
                                                         const float* __restrict__ nsig, T* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char dxsm[];
    const int q = blockIdx.x;
    const int winsz = (2 * sr + 1) * (2 * sr + 1);
    const int maxt = (4 * sr + 1) * (4 * sr + 1) + 10;
    T* co = (T*)dxsm;                        // [maxt] coefficients
    int* nbs = (int*)(co + maxt);           // [maxt] the other pixel
    __shared__ int nwt, nterm;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x, jq = q / ncols, iq = q - (q / ncols) * ncols;
        const int nw = list_near(
            q, nrows, ncols, 2 * sr, lane, 0,
            [&](int p, int jp, int ip) {
                return p != q && (slot_of(jp, ip, jq, iq, sr, nrows, ncols) >= 0 ||
                                  slot_of(jq, iq, jp, ip, sr, nrows, ncols) >= 0);
            },
            [&](int t, int p, int jp, int ip) {
                const int mine = slot_of(jq, iq, jp, ip, sr, nrows, ncols);
                const int theirs = slot_of(jp, ip, jq, iq, sr, nrows, ncols);
                double a = 0.0;
                if (mine >= 0) a = 2.0 * alpha[(int64_t)q * winsz + mine];
                if (theirs >= 0) a += 2.0 * alpha[(int64_t)p * winsz + theirs];
                co[t] = (T)a;
                nbs[t] = p;
            });
        // noise sigma: sigma_p^2 = SSD(p, arg_p) / (2 n_p)
        int nt = nw;
        const int aq = arg[q];
        if (aq >= 0) {
            if (lane == 0) {
                co[nt] = (T)(gamma[q] / (double)nsig[q]);
                nbs[nt] = aq;
            }
            ++nt;
        }
        nt = list_near(
            q, nrows, ncols, 1, lane, nt, [&](int p, int, int) { return p != q && arg[p] == q; },
            [&](int t, int p, int, int) {
                co[t] = (T)(gamma[p] / (double)nsig[p]);
                nbs[t] = p;
            });
        if (lane == 0) {
            nwt = nw;
            nterm = nt;
        }
    }
    __syncthreads();
    const int nw = nwt, nt = nterm;
    const T* xq_row = x + (int64_t)q * npx;
    for (int k0 = blockIdx.y * (kDxThreads * kDxVals) + threadIdx.x; k0 < npx;
         k0 += gridDim.y * (kDxThreads * kDxVals)) {
        int kk[kDxVals];
        T xq[kDxVals], lim[kDxVals], acc[kDxVals];
        bool on[kDxVals];
#pragma unroll
        for (int i = 0; i < kDxVals; ++i) {
            const int k = k0 + i * kDxThreads;
            kk[i] = k < npx ? k : k0;
            on[i] = pmask[kk[i]] != 0;
            xq[i] = xq_row[kk[i]];
            lim[i] = on[i] && xq[i] < (T)mxw ? (T)mxw : (T)-INFINITY;
            acc[i] = (T)0;
        }
        auto add = [&](int t) {
            const T* xn_row = x + (int64_t)nbs[t] * npx;
            const T c = co[t];
            T xn[kDxVals];
#pragma unroll
            for (int i = 0; i < kDxVals; ++i) xn[i] = __ldg(xn_row + kk[i]);
#pragma unroll
            for (int i = 0; i < kDxVals; ++i)
                if (xn[i] < lim[i]) acc[i] += c * (xq[i] - xn[i]);
        };
#pragma unroll 2
        for (int t = 0; t < nw; ++t) add(t);
#pragma unroll
        for (int i = 0; i < kDxVals; ++i) lim[i] = on[i] && xq[i] < (T)mxs ? (T)mxs : (T)-INFINITY;
        for (int t = nw; t < nt; ++t) add(t);
#pragma unroll
        for (int i = 0; i < kDxVals; ++i)
            if (k0 + i * kDxThreads < npx) out[(int64_t)q * npx + kk[i]] = acc[i];
    }
}

}  // namespace
}  // namespace ebsd

using namespace ebsd;

extern "C" {

int ebsd_linop_create(int64_t nrows, int64_t ncols, const int64_t* rowptr, const int32_t* col, const float* val,
                      int device, ebsd_linop_t* out) {
    if (!out || nrows <= 0 || ncols <= 0 || !rowptr || (!col && rowptr[nrows] > 0) || (!val && rowptr[nrows] > 0))
        return EBSD_E_ARG;
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return EBSD_E_DEVICE;
    int64_t nnz = rowptr[nrows];
    for (int64_t e = 0; e < nnz; ++e)
        if (col[e] < 0 || col[e] >= ncols) return EBSD_E_ARG;
    ebsd_linop_s* op = new (std::nothrow) ebsd_linop_s();
    if (!op) return EBSD_E_NOMEM;
    op->device = device;
    op->nrows = nrows;
    op->ncols = ncols;
    op->nnz = nnz;
    std::vector<double> v64(val, val + nnz);
    std::vector<int2> ent((size_t)nnz);
    for (int64_t e = 0; e < nnz; ++e) {
        ent[e].x = col[e];
        std::memcpy(&ent[e].y, &val[e], sizeof(float));
    }
    bool ok = cudaMalloc((void**)&op->rowptr, (nrows + 1) * sizeof(int64_t)) == cudaSuccess &&
              cudaMalloc((void**)&op->col, std::max<int64_t>(nnz, 1) * sizeof(int32_t)) == cudaSuccess &&
              cudaMalloc((void**)&op->val, std::max<int64_t>(nnz, 1) * sizeof(float)) == cudaSuccess &&
              cudaMalloc((void**)&op->val64, std::max<int64_t>(nnz, 1) * sizeof(double)) == cudaSuccess &&
              cudaMalloc((void**)&op->ent, std::max<int64_t>(nnz, 1) * sizeof(int2)) == cudaSuccess;
    ok = ok && cudaMemcpy(op->rowptr, rowptr, (nrows + 1) * sizeof(int64_t), cudaMemcpyHostToDevice) == cudaSuccess;
    if (ok && nnz > 0) {
        ok = cudaMemcpy(op->col, col, nnz * sizeof(int32_t), cudaMemcpyHostToDevice) == cudaSuccess &&
             cudaMemcpy(op->val, val, nnz * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess &&
             cudaMemcpy(op->val64, v64.data(), nnz * sizeof(double), cudaMemcpyHostToDevice) == cudaSuccess &&
             cudaMemcpy(op->ent, ent.data(), nnz * sizeof(int2), cudaMemcpyHostToDevice) == cudaSuccess;
    }
    if (!ok) {
        cudaFree(op->rowptr);
        cudaFree(op->col);
        cudaFree(op->val);
        cudaFree(op->val64);
        cudaFree(op->ent);
        delete op;
        return EBSD_E_NOMEM;
    }
    *out = op;
    return EBSD_OK;
}

int ebsd_linop_apply(ebsd_linop_t op, int fp64, const void* d_x, int64_t n, void* d_y, void* stream) {
    if (!op || n < 0 || (n > 0 && (!d_x || !d_y)) || n > 65535) return EBSD_E_ARG;
    if (n == 0) return EBSD_OK;
    if (cudaSetDevice(op->device) != cudaSuccess) return EBSD_E_DEVICE;
    dim3 grid((unsigned)((op->nrows + 255) / 256), (unsigned)n);
    if (fp64)
        k_csr_gather<double><<<grid, 256, 0, (cudaStream_t)stream>>>(op->rowptr, op->col, op->val64,
                                                                    (const double*)d_x, (double*)d_y,
                                                                    op->nrows, op->ncols);
    else
        k_csr_gather<float><<<grid, 256, 0, (cudaStream_t)stream>>>(op->rowptr, op->col, op->val,
                                                                   (const float*)d_x, (float*)d_y,
                                                                   op->nrows, op->ncols);
    return launch_status();
}

int ebsd_linop_apply_cols(ebsd_linop_t op, int fp64, const void* d_xT, int64_t ldx, int64_t n, void* d_yT,
                          int64_t ldy, void* stream) {
    if (!op || n < 0 || (n > 0 && (!d_xT || !d_yT)) || ldx < n || ldy < n || (n + 31) / 32 > 65535) return EBSD_E_ARG;
    if (n == 0) return EBSD_OK;
    if (cudaSetDevice(op->device) != cudaSuccess) return EBSD_E_DEVICE;
    // without an image the rows stand as one of kCsrTileX columns: a tile is kCsrTileY * kCsrTileX rows in a row
    const int64_t width = op->width > 0 ? op->width : kCsrTileX;
    if ((op->nrows + kCsrTileY * width - 1) / (kCsrTileY * width) * ((width + kCsrTileX - 1) / kCsrTileX) > 0x7fffffff) return EBSD_E_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (fp64)
        launch_csr_cols<double>(st, op->rowptr, CsrEnt<double>{op->col, op->val64}, (const double*)d_xT, ldx, (double*)d_yT, ldy,
                                op->nrows, width, n);
    else
        launch_csr_cols<float>(st, op->rowptr, CsrEnt<float>{op->ent}, (const float*)d_xT, ldx, (float*)d_yT, ldy, op->nrows,
                               width, n);
    return launch_status();
}

int ebsd_linop_set_width(ebsd_linop_t op, int64_t width) {
    if (!op || width < 0 || width > op->nrows) return EBSD_E_ARG;
    op->width = width;
    return EBSD_OK;
}

int ebsd_linop_destroy(ebsd_linop_t op) {
    if (!op) return EBSD_E_ARG;
    cudaSetDevice(op->device);
    cudaFree(op->rowptr);
    cudaFree(op->col);
    cudaFree(op->val);
    cudaFree(op->val64);
    cudaFree(op->ent);
    delete op;
    return EBSD_OK;
}

int ebsd_nlpar_weights(const float* d_data, int32_t nrows, int32_t ncols, int32_t npx, const int32_t* d_indices,
                       int32_t nind, float datamax, float lam, int32_t sr, float dthresh, const float* d_sigma,
                       int saturation_protect, float* d_w, float* d_m, void* stream) {
    if (!d_data || !d_indices || !d_sigma || !d_w || !d_m || nrows <= 0 || ncols <= 0 || npx <= 0 || nind < 0 ||
        nind > npx || sr < 0 || sr > 10 || !(lam > 0.0f) || 2 * sr + 1 > nrows || 2 * sr + 1 > ncols)
        return EBSD_E_ARG;
    float mxval = saturation_protect ? datamax * 0.999f : datamax + 1.0f;
    float lam2 = 1.0f / (lam * lam);
    int winsz = (2 * sr + 1) * (2 * sr + 1);
    k_nlpar_weights2<<<(unsigned)(nrows * ncols), ((winsz + 31) / 32) * 32, winsz * sizeof(float),
                       (cudaStream_t)stream>>>(d_data, nrows, ncols, npx, d_indices, nind, mxval, d_sigma, lam2,
                                               dthresh, sr, d_w, d_m);
    return launch_status();
}

int ebsd_blur1d(int fp64, int adjoint, int axis, const void* d_in, int64_t n, int32_t H, int32_t W,
                const void* d_taps, int32_t r, void* d_out, void* stream) {
    if (!d_in || !d_taps || !d_out || n < 0 || H <= 0 || W <= 0 || r < 0 || (axis != 0 && axis != 1) ||
        r >= (axis == 0 ? H : W))
        return EBSD_E_ARG;
    const int64_t total = n * H * W;
    if (total == 0) return EBSD_OK;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    cudaStream_t st = (cudaStream_t)stream;
    if (fp64) {
        if (adjoint) k_blur1d_t<double><<<blocks, 256, 0, st>>>((const double*)d_in, (double*)d_out, total, H, W, axis, (const double*)d_taps, r);
        else k_blur1d<double><<<blocks, 256, 0, st>>>((const double*)d_in, (double*)d_out, total, H, W, axis, (const double*)d_taps, r);
    } else if (blur_blocked(n, H, W, axis, r)) {
        const float *in = (const float*)d_in, *tp = (const float*)d_taps;
        float* o = (float*)d_out;
        if (axis == 0) return adjoint ? launch_blur<0, true>(in, n, H, W, tp, r, o, st) : launch_blur<0, false>(in, n, H, W, tp, r, o, st);
        return adjoint ? launch_blur<1, true>(in, n, H, W, tp, r, o, st) : launch_blur<1, false>(in, n, H, W, tp, r, o, st);
    } else {
        if (adjoint) k_blur1d_t<float><<<blocks, 256, 0, st>>>((const float*)d_in, (float*)d_out, total, H, W, axis, (const float*)d_taps, r);
        else k_blur1d<float><<<blocks, 256, 0, st>>>((const float*)d_in, (float*)d_out, total, H, W, axis, (const float*)d_taps, r);
    }
    return launch_status();
}

int ebsd_softargmax(int fp64, const void* d_c, int64_t n, int64_t ncell, const int32_t* d_cells, int32_t ncm,
                    double tau, double* d_J, void* d_grad, void* stream) {
    if (!d_c || !d_cells || !d_J || !d_grad || n < 0 || ncell <= 0 || ncm <= 0 || ncm > ncell || !(tau > 0.0))
        return EBSD_E_ARG;
    if (n == 0) return EBSD_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (fp64) k_softargmax<double><<<(unsigned)n, 256, 0, st>>>((const double*)d_c, ncell, d_cells, ncm, 1.0 / tau, d_J, (double*)d_grad);
    else k_softargmax<float><<<(unsigned)n, 256, 0, st>>>((const float*)d_c, ncell, d_cells, ncm, 1.0 / tau, d_J, (float*)d_grad);
    return launch_status();
}

int ebsd_nlpar_sigma_arg(const float* d_data, int32_t nrows, int32_t ncols, int32_t npx, const int32_t* d_indices,
                         int32_t nind, float datamax, int saturation_protect, float* d_sig2, int32_t* d_arg,
                         float* d_nsig, void* stream) {
    if (!d_data || !d_indices || !d_sig2 || !d_arg || !d_nsig || nrows <= 0 || ncols <= 0 || npx <= 0 || nind < 0 ||
        nind > npx)
        return EBSD_E_ARG;
    const float mxval = saturation_protect ? datamax * 0.9961f : datamax + 1.0f;
    const int npix = nrows * ncols;
    k_sigma_arg<<<(unsigned)(((int64_t)npix * 8 + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
        d_data, nrows, ncols, npx, d_indices, nind, mxval, d_sig2, d_arg, d_nsig);
    return launch_status();
}

int ebsd_nlpar_weights_d(const float* d_data, int32_t nrows, int32_t ncols, int32_t npx, const int32_t* d_indices,
                         int32_t nind, float datamax, float lam, int32_t sr, float dthresh, const float* d_sig2,
                         int saturation_protect, float* d_w, float* d_m, float* d_dS, float* d_dsig, void* stream) {
    if (!d_data || !d_indices || !d_sig2 || !d_w || !d_m || !d_dS || !d_dsig || nrows <= 0 || ncols <= 0 ||
        npx <= 0 || nind < 0 || nind > npx || sr < 0 || sr > 10 || !(lam > 0.0f) || 2 * sr + 1 > nrows ||
        2 * sr + 1 > ncols)
        return EBSD_E_ARG;
    const float mxval = saturation_protect ? datamax * 0.999f : datamax + 1.0f;
    const int winsz = (2 * sr + 1) * (2 * sr + 1);
    k_nlpar_weights_d<<<(unsigned)(nrows * ncols), ((winsz + 31) / 32) * 32, winsz * sizeof(float),
                        (cudaStream_t)stream>>>(d_data, nrows, ncols, npx, d_indices, nind, mxval, d_sig2,
                                                1.0f / (lam * lam), dthresh, sr, d_w, d_m, d_dS, d_dsig);
    return launch_status();
}

int ebsd_nlpar_weights_grad(int fp64, const void* d_g, const void* d_x, int32_t nrows, int32_t ncols, int32_t npx,
                            int32_t sr, const float* d_w, const float* d_m, const float* d_dS, const float* d_dsig,
                            double lam, const uint8_t* d_pmask, float datamax, int saturation_protect,
                            const int32_t* d_arg, const float* d_nsig, double* d_scratch, double* d_glam,
                            void* d_gx, void* stream) {
    if (!d_g || !d_x || !d_w || !d_m || !d_dS || !d_dsig || !d_pmask || !d_arg || !d_nsig || !d_scratch ||
        !d_glam || !d_gx || nrows <= 0 || ncols <= 0 || npx <= 0 || sr < 0 || sr > 10 || !(lam > 0.0))
        return EBSD_E_ARG;
    const int npix = nrows * ncols, winsz = (2 * sr + 1) * (2 * sr + 1);
    double* G = d_scratch;
    double* alpha = G + (int64_t)npix * winsz;
    double* beta = alpha + (int64_t)npix * winsz;
    double* gamma = beta + (int64_t)npix * winsz;
    cudaStream_t st = (cudaStream_t)stream;
    const float mxw = saturation_protect ? datamax * 0.999f : datamax + 1.0f;
    const float mxs = saturation_protect ? datamax * 0.9961f : datamax + 1.0f;
    if (fp64) k_nlpar_dots<double><<<(unsigned)npix, 256, 0, st>>>((const double*)d_g, (const double*)d_x, nrows, ncols, npx, sr, G);
    else k_nlpar_dots<float><<<(unsigned)npix, 256, 0, st>>>((const float*)d_g, (const float*)d_x, nrows, ncols, npx, sr, G);
    k_nlpar_coef<<<(unsigned)((npix + 127) / 128), 128, 0, st>>>(G, d_w, d_m, d_dS, d_dsig, npix, winsz, lam, alpha,
                                                                 beta, d_glam);
    k_nlpar_gamma<<<(unsigned)((npix + 127) / 128), 128, 0, st>>>(beta, nrows, ncols, sr, gamma);
    const size_t maxt = (size_t)(4 * sr + 1) * (4 * sr + 1) + 10;
    const size_t dsm = maxt * ((fp64 ? sizeof(double) : sizeof(float)) + sizeof(int));
    // the values of a pixel over as many blocks as it takes to fill the chip (sixteen an SM)
    const int chunks = (npx + kDxThreads * kDxVals - 1) / (kDxThreads * kDxVals), want = (152 * 16 + npix - 1) / npix;
    const dim3 xgrid((unsigned)npix, (unsigned)(want < chunks ? want : chunks));
    if (fp64) k_nlpar_dx<double><<<xgrid, kDxThreads, dsm, st>>>((const double*)d_x, nrows, ncols, npx, sr, d_pmask, mxw, mxs, alpha, gamma, d_arg, d_nsig, (double*)d_gx);
    else k_nlpar_dx<float><<<xgrid, kDxThreads, dsm, st>>>((const float*)d_x, nrows, ncols, npx, sr, d_pmask, mxw, mxs, alpha, gamma, d_arg, d_nsig, (float*)d_gx);
    return launch_status();
}

int ebsd_nlpar_apply_t(const float* d_g, int32_t nrows, int32_t ncols, int32_t npx, const float* d_w, int32_t sr,
                       float* d_out, void* stream) {
    if (!d_g || !d_w || !d_out || nrows <= 0 || ncols <= 0 || npx <= 0 || sr < 0 || sr > 10) return EBSD_E_ARG;
    dim3 grid((unsigned)((npx + 256 * kAtVals - 1) / (256 * kAtVals)), (unsigned)(nrows * ncols));
    k_nlpar_apply_t<float><<<grid, 256, (size_t)(4 * sr + 1) * (4 * sr + 1) * (sizeof(float) + sizeof(int)),
                             (cudaStream_t)stream>>>(d_g, nrows, ncols, npx, d_w, sr, d_out);
    return launch_status();
}

int ebsd_nlpar_apply_t64(const double* d_g, int32_t nrows, int32_t ncols, int32_t npx, const double* d_w,
                         int32_t sr, double* d_out, void* stream) {
    if (!d_g || !d_w || !d_out || nrows <= 0 || ncols <= 0 || npx <= 0 || sr < 0 || sr > 10) return EBSD_E_ARG;
    dim3 grid((unsigned)((npx + 256 * kAtVals - 1) / (256 * kAtVals)), (unsigned)(nrows * ncols));
    k_nlpar_apply_t<double><<<grid, 256, (size_t)(4 * sr + 1) * (4 * sr + 1) * (sizeof(double) + sizeof(int)),
                              (cudaStream_t)stream>>>(d_g, nrows, ncols, npx, d_w, sr, d_out);
    return launch_status();
}

int ebsd_nlpar_lambda_grad(const float* d_g, const float* d_x, int32_t nrows, int32_t ncols, int32_t npx,
                           const float* d_w, const float* d_m, int32_t sr, float lam, double* d_out,
                           void* stream) {
    if (!d_g || !d_x || !d_w || !d_m || !d_out || nrows <= 0 || ncols <= 0 || npx <= 0 || sr < 0 || sr > 10 ||
        !(lam > 0.0f))
        return EBSD_E_ARG;
    k_nlpar_lam_grad<float><<<(unsigned)(nrows * ncols), 256, 0, (cudaStream_t)stream>>>(
        d_g, d_x, nrows, ncols, npx, d_w, d_m, sr, lam, d_out);
    return launch_status();
}

int ebsd_nlpar_lambda_grad64(const double* d_g, const double* d_x, int32_t nrows, int32_t ncols, int32_t npx,
                             const float* d_w, const float* d_m, int32_t sr, float lam, double* d_out,
                             void* stream) {
    if (!d_g || !d_x || !d_w || !d_m || !d_out || nrows <= 0 || ncols <= 0 || npx <= 0 || sr < 0 || sr > 10 ||
        !(lam > 0.0f))
        return EBSD_E_ARG;
    k_nlpar_lam_grad<double><<<(unsigned)(nrows * ncols), 256, 0, (cudaStream_t)stream>>>(
        d_g, d_x, nrows, ncols, npx, d_w, d_m, sr, lam, d_out);
    return launch_status();
}

}  // extern "C"
