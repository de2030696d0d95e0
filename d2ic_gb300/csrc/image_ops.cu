// Image preparation kernels: cubic B-spline prefilter, halo padding, point
// sampling and pixel-record packing.
//
// The prefilter computes the interpolating cubic B-spline coefficients of the
// edge-extended image.  The exact inverse of the sampled B-spline kernel
// (1, 4, 1)/6 has impulse response h[k] = sqrt(3) * z^|k|, z = sqrt(3) - 2
// (Unser, "B-spline signal processing", IEEE TSP 1993).  |z|^17 < 2e-10, so a
// 33-tap FIR (|k| <= 16) applied separably to the edge-replicated image gives
// the coefficients to FP32 precision with fully parallel, coalesced passes
// (instead of the sequential causal/anti-causal recursion).
#include "common.cuh"

namespace d2ic {

constexpr int KF = 16;                 // FIR half-length
__constant__ float c_fir[2 * KF + 1];
static bool g_fir_ready[64] = {false};

static int ensure_fir() {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && g_fir_ready[dev]) return D2IC_OK;
    float h[2 * KF + 1];
    const double z = 1.7320508075688772 - 2.0;
    for (int k = -KF; k <= KF; ++k) {
        double v = 1.7320508075688772;
        for (int i = 0; i < (k < 0 ? -k : k); ++i) v *= z;
        h[k + KF] = (float)v;
    }
    cudaError_t e = cudaMemcpyToSymbol(c_fir, h, sizeof(h));
    if (e != cudaSuccess) return cuda_status(e, "prefilter constants");
    if (dev >= 0 && dev < 64) g_fir_ready[dev] = true;
    return D2IC_OK;
}

// One launch filters rows and columns: coeff[cy][cx] = sum_k h[k] f[clamp(cy - pad + k)][cx], with
// f[y][cx] = sum_k h[k] img[y][clamp(cx - pad + k)], k = -KF .. KF, for cy in [0, H + 2 pad), cx in [0, W + 2 pad),
// of image blockIdx.z of a batch (contiguous images and buffers).  T: float or 8-bit camera pixels.
//
// A block makes PF_W columns x `rows` rows of the result.  It filters the rows + 2 KF image rows that these need,
// PF_STAGE at a time from an edge-extended copy in shared memory (the next ones are loaded while a stage is
// filtered), keeps the filtered rows in shared memory and filters their columns.  A thread makes 8 neighbouring
// outputs of two rows, then 8 of two columns, two per instruction; every output's taps are summed in order
// k = -KF .. KF.
//
// 66 multiply-adds per pixel, and 33 more for the 2 KF extra rows per block, bound it (58 % of the FMA rate; the
// rest is the barriers between the stages of two blocks per SM).  Two launches with the row sums in memory took
// 482 us for 64 images of 1024 x 1024, 144 us for one of 4096 x 4096 and 15.4 us for one of 512 x 512 (two more
// passes over memory, loads that nothing overlapped); this takes 270, 68 and 9.6 us, and 302, 74 and 8.9 us with one
// output per instruction.  128 rows per block are best when there are blocks enough for the chip (64 rows and three
// blocks per SM: 275 us for the 64 images); smaller images take 64 or 32 rows (prefilter_rows_per_block).
constexpr int PF_W = 128, PF_STAGE = 32, PF_THREADS = 256;
constexpr int PF_IN = PF_W + 2 * KF;                       // staged columns
constexpr int PF_PITCH = 2 * PF_IN + PF_IN / 16 * 4;       // two staged rows side by side (see pf_at)
constexpr int PF_LOADS = PF_STAGE * PF_IN / PF_THREADS;    // staged elements per thread
static_assert(PF_IN % 32 == 0 && PF_STAGE % (PF_THREADS / 32) == 0, "a warp stages whole rows");
// Element i of a pair of staged rows (a float of each), with 4 floats after every 16: a quarter warp's 16-byte
// reads at a stride of 8 elements then fall into different banks.
__device__ __forceinline__ int pf_at(int i) { return 2 * i + ((i >> 4) << 2); }

// GRADIENTS: the batch is one image and its central-difference gradient images (zero on the first and last column, row),
// formed while the rows are loaded, with their results at coeff, coeff_gx and coeff_gy.
template <class T, bool GRADIENTS = false>
__global__ void __launch_bounds__(PF_THREADS, 2) prefilter_kernel(const T *__restrict__ img, int H, int W, int pad, int cpitch,
                                                                  int rows, float *__restrict__ coeff,
                                                                  float *__restrict__ coeff_gx, float *__restrict__ coeff_gy) {
    extern __shared__ __align__(16) float pf_smem[];
    float *stage = pf_smem;                                // PF_STAGE / 2 x PF_PITCH
    float *filt = pf_smem + PF_STAGE / 2 * PF_PITCH;       // (rows + 2 KF) x PF_W: the filtered rows
    const int which = GRADIENTS ? (int)blockIdx.z : 0;
    if (!GRADIENTS) {
        img += (size_t)blockIdx.z * H * W;
        coeff += (size_t)blockIdx.z * (H + 2 * pad) * cpitch;
    } else if (which) {
        coeff = which == 1 ? coeff_gx : coeff_gy;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cx0 = blockIdx.x * PF_W, cy0 = blockIdx.y * rows;
    const int out_rows = min(rows, H + 2 * pad - cy0), in_rows = out_rows + 2 * KF;
    const int n_cols = min(PF_W, W + 2 * pad - cx0);
    Pair h[KF + 1];                                        // h[k] = h[-k]
#pragma unroll
    for (int k = 0; k <= KF; ++k) h[k] = pair(c_fir[KF + k]);
    int col[PF_IN / 32];
#pragma unroll
    for (int j = 0; j < PF_IN / 32; ++j) col[j] = clampi(cx0 - pad - KF + 32 * j + lane, 0, W - 1);
    constexpr int RPW = PF_STAGE / (PF_THREADS / 32);      // staged rows per warp
    float next[PF_LOADS];
    auto load = [&](int r0) {                              // rows r0 .. of the block's image rows
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const int y = clampi(cy0 - pad - KF + r0 + warp * RPW + r, 0, H - 1);
            const T *row = img + (size_t)y * W;
#pragma unroll
            for (int j = 0; j < PF_IN / 32; ++j) {
                float v = 0.f;
                if (which == 0) v = (float)__ldg(row + col[j]);
                else if (which == 1 && col[j] > 0 && col[j] < W - 1)
                    v = 0.5f * ((float)__ldg(row + col[j] + 1) - (float)__ldg(row + col[j] - 1));
                else if (which == 2 && y > 0 && y < H - 1)
                    v = 0.5f * ((float)__ldg(row + W + col[j]) - (float)__ldg(row - W + col[j]));
                next[r * (PF_IN / 32) + j] = v;
            }
        }
    };
    load(0);
    const int lg = 32 - __clz((n_cols - 1) / 8);           // 2^lg threads per row, 8 outputs each
    for (int r0 = 0; r0 < in_rows; r0 += PF_STAGE) {
        __syncthreads();                                   // the previous stage is filtered
#pragma unroll
        for (int r = 0; r < RPW; r += 2)
#pragma unroll
            for (int j = 0; j < PF_IN / 32; ++j)
                *reinterpret_cast<float2 *>(stage + (warp * RPW + r) / 2 * PF_PITCH + pf_at(32 * j + lane)) =
                    make_float2(next[r * (PF_IN / 32) + j], next[(r + 1) * (PF_IN / 32) + j]);
        __syncthreads();
        if (r0 + PF_STAGE < in_rows) load(r0 + PF_STAGE);
#pragma unroll 1
        for (int i = threadIdx.x; i < (PF_STAGE / 2) << lg; i += PF_THREADS) {
            const int r = 2 * (i >> lg), x = 8 * (i & ((1 << lg) - 1));
            if (r0 + r >= in_rows) break;
            const float *src = stage + r / 2 * PF_PITCH;
            Pair acc[8];
#pragma unroll
            for (int o = 0; o < 8; ++o) acc[o] = 0ull;
#pragma unroll
            for (int m = 0; m < (2 * KF + 8) / 2; ++m) {
                const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(src + pf_at(x + 2 * m));
                const Pair v[2] = {q.x, q.y};
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int o = 0; o < 8; ++o) {
                        const int k = 2 * m + e - o - KF;
                        if (k >= -KF && k <= KF) acc[o] = pair_fma(h[k < 0 ? -k : k], v[e], acc[o]);
                    }
            }
            float4 *dst = reinterpret_cast<float4 *>(filt + (size_t)(r0 + r) * PF_W + x);
            dst[0] = make_float4(pair_lo(acc[0]), pair_lo(acc[1]), pair_lo(acc[2]), pair_lo(acc[3]));
            dst[1] = make_float4(pair_lo(acc[4]), pair_lo(acc[5]), pair_lo(acc[6]), pair_lo(acc[7]));
            dst += PF_W / 4;
            dst[0] = make_float4(pair_hi(acc[0]), pair_hi(acc[1]), pair_hi(acc[2]), pair_hi(acc[3]));
            dst[1] = make_float4(pair_hi(acc[4]), pair_hi(acc[5]), pair_hi(acc[6]), pair_hi(acc[7]));
        }
    }
    __syncthreads();
    constexpr int R = 8;
    const int lg2 = 32 - __clz((n_cols - 1) / 2);          // 2^lg2 threads per strip of R rows, 2 columns each
    const int x = 2 * ((int)threadIdx.x & ((1 << lg2) - 1));
    if (x >= n_cols) return;
    const bool both = x + 1 < n_cols;
#pragma unroll 1
    for (int y0 = R * ((int)threadIdx.x >> lg2); y0 < out_rows; y0 += R * (PF_THREADS >> lg2)) {
        Pair acc[R];
#pragma unroll
        for (int o = 0; o < R; ++o) acc[o] = 0ull;
#pragma unroll
        for (int j = 0; j < R + 2 * KF; ++j) {
            // rows past in_rows: of outputs that are not stored
            const Pair v = *reinterpret_cast<const Pair *>(filt + (y0 + j) * PF_W + x);
#pragma unroll
            for (int o = 0; o < R; ++o) {
                const int k = j - o - KF;
                if (k >= -KF && k <= KF) acc[o] = pair_fma(h[k < 0 ? -k : k], v, acc[o]);
            }
        }
#pragma unroll
        for (int o = 0; o < R; ++o)
            if (y0 + o < out_rows) {
                float *out = coeff + (size_t)(cy0 + y0 + o) * cpitch + cx0 + x;
                out[0] = pair_lo(acc[o]);
                if (both) out[1] = pair_hi(acc[o]);
            }
    }
}

static size_t prefilter_smem(int rows) {
    return sizeof(float) * ((size_t)PF_STAGE / 2 * PF_PITCH + (size_t)(rows + 2 * KF) * PF_W);
}

// The most rows per block that still give the chip two blocks per SM; small images take the fewest.
static int prefilter_rows_per_block(int CW, int CH, int n_images, int sms) {
    for (int rows = 128; rows > 32; rows /= 2)
        if ((long long)((CW + PF_W - 1) / PF_W) * ((CH + rows - 1) / rows) * n_images >= 2ll * sms) return rows;
    return 32;
}

template <class T, bool GRADIENTS = false>
static int prefilter_launch(const T *img, int n_images, int H, int W, int pad, int cpitch, float *coeff, cudaStream_t s,
                            float *coeff_gx = nullptr, float *coeff_gy = nullptr) {
    int st = ensure_fir();
    if (st) return st;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(prefilter_kernel<T, GRADIENTS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)prefilter_smem(128));
    if (e != cudaSuccess) return cuda_status(e, "prefilter");
    const int CW = W + 2 * pad, CH = H + 2 * pad;
    const int rows = prefilter_rows_per_block(CW, CH, n_images, sms);
    prefilter_kernel<T, GRADIENTS><<<dim3((CW + PF_W - 1) / PF_W, (CH + rows - 1) / rows, n_images), PF_THREADS,
                                     prefilter_smem(rows), s>>>(img, H, W, pad, cpitch, rows, coeff, coeff_gx, coeff_gy);
    D2IC_CHECK_LAUNCH("prefilter");
    return D2IC_OK;
}

template <class T>
__global__ void pad_image_kernel(const T *__restrict__ img, int H, int W, int pad, int cpitch,
                                 float *__restrict__ out) {
    const int cx = blockIdx.x * blockDim.x + threadIdx.x;
    const int cy = blockIdx.y;
    if (cx >= W + 2 * pad) return;
    const int sy = clampi(cy - pad, 0, H - 1), sx = clampi(cx - pad, 0, W - 1);
    out[(size_t)cy * cpitch + cx] = (float)__ldg(img + (size_t)sy * W + sx);
}

template <class T>
static int prefilter_one(const T *img, int H, int W, int pad, int cpitch, float *tmp, float *coeff, cudaStream_t s,
                         const char *name) {
    D2IC_REQUIRE(img && tmp && coeff, "%s: null pointer", name);
    D2IC_REQUIRE(H > 0 && W > 0 && H < 65536 && W < 65536, "%s: bad image size %dx%d", name, H, W);
    D2IC_REQUIRE(pad >= KF && cpitch >= W + 2 * pad, "%s: need pad >= %d and cpitch >= W + 2 pad", name, KF);
    return prefilter_launch(img, 1, H, W, pad, cpitch, coeff, s);
}

template <class T>
static int pad_one(const T *img, int H, int W, int pad, int cpitch, float *out, cudaStream_t s, const char *name) {
    D2IC_REQUIRE(img && out, "%s: null pointer", name);
    D2IC_REQUIRE(H > 0 && W > 0 && H < 65536 && W < 65536, "%s: bad image size %dx%d", name, H, W);
    D2IC_REQUIRE(pad >= 0 && cpitch >= W + 2 * pad, "%s: need cpitch >= W + 2 pad", name);
    const int CW = W + 2 * pad;
    pad_image_kernel<T><<<dim3((CW + 255) / 256, H + 2 * pad), 256, 0, s>>>(img, H, W, pad, cpitch, out);
    D2IC_CHECK_LAUNCH("pad_image");
    return D2IC_OK;
}

template <int KIND>
__global__ void sample_points_kernel(Img im, const float2 *__restrict__ xy, int n, float *val, float *gx,
                                     float *gy) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 p = xy[i];
    const float fx = safe_floor(p.x), fy = safe_floor(p.y);
    float a, b;
    const float v = sample<KIND>(im, (int)fx, (int)fy, p.x - fx, p.y - fy, a, b);
    val[i] = v;
    if (gx) gx[i] = a;
    if (gy) gy[i] = b;
}

template <int KIND>
__global__ void pack_pixels_kernel(const int2 *__restrict__ colrow, const float2 *__restrict__ xieta, int n,
                                   Img im, uint4 *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int2 cr = colrow[i];
    const float2 xe = xieta[i];
    float a, b;
    const float I1 = sample<KIND>(im, cr.x, cr.y, 0.f, 0.f, a, b);
    out[i] = make_uint4((uint32_t)cr.x | ((uint32_t)cr.y << 16), __float_as_uint(I1), __float_as_uint(xe.x),
                        __float_as_uint(xe.y));
}

}  // namespace d2ic

using namespace d2ic;

extern "C" int d2ic_bspline_prefilter_batch(const float *img, int n_images, int H, int W, int pad, int cpitch,
                                            float *tmp, float *coeff, void *stream) {
    D2IC_REQUIRE(img && tmp && coeff, "d2ic_bspline_prefilter_batch: null pointer");
    D2IC_REQUIRE(n_images >= 1 && n_images < 65536, "d2ic_bspline_prefilter_batch: bad image count %d", n_images);
    D2IC_REQUIRE(H > 0 && W > 0 && H < 65536 && W < 65536, "d2ic_bspline_prefilter_batch: bad image size %dx%d", H, W);
    D2IC_REQUIRE(pad >= KF && cpitch >= W + 2 * pad,
                 "d2ic_bspline_prefilter_batch: need pad >= %d and cpitch >= W + 2 pad", KF);
    return prefilter_launch(img, n_images, H, W, pad, cpitch, coeff, (cudaStream_t)stream);
}

extern "C" int d2ic_bspline_prefilter(const float *img, int H, int W, int pad, int cpitch, float *tmp,
                                      float *coeff, void *stream) {
    return prefilter_one(img, H, W, pad, cpitch, tmp, coeff, (cudaStream_t)stream, "d2ic_bspline_prefilter");
}

extern "C" int d2ic_bspline_prefilter_u8(const unsigned char *img, int H, int W, int pad, int cpitch, float *tmp,
                                         float *coeff, void *stream) {
    return prefilter_one(img, H, W, pad, cpitch, tmp, coeff, (cudaStream_t)stream, "d2ic_bspline_prefilter_u8");
}

extern "C" int d2ic_bspline_prefilter_gradients(const float *img, int H, int W, int pad, int cpitch, float *coeff,
                                                float *coeff_gx, float *coeff_gy, void *stream) {
    D2IC_REQUIRE(img && coeff && coeff_gx && coeff_gy, "d2ic_bspline_prefilter_gradients: null pointer");
    D2IC_REQUIRE(H > 0 && W > 0 && H < 65536 && W < 65536, "d2ic_bspline_prefilter_gradients: bad image size %dx%d", H, W);
    D2IC_REQUIRE(pad >= KF && cpitch >= W + 2 * pad,
                 "d2ic_bspline_prefilter_gradients: need pad >= %d and cpitch >= W + 2 pad", KF);
    return prefilter_launch<float, true>(img, 3, H, W, pad, cpitch, coeff, (cudaStream_t)stream, coeff_gx, coeff_gy);
}

extern "C" int d2ic_pad_image(const float *img, int H, int W, int pad, int cpitch, float *out, void *stream) {
    return pad_one(img, H, W, pad, cpitch, out, (cudaStream_t)stream, "d2ic_pad_image");
}

extern "C" int d2ic_pad_image_u8(const unsigned char *img, int H, int W, int pad, int cpitch, float *out,
                                 void *stream) {
    return pad_one(img, H, W, pad, cpitch, out, (cudaStream_t)stream, "d2ic_pad_image_u8");
}

extern "C" int d2ic_sample_points(const float *coeff, int H, int W, int pad, int cpitch, int kind, const float *xy,
                                  int n, float *val, float *gx, float *gy, void *stream) {
    D2IC_REQUIRE(coeff && xy && val, "d2ic_sample_points: null pointer");
    D2IC_REQUIRE(n >= 0 && H > 0 && W > 0 && pad >= 0 && cpitch >= W + 2 * pad, "d2ic_sample_points: bad sizes");
    D2IC_REQUIRE(kind == D2IC_INTERP_CUBIC || kind == D2IC_INTERP_LINEAR, "d2ic_sample_points: unknown kind %d", kind);
    if (n == 0) return D2IC_OK;
    Img im{coeff, W, H, cpitch, pad};
    const int nb = (n + 255) / 256;
    if (kind == D2IC_INTERP_CUBIC)
        sample_points_kernel<D2IC_INTERP_CUBIC><<<nb, 256, 0, (cudaStream_t)stream>>>(im, (const float2 *)xy, n, val, gx, gy);
    else
        sample_points_kernel<D2IC_INTERP_LINEAR><<<nb, 256, 0, (cudaStream_t)stream>>>(im, (const float2 *)xy, n, val, gx, gy);
    D2IC_CHECK_LAUNCH("sample_points");
    return D2IC_OK;
}

extern "C" int d2ic_pack_pixels(const int *colrow, const float *xieta, int n, const float *coeff1, int H, int W,
                                int pad, int cpitch, int kind, d2ic_pixrec_t *out, void *stream) {
    D2IC_REQUIRE(colrow && xieta && coeff1 && out, "d2ic_pack_pixels: null pointer");
    D2IC_REQUIRE(n >= 0 && H > 0 && W > 0 && H < 65536 && W < 65536 && cpitch >= W + 2 * pad,
                 "d2ic_pack_pixels: bad sizes");
    D2IC_REQUIRE(kind == D2IC_INTERP_CUBIC || kind == D2IC_INTERP_LINEAR, "d2ic_pack_pixels: unknown kind %d", kind);
    if (n == 0) return D2IC_OK;
    Img im{coeff1, W, H, cpitch, pad};
    const int nb = (n + 255) / 256;
    if (kind == D2IC_INTERP_CUBIC)
        pack_pixels_kernel<D2IC_INTERP_CUBIC><<<nb, 256, 0, (cudaStream_t)stream>>>((const int2 *)colrow, (const float2 *)xieta, n, im, (uint4 *)out);
    else
        pack_pixels_kernel<D2IC_INTERP_LINEAR><<<nb, 256, 0, (cudaStream_t)stream>>>((const int2 *)colrow, (const float2 *)xieta, n, im, (uint4 *)out);
    D2IC_CHECK_LAUNCH("pack_pixels");
    return D2IC_OK;
}
