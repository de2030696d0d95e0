// Shared device helpers of the d2ic_gb300 library (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/d2ic_gb300.h"

namespace d2ic {

// ---- error reporting (thread-local message behind d2ic_last_error_string) ----
void set_error(const char *fmt, ...);
int cuda_status(cudaError_t e, const char *what);

#define D2IC_CHECK_LAUNCH(what)                                       \
    do {                                                              \
        cudaError_t _e = cudaGetLastError();                          \
        if (_e != cudaSuccess) return ::d2ic::cuda_status(_e, what);  \
    } while (0)

#define D2IC_REQUIRE(cond, ...)                 \
    do {                                        \
        if (!(cond)) {                          \
            ::d2ic::set_error(__VA_ARGS__);     \
            return D2IC_BAD_ARG;                \
        }                                       \
    } while (0)

// Two FP32 values in a 64-bit register pair, and IEEE operations on both with one instruction
// (add/mul/fma.rn.f32x2): the same bits as two scalar operations in half the issue slots.
typedef unsigned long long Pair;
__device__ __forceinline__ Pair pair(float lo, float hi) {
    Pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ Pair pair(float v) { return pair(v, v); }
__device__ __forceinline__ float pair_lo(Pair p) { return __uint_as_float((unsigned)p); }
__device__ __forceinline__ float pair_hi(Pair p) { return __uint_as_float((unsigned)(p >> 32)); }
__device__ __forceinline__ Pair pair_fma(Pair a, Pair b, Pair c) {
    Pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ Pair pair_mul(Pair a, Pair b) {
    Pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) {
    Pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ Pair pair_add_down(Pair a, Pair b) {   // rounded towards minus infinity
    Pair r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The arithmetic shared by one pixel (float) and two pixels (Pair): the same operations, the same bits.
__device__ __forceinline__ float op_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float op_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float op_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ Pair op_add(Pair a, Pair b) { return pair_add(a, b); }
__device__ __forceinline__ Pair op_fma(Pair a, Pair b, Pair c) { return pair_fma(a, b, c); }
__device__ __forceinline__ Pair op_mul(Pair a, Pair b) { return pair_mul(a, b); }
template <class T> __device__ __forceinline__ T op_const(float v);
template <> __device__ __forceinline__ float op_const<float>(float v) { return v; }
template <> __device__ __forceinline__ Pair op_const<Pair>(float v) { return pair(v); }

// ---- cubic B-spline weights for taps -1..2 at fractional offset t in [0,1) ----
// w = ((1 - t)^3, 4 - 6 t^2 + 3 t^3, 1 + 3 t + 3 t^2 - 3 t^3, t^3) / 6, dw its derivative; the order of the
// operations is written out, so that one and two pixels give the same bits.  (A Horner form with 18 operations
// instead of 23 gains 1 % of a round at 2048 x 2048; other bits let a solve near its rounding floor stop some
// iterations earlier or later.)
template <class T>
__device__ __forceinline__ void bspline_w(T t, T w[4], T dw[4]) {
    const T s = op_const<T>(1.f / 6.f), three = op_const<T>(3.f), mone = op_const<T>(-1.f);
    const T o = op_fma(t, mone, op_const<T>(1.f)), t2 = op_mul(t, t), t3 = op_mul(t2, t);
    const T m3 = op_mul(op_const<T>(-3.f), t3);
    w[0] = op_mul(op_mul(op_mul(o, o), o), s);
    w[1] = op_mul(op_fma(op_fma(op_const<T>(6.f), t2, m3), mone, op_const<T>(4.f)), s);
    w[2] = op_mul(op_add(op_fma(three, t, op_fma(three, t2, m3)), op_const<T>(1.f)), s);
    w[3] = op_mul(t3, s);
    dw[0] = op_mul(op_mul(op_const<T>(-0.5f), o), o);
    dw[1] = op_fma(op_const<T>(1.5f), t2, op_mul(op_const<T>(-2.f), t));
    dw[2] = op_add(op_fma(op_const<T>(-1.5f), t2, t), op_const<T>(0.5f));
    dw[3] = op_mul(op_const<T>(0.5f), t2);
}

// The bilinear shape functions of an element at (xi, eta)
template <class T>
__device__ __forceinline__ void shape4(T xi, T eta, T N[4]) {
    const T half = op_const<T>(0.5f), mhalf = op_const<T>(-0.5f);
    const T a0 = op_fma(xi, mhalf, half), a1 = op_fma(xi, half, half);
    const T b0 = op_fma(eta, mhalf, half), b1 = op_fma(eta, half, half);
    N[0] = op_mul(a0, b0);
    N[1] = op_mul(a1, b0);
    N[2] = op_mul(a1, b1);
    N[3] = op_mul(a0, b1);
}
template <class T>
__device__ __forceinline__ T dot4(const T a[4], const T b[4]) {
    return op_fma(a[3], b[3], op_fma(a[2], b[2], op_fma(a[1], b[1], op_mul(a[0], b[0]))));
}
// a displacement component at a pixel
template <class T>
__device__ __forceinline__ T shape_sum(const T N[4], const T u[4]) {
    return op_fma(N[3], u[3], op_fma(N[2], u[2], op_fma(N[0], u[0], op_mul(N[1], u[1]))));
}

struct Img {
    const float *c;   // halo'd array
    int W, H, cp, pad;
    __device__ __forceinline__ float at(int r, int col) const {   // r, col: pixel indices (may be in the halo)
        return __ldg(c + (size_t)(r + pad) * cp + (col + pad));
    }
};

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return min(max(v, lo), hi); }

// The 4x4 tap arithmetic of the cubic B-spline, shared by every source of
// coefficients (global memory, clamped global, shared-memory tile) so that all
// paths produce identical bits.  Taps c[a][b]: row iy - 1 + a, column ix - 1 + b.
template <class T>
__device__ __forceinline__ T cubic_taps(const T c[4][4], T tx, T ty, T &gx, T &gy) {
    T wx[4], dwx[4], wy[4], dwy[4], rv[4], rd[4];
    bspline_w(tx, wx, dwx);
    bspline_w(ty, wy, dwy);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        rv[a] = dot4(wx, c[a]);
        rd[a] = dot4(dwx, c[a]);
    }
    gx = dot4(wy, rd);
    gy = dot4(dwy, rv);
    return dot4(wy, rv);
}

// Cubic B-spline value and gradient at pixel (ix + tx, iy + ty), with integer
// base (ix, iy) and fractional parts tx, ty in [0, 1).  Taps outside the halo'd
// array clamp to its border, where the coefficients equal the edge value.
__device__ __forceinline__ float sample_cubic(const Img &im, int ix, int iy, float tx, float ty,
                                              float &gx, float &gy) {
    float c[4][4];
    const int x0 = ix - 1, y0 = iy - 1;
    if (x0 >= -im.pad && x0 + 3 < im.W + im.pad && y0 >= -im.pad && y0 + 3 < im.H + im.pad) {
        const float *base = im.c + (size_t)(y0 + im.pad) * im.cp + (x0 + im.pad);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) c[a][b] = __ldg(base + (size_t)a * im.cp + b);
    } else {
        int cx[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) cx[b] = clampi(x0 + b, -im.pad, im.W - 1 + im.pad);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int r = clampi(y0 + a, -im.pad, im.H - 1 + im.pad);
#pragma unroll
            for (int b = 0; b < 4; ++b) c[a][b] = im.at(r, cx[b]);
        }
    }
    return cubic_taps(c, tx, ty, gx, gy);
}

// Same, with the taps read from a shared-memory tile whose element (0, 0) is the
// tap at (row ly, column lx) relative to the tile; the caller guarantees
// 0 <= lx <= tw - 4 and 0 <= ly <= th - 4.
__device__ __forceinline__ float sample_cubic_tile(const float *tile, int tw, int lx, int ly, float tx, float ty,
                                                   float &gx, float &gy) {
    float c[4][4];
    const float *base = tile + ly * tw + lx;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) c[a][b] = base[a * tw + b];
    return cubic_taps(c, tx, ty, gx, gy);
}

// Two pixels at once, with the taps at elements ia and ib of the tile.
__device__ __forceinline__ Pair sample_cubic_tile2(const float *tile, int tw, unsigned ia, unsigned ib, Pair tx, Pair ty,
                                                   Pair &gx, Pair &gy) {
    Pair c[4][4];
    const float *pa = tile + ia, *pb = tile + ib;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) c[a][b] = pair(pa[a * tw + b], pb[a * tw + b]);
    return cubic_taps(c, tx, ty, gx, gy);
}

// Bilinear value and gradient at pixel (ix + tx, iy + ty); taps clamped into the image.
__device__ __forceinline__ float sample_linear(const Img &im, int ix, int iy, float tx, float ty,
                                               float &gx, float &gy) {
    const int x0 = clampi(ix, 0, im.W - 1), x1 = clampi(ix + 1, 0, im.W - 1);
    const int y0 = clampi(iy, 0, im.H - 1), y1 = clampi(iy + 1, 0, im.H - 1);
    const float i00 = im.at(y0, x0), i10 = im.at(y0, x1), i01 = im.at(y1, x0), i11 = im.at(y1, x1);
    gx = (1.f - ty) * (i10 - i00) + ty * (i11 - i01);
    gy = (1.f - tx) * (i01 - i00) + tx * (i11 - i10);
    return (1.f - tx) * (1.f - ty) * i00 + tx * (1.f - ty) * i10 + (1.f - tx) * ty * i01 + tx * ty * i11;
}

template <int KIND>
__device__ __forceinline__ float sample(const Img &im, int ix, int iy, float tx, float ty, float &gx, float &gy) {
    if (KIND == D2IC_INTERP_LINEAR) return sample_linear(im, ix, iy, tx, ty, gx, gy);
    return sample_cubic(im, ix, iy, tx, ty, gx, gy);
}

// floor(d) clamped to +-2^24 before the integer conversion, so that huge or
// NaN coordinates give a far-outside (clamped) tap instead of a saturated
// integer that could overflow the bounds arithmetic.  NaN propagates through
// the fraction, never through an index.
__device__ __forceinline__ float safe_floor(float d) {
    return fminf(fmaxf(floorf(d), -16777216.0f), 16777216.0f);
}

// Split an image-index coordinate x = i + d (i integer pixel, d small
// displacement) into integer base and fraction in [0,1) without forming the
// rounded sum i + d.
__device__ __forceinline__ void split_coord(int i, float d, int &ib, float &t) {
    const float fl = safe_floor(d);
    ib = i + (int)fl;
    t = d - fl;
}

// Double-float ("hi + lo") accumulation: TwoSum / TwoProduct are error-free
// transformations in FP32 (Knuth; Ogita, Rump & Oishi, "Accurate sum and dot
// product", SIAM J. Sci. Comput. 2005), giving ~48-bit sums at FP32 issue
// rate.  GB300's FP64 pipe runs at a small fraction of FP32, so the inner
// products of the CG control are accumulated this way and converted to FP64
// once per group.  df_add is commutative bit for bit, so xor-butterfly warp
// reductions leave every lane with the same value.
struct DF {
    float hi, lo;
};
__device__ __forceinline__ DF df_two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ DF df_add(DF x, DF y) {
    const DF s = df_two_sum(x.hi, y.hi);
    const float e = s.lo + (x.lo + y.lo);
    const float h = s.hi + e;
    return {h, e - (h - s.hi)};
}
__device__ __forceinline__ DF df_prod(float a, float b) {
    const float p = a * b;
    return {p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ DF df_warp_sum(DF v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const DF w = {__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
        v = df_add(v, w);
    }
    return v;
}
__device__ __forceinline__ double df_to_double(DF v) { return (double)v.hi + (double)v.lo; }

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Orders this thread's earlier accesses (and those it has observed) before its later ones for the GPU:
// the acquire/release fence, lighter than __threadfence(), which is sequentially consistent.
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// 16-byte records that carry their own round tag: one 128-bit access is a single memory operation
// (ld/st.b128 of the PTX memory model), so a reader that finds the tag has the data of the same
// write.  A producer therefore needs no fence and no counter to hand over a record, and the
// consumer polls the record itself: one L2 round trip from the store to the value, instead of
// store, fence, atomic, polled counter, load.
__device__ __forceinline__ uint4 ld_record(const void *p) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
    return make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
}
__device__ __forceinline__ void st_record(void *p, uint4 v) {
    const unsigned long long lo = (unsigned long long)v.x | ((unsigned long long)v.y << 32);
    const unsigned long long hi = (unsigned long long)v.z | ((unsigned long long)v.w << 32);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(lo), "l"(hi)
                 : "memory");
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace d2ic
