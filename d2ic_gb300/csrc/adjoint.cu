// Implicit-function derivative of the converged solve (uncertainty propagation).
//
// At the converged u*, grad_u J(u*, I2) = 0 defines u*(I2); its derivative is
//     du* = -H^-1 (d grad_u J / dI2) dI,
// H the exact Hessian of J.  Kernels:
//   * hessian_chunks: one pixel pass at u*; per chunk the 10 distinct 2x2 blocks
//     N_a N_b (grad I2 grad I2^T + r hess I2) summed over the chunk's pixels
//     (3 numbers each: xx, xy, yy), i.e. the element Hessian of the pixel term;
//   * hv_chunks / hv_nodes: H V for K right-hand sides at once (V: n_nodes x 2 x K,
//     K fastest): chunk blocks times the chunk's 4 nodal vectors into the same
//     per-node slots the CG engine uses, then a node pass that sums the slots
//     and adds the spring Hessian (no atomics);
//   * mixed_chunks / slots_to_nodes: (d grad_u J / dI2) dI for an image
//     direction given by its B-spline coefficients;
//   * mixed_T_chunks + prefilter_T: the adjoint of that map (the backward of
//     the bicubic sampling): per pixel the coefficient-space weights, merged
//     along runs of pixels and scattered with atomics, then the transpose of
//     the clamped separable prefilter.
#include "common.cuh"

namespace d2ic {

constexpr int KF_T = 16;                    // prefilter half-length (matches image_ops.cu)
__constant__ float c_fir_t[2 * KF_T + 1];
__constant__ float c_cum_lo[2 * KF_T + 2];  // c_cum_lo[m + KF] = sum_{k <= m} h[k], m in [-KF, KF]
static bool g_firt_ready[64] = {false};

static int ensure_fir_t() {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && g_firt_ready[dev]) return D2IC_OK;
    float h[2 * KF_T + 1], cl[2 * KF_T + 2];
    const double z = 1.7320508075688772 - 2.0;
    double acc = 0.0;
    for (int k = -KF_T; k <= KF_T; ++k) {
        double v = 1.7320508075688772;
        for (int i = 0; i < (k < 0 ? -k : k); ++i) v *= z;
        h[k + KF_T] = (float)v;
    }
    for (int k = -KF_T; k <= KF_T; ++k) {
        acc += h[k + KF_T];
        cl[k + KF_T] = (float)acc;
    }
    cl[2 * KF_T + 1] = (float)acc;
    cudaError_t e = cudaMemcpyToSymbol(c_fir_t, h, sizeof(h));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_cum_lo, cl, sizeof(cl));
    if (e != cudaSuccess) return cuda_status(e, "adjoint constants");
    if (dev >= 0 && dev < 64) g_firt_ready[dev] = true;
    return D2IC_OK;
}

__device__ __forceinline__ void bspline_w2(float t, float w2[4]) {
    w2[0] = 1.f - t;
    w2[1] = 3.f * t - 2.f;
    w2[2] = -3.f * t + 1.f;
    w2[3] = t;
}

// value, gradient and Hessian of the cubic B-spline (taps clamped as the forward sampler)
__device__ __forceinline__ void sample_cubic_h(const Img &im, int ix, int iy, float tx, float ty, float o[6]) {
    float wx[4], dwx[4], wy[4], dwy[4], ddx[4], ddy[4];
    bspline_w(tx, wx, dwx);
    bspline_w(ty, wy, dwy);
    bspline_w2(tx, ddx);
    bspline_w2(ty, ddy);
    for (int i = 0; i < 6; ++i) o[i] = 0.f;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int r = clampi(iy - 1 + a, -im.pad, im.H - 1 + im.pad);
        float rv = 0.f, rd = 0.f, rdd = 0.f;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float c = im.at(r, clampi(ix - 1 + b, -im.pad, im.W - 1 + im.pad));
            rv += wx[b] * c;
            rd += dwx[b] * c;
            rdd += ddx[b] * c;
        }
        o[0] += wy[a] * rv;     // value
        o[1] += wy[a] * rd;     // d/dx
        o[2] += dwy[a] * rv;    // d/dy
        o[3] += wy[a] * rdd;    // d2/dx2
        o[4] += dwy[a] * rd;    // d2/dxdy
        o[5] += ddy[a] * rv;    // d2/dy2
    }
}

struct ChunkPix {
    int x, y;
    float I1, N[4];
};
__device__ __forceinline__ ChunkPix unpack(const uint4 r) {
    ChunkPix p;
    p.x = (int)(r.x & 0xffffu);
    p.y = (int)(r.x >> 16);
    p.I1 = __uint_as_float(r.y);
    const float xi = __uint_as_float(r.z), eta = __uint_as_float(r.w);
    const float a0 = 0.5f * (1.f - xi), a1 = 0.5f * (1.f + xi), b0 = 0.5f * (1.f - eta), b1 = 0.5f * (1.f + eta);
    p.N[0] = a0 * b0;
    p.N[1] = a1 * b0;
    p.N[2] = a1 * b1;
    p.N[3] = a0 * b1;
    return p;
}

__device__ __forceinline__ void chunk_nodes_u(const d2ic_frame_t &F, const float2 *u, int c, int lane, float ux[4],
                                              float uy[4], int &nd, int &slot) {
    float2 uc = make_float2(0.f, 0.f);
    nd = 0;
    slot = 0;
    if (lane < 4) {
        nd = __ldg(F.chunk_nodes + 4 * c + lane);
        slot = (int)(((unsigned)__ldg(F.chunk_slot + c) >> (8 * lane)) & 0xffu);
        uc = u[nd];
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        ux[a] = __shfl_sync(0xffffffffu, uc.x, a);
        uy[a] = __shfl_sync(0xffffffffu, uc.y, a);
    }
}

// pair (a <= b) index in 0..9
__device__ __forceinline__ int pair_index(int a, int b) { return a * 4 - (a * (a - 1)) / 2 + (b - a); }

__global__ void __launch_bounds__(256) hessian_chunks(const d2ic_frame_t *__restrict__ fp, const float2 *__restrict__ u,
                                                      int exact, float *__restrict__ out) {
    const d2ic_frame_t &F = *fp;
    const int lane = threadIdx.x & 31;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= F.n_chunks) return;
    float ux[4], uy[4];
    int nd, slot;
    chunk_nodes_u(F, u, c, lane, ux, uy, nd, slot);
    const Img im{F.coeff, F.W, F.H, F.cpitch, F.pad};
    float acc[30];
#pragma unroll
    for (int i = 0; i < 30; ++i) acc[i] = 0.f;
    const int pb = __ldg(F.chunk_begin + c), pe = __ldg(F.chunk_begin + c + 1);
    for (int p = pb + lane; p < pe; p += 32) {
        const ChunkPix q = unpack(__ldg(reinterpret_cast<const uint4 *>(F.pix) + p));
        const float dx = q.N[0] * ux[0] + q.N[1] * ux[1] + q.N[2] * ux[2] + q.N[3] * ux[3];
        const float dy = q.N[0] * uy[0] + q.N[1] * uy[1] + q.N[2] * uy[2] + q.N[3] * uy[3];
        int ix, iy;
        float tx, ty;
        split_coord(q.x, dx, ix, tx);
        split_coord(q.y, dy, iy, ty);
        float o[6];
        sample_cubic_h(im, ix, iy, tx, ty, o);
        const float r = o[0] - q.I1;
        float mxx = o[1] * o[1], mxy = o[1] * o[2], myy = o[2] * o[2];
        if (exact) {
            mxx += r * o[3];
            mxy += r * o[4];
            myy += r * o[5];
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = a; b < 4; ++b) {
                const float nn = q.N[a] * q.N[b];
                const int k = 3 * pair_index(a, b);
                acc[k] += nn * mxx;
                acc[k + 1] += nn * mxy;
                acc[k + 2] += nn * myy;
            }
    }
#pragma unroll
    for (int i = 0; i < 30; ++i) acc[i] = warp_sum_f(acc[i]);
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < 30; ++i) out[32 * (size_t)c + i] = acc[i];
        out[32 * (size_t)c + 30] = 0.f;
        out[32 * (size_t)c + 31] = 0.f;
    }
}

// H V, pixel part: for chunk c and right-hand side k, y_a = sum_b K_ab v_b into node slots.
// V, slots: (node, comp, k) with k fastest; slots: node_chunk_k planes of n_nodes * 2 * K.
__global__ void hv_chunks(const d2ic_frame_t *__restrict__ fp, const float *__restrict__ hess, const float *__restrict__ V,
                          int K, float *__restrict__ slots) {
    const d2ic_frame_t &F = *fp;
    const int c = blockIdx.x;
    __shared__ float Kc[32];
    __shared__ int s_nd[4], s_sl[4];
    if (threadIdx.x < 32) Kc[threadIdx.x] = hess[32 * (size_t)c + threadIdx.x];
    if (threadIdx.x < 4) {
        s_nd[threadIdx.x] = __ldg(F.chunk_nodes + 4 * c + threadIdx.x);
        s_sl[threadIdx.x] = (int)(((unsigned)__ldg(F.chunk_slot + c) >> (8 * threadIdx.x)) & 0xffu);
    }
    __syncthreads();
    const size_t Nn = F.n_nodes;
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        float vx[4], vy[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            vx[b] = V[((size_t)s_nd[b] * 2 + 0) * K + k];
            vy[b] = V[((size_t)s_nd[b] * 2 + 1) * K + k];
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            float yx = 0.f, yy = 0.f;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int pi = 3 * (a <= b ? pair_index(a, b) : pair_index(b, a));
                yx += Kc[pi] * vx[b] + Kc[pi + 1] * vy[b];
                yy += Kc[pi + 1] * vx[b] + Kc[pi + 2] * vy[b];
            }
            float *sp = slots + ((size_t)s_sl[a] * Nn + s_nd[a]) * 2 * K;
            sp[k] = yx;
            sp[K + k] = yy;
        }
    }
}

// H V, node part: slots (in slot order) / Np + alpha * spring Hessian V; Y (node, comp, k).
__global__ void hv_nodes(const d2ic_frame_t *__restrict__ fp, const float *__restrict__ slots, const float *__restrict__ V,
                         int K, float inv_np, float alpha, float *__restrict__ Y) {
    const d2ic_frame_t &F = *fp;
    const size_t Nn = F.n_nodes;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= Nn * K) return;
    const int n = (int)(t / K), k = (int)(t % K);
    float sx = 0.f, sy = 0.f;
    for (int s = 0; s < F.node_chunk_k; ++s) {
        const float *sp = slots + ((size_t)s * Nn + n) * 2 * K;
        sx += sp[k];
        sy += sp[K + k];
    }
    const float vx = V[((size_t)n * 2) * K + k], vy = V[((size_t)n * 2 + 1) * K + k];
    float rx = 0.f, ry = 0.f;
    for (int q = 0; q < F.max_deg; ++q) {
        const int j = __ldg(F.nbr_index + (size_t)q * Nn + n);
        if (j < 0) break;
        const float w = __ldg(F.nbr_weight + (size_t)q * Nn + n);
        rx += w * (vx - V[((size_t)j * 2) * K + k]);
        ry += w * (vy - V[((size_t)j * 2 + 1) * K + k]);
    }
    Y[((size_t)n * 2) * K + k] = sx * inv_np + alpha * rx;
    Y[((size_t)n * 2 + 1) * K + k] = sy * inv_np + alpha * ry;
}

// (d grad_u J / dI2) dI for the images of a batch, one block per chunk: its pixels are located and
// sampled in the frame once (position, residual r, gradient g; one pixel per thread, kept in shared
// memory), then every warp takes images: per pixel dv and grad dv of the image's
// coefficients at the same position, t = dv g + r grad dv, and the chunk's node sums N_a t (lane
// order, then a warp sum) into the image's node slots.  The frame sample is shared by all images
// of the batch instead of being repeated per image.
//
// A warp takes up to MIX images at a time (as few as give every warp some): their windows are copied to shared
// memory while the frame is sampled, and two pixels per lane and instruction are sampled from them with
// weights computed once for all of them.  64 images at 1024 x 1024 with 12-px elements took 478 us with one
// image at a time from global memory (16 loads per pixel and image of several cache lines each, the weights every
// time), now 394 us (two images at a time and three blocks per SM 419, one and four 457): 40 % of the multiply-add
// rate, the rest is the start of each block.  A window that does not fit (MIX_TILE floats) or leaves the halo'd array: global memory, one pixel at a time.
constexpr int MIX = 4, MIX_TILE = D2IC_TILE_MAX_FLOATS, MIX_WARPS = 8;

__device__ __forceinline__ void cp_async16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

__global__ void __launch_bounds__(32 * MIX_WARPS, 2) mixed_chunks(const d2ic_frame_t *__restrict__ fp,
                                                                  const float2 *__restrict__ u,
                                                                  const float *__restrict__ dcoeff,
                                                                  float2 *__restrict__ slots, size_t coeff_stride,
                                                                  size_t slot_stride, int n_images) {
    extern __shared__ __align__(16) float mix_smem[];
    __shared__ int s_at[D2IC_CHUNK_MAX], s_ix[D2IC_CHUNK_MAX], s_iy[D2IC_CHUNK_MAX];
    __shared__ float s_tx[D2IC_CHUNK_MAX], s_ty[D2IC_CHUNK_MAX];
    __shared__ float s_r[D2IC_CHUNK_MAX], s_gx[D2IC_CHUNK_MAX], s_gy[D2IC_CHUNK_MAX];
    __shared__ float s_N[4][D2IC_CHUNK_MAX];
    const d2ic_frame_t &F = *fp;
    const int c = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float *tiles = mix_smem + w * MIX * MIX_TILE;
    float ux[4], uy[4];
    int nd, slot;
    chunk_nodes_u(F, u, c, lane, ux, uy, nd, slot);
    const int pb = __ldg(F.chunk_begin + c), n = min(__ldg(F.chunk_begin + c + 1) - pb, D2IC_CHUNK_MAX);
    // the window: the pixel box moved by [floor(min u), floor(max u)] (0.5 px of slack) and the stencil, in
    // columns and rows of the halo'd array; its first column a multiple of 4 if rows can be copied 16 bytes at a time
    const bool wide = ((reinterpret_cast<uintptr_t>(dcoeff) & 15) | (coeff_stride & 3) | (F.cpitch & 3)) == 0;
    int x0, y0, tw, th;
    bool tiled;
    {
        const unsigned b0 = (unsigned)__ldg(F.chunk_box + 2 * c), b1 = (unsigned)__ldg(F.chunk_box + 2 * c + 1);
        bool fin = true;
#pragma unroll
        for (int a = 0; a < 4; ++a) fin = fin && isfinite(ux[a]) && isfinite(uy[a]);
        const float lox = fminf(fminf(ux[0], ux[1]), fminf(ux[2], ux[3])), hix = fmaxf(fmaxf(ux[0], ux[1]), fmaxf(ux[2], ux[3]));
        const float loy = fminf(fminf(uy[0], uy[1]), fminf(uy[2], uy[3])), hiy = fmaxf(fmaxf(uy[0], uy[1]), fmaxf(uy[2], uy[3]));
        x0 = (int)(b0 & 0xffffu) + (int)safe_floor(lox - 0.5f) - 1 + F.pad;
        y0 = (int)(b0 >> 16) + (int)safe_floor(loy - 0.5f) - 1 + F.pad;
        const int x1 = (int)(b1 & 0xffffu) + (int)safe_floor(hix + 0.5f) + 3 + F.pad;
        const int y1 = (int)(b1 >> 16) + (int)safe_floor(hiy + 0.5f) + 3 + F.pad;
        const bool in = x0 >= 0 && y0 >= 0 && x1 <= F.W + 2 * F.pad && y1 <= F.H + 2 * F.pad;
        if (wide) x0 &= ~3;
        tw = wide ? (x1 - x0 + 3) & ~3 : x1 - x0;
        th = y1 - y0;
        tiled = fin && in && tw >= 4 && th >= 4 && tw <= MIX_TILE / 4 && th <= MIX_TILE / 4 && tw * th <= MIX_TILE;
    }
    auto load_tile = [&](float *dst, const float *src) {   // src: element (y0, x0) of an image
        if (wide) {
            const int q = tw >> 2;
            int r = 0, k = lane;
            for (int i = lane; i < q * th; i += 32) {
                while (k >= q) {
                    k -= q;
                    ++r;
                }
                cp_async16(dst + 4 * i, src + (size_t)r * F.cpitch + 4 * k);
                k += 32;
            }
        } else {
            int r = 0, k = lane;
            for (int i = lane; i < tw * th; i += 32) {
                while (k >= tw) {
                    k -= tw;
                    ++r;
                }
                cp_async4(dst + i, src + (size_t)r * F.cpitch + k);
                k += 32;
            }
        }
    };
    const int per = min((n_images + MIX_WARPS - 1) / MIX_WARPS, MIX);   // images of a warp at a time
    const size_t origin = (size_t)y0 * F.cpitch + x0;
    if (tiled)
        for (int j = 0; j < per && w * per + j < n_images; ++j)
            load_tile(tiles + j * MIX_TILE, dcoeff + (size_t)(w * per + j) * coeff_stride + origin);
    bool inside = true;                                        // of the window
    if ((int)threadIdx.x < n) {
        const int i = threadIdx.x;
        const ChunkPix q = unpack(__ldg(reinterpret_cast<const uint4 *>(F.pix) + pb + i));
        const float dx = q.N[0] * ux[0] + q.N[1] * ux[1] + q.N[2] * ux[2] + q.N[3] * ux[3];
        const float dy = q.N[0] * uy[0] + q.N[1] * uy[1] + q.N[2] * uy[2] + q.N[3] * uy[3];
        int ix, iy;
        float tx, ty;
        split_coord(q.x, dx, ix, tx);
        split_coord(q.y, dy, iy, ty);
        const Img im{F.coeff, F.W, F.H, F.cpitch, F.pad};
        float gx, gy;
        s_r[i] = sample_cubic(im, ix, iy, tx, ty, gx, gy) - q.I1;
        s_gx[i] = gx;
        s_gy[i] = gy;
        const int lx = ix - 1 + F.pad - x0, ly = iy - 1 + F.pad - y0;
        inside = (unsigned)lx <= (unsigned)(tw - 4) && (unsigned)ly <= (unsigned)(th - 4);
        s_at[i] = ly * tw + lx;                                // the first tap's element of the window
        s_ix[i] = ix;
        s_iy[i] = iy;
        s_tx[i] = tx;
        s_ty[i] = ty;
#pragma unroll
        for (int a = 0; a < 4; ++a) s_N[a][i] = q.N[a];
    }
    // every pixel of an element lies inside; one beyond it (a caller's own shape functions) may not: global memory
    if (!__syncthreads_and(inside)) tiled = false;
    for (int b0 = w * per; b0 < n_images; b0 += MIX_WARPS * per) {
        const int nb = min(per, n_images - b0);
        float v[8 * MIX];                            // node sums: image j's x of node a at 8 j + 2 a, its y after it
#pragma unroll
        for (int i = 0; i < 8 * MIX; ++i) v[i] = 0.f;
        if (tiled) {
            if (b0 != w * per) {
                __syncwarp();                        // every lane is done with the last images' windows
                for (int j = 0; j < nb; ++j)
                    load_tile(tiles + j * MIX_TILE, dcoeff + (size_t)(b0 + j) * coeff_stride + origin);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
#pragma unroll 1
            for (int i0 = 0; i0 < n; i0 += 64) {
                const int ia = min(i0 + lane, n - 1), ib = min(i0 + lane + 32, n - 1);
                const float ga = i0 + lane < n ? 1.f : 0.f, gb = i0 + lane + 32 < n ? 1.f : 0.f;
                Pair wx[4], dwx[4], wy[4], dwy[4];
                bspline_w(pair(s_tx[ia], s_tx[ib]), wx, dwx);
                bspline_w(pair(s_ty[ia], s_ty[ib]), wy, dwy);
                const Pair r = pair(ga * s_r[ia], gb * s_r[ib]);
                const Pair gx = pair(ga * s_gx[ia], gb * s_gx[ib]), gy = pair(ga * s_gy[ia], gb * s_gy[ib]);
                const float *pa = tiles + s_at[ia], *pc = tiles + s_at[ib];
#pragma unroll
                for (int j = 0; j < MIX; ++j) {
                    if (j >= nb) break;
                    Pair rv[4], rd[4];
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        Pair t[4];
#pragma unroll
                        for (int x = 0; x < 4; ++x)
                            t[x] = pair(pa[j * MIX_TILE + y * tw + x], pc[j * MIX_TILE + y * tw + x]);
                        rv[y] = dot4(wx, t);
                        rd[y] = dot4(dwx, t);
                    }
                    const Pair dv = dot4(wy, rv), dgx = dot4(wy, rd), dgy = dot4(dwy, rv);
                    const Pair tx = pair_fma(r, dgx, pair_mul(dv, gx)), ty = pair_fma(r, dgy, pair_mul(dv, gy));
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        const float Na = s_N[a][ia], Nb = s_N[a][ib];
                        v[8 * j + 2 * a] = __fmaf_rn(Nb, pair_hi(tx), __fmaf_rn(Na, pair_lo(tx), v[8 * j + 2 * a]));
                        v[8 * j + 2 * a + 1] = __fmaf_rn(Nb, pair_hi(ty), __fmaf_rn(Na, pair_lo(ty), v[8 * j + 2 * a + 1]));
                    }
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < MIX; ++j) {
                if (j >= nb) break;
                const Img dm{dcoeff + (size_t)(b0 + j) * coeff_stride, F.W, F.H, F.cpitch, F.pad};
                for (int i = lane; i < n; i += 32) {
                    float dgx, dgy;
                    const float dv = sample_cubic(dm, s_ix[i], s_iy[i], s_tx[i], s_ty[i], dgx, dgy);
                    const float r = s_r[i];
                    const float txv = __fmaf_rn(r, dgx, __fmul_rn(dv, s_gx[i]));
                    const float tyv = __fmaf_rn(r, dgy, __fmul_rn(dv, s_gy[i]));
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        v[8 * j + 2 * a] = __fmaf_rn(s_N[a][i], txv, v[8 * j + 2 * a]);
                        v[8 * j + 2 * a + 1] = __fmaf_rn(s_N[a][i], tyv, v[8 * j + 2 * a + 1]);
                    }
                }
            }
        }
        // the warp sums by a reduce-scatter: at each step over a lane bit a lane keeps half of its values and adds
        // its partner's copy of that half; lane l ends with value l
        static_assert(8 * MIX == 32, "one sum per lane");
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int q = 0; q < o; ++q) {
                const float give = up ? v[q] : v[q + o], keep = up ? v[q + o] : v[q];
                v[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        const int j = lane >> 3, a = (lane >> 1) & 3;
        const int nda = __shfl_sync(0xffffffffu, nd, a), sla = __shfl_sync(0xffffffffu, slot, a);
        if (j < nb)
            reinterpret_cast<float *>(slots + (size_t)(b0 + j) * slot_stride + (size_t)sla * F.n_nodes + nda)[lane & 1] = v[0];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");       // windows of a chunk that did without them
}

// Few images: one image per warp, from global memory, with more blocks per SM and no windows to copy.  The same bits.
__global__ void __launch_bounds__(256) mixed_chunks_few(const d2ic_frame_t *__restrict__ fp, const float2 *__restrict__ u,
                                                    const float *__restrict__ dcoeff, float2 *__restrict__ slots,
                                                    size_t coeff_stride, size_t slot_stride, int n_images) {
    __shared__ int s_ix[D2IC_CHUNK_MAX], s_iy[D2IC_CHUNK_MAX];
    __shared__ float s_tx[D2IC_CHUNK_MAX], s_ty[D2IC_CHUNK_MAX];
    __shared__ float s_r[D2IC_CHUNK_MAX], s_gx[D2IC_CHUNK_MAX], s_gy[D2IC_CHUNK_MAX];
    __shared__ float s_N[4][D2IC_CHUNK_MAX];
    const d2ic_frame_t &F = *fp;
    const int c = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float ux[4], uy[4];
    int nd, slot;
    chunk_nodes_u(F, u, c, lane, ux, uy, nd, slot);
    const int pb = __ldg(F.chunk_begin + c), n = min(__ldg(F.chunk_begin + c + 1) - pb, D2IC_CHUNK_MAX);
    if ((int)threadIdx.x < n) {
        const int i = threadIdx.x;
        const ChunkPix q = unpack(__ldg(reinterpret_cast<const uint4 *>(F.pix) + pb + i));
        const float dx = q.N[0] * ux[0] + q.N[1] * ux[1] + q.N[2] * ux[2] + q.N[3] * ux[3];
        const float dy = q.N[0] * uy[0] + q.N[1] * uy[1] + q.N[2] * uy[2] + q.N[3] * uy[3];
        int ix, iy;
        float tx, ty;
        split_coord(q.x, dx, ix, tx);
        split_coord(q.y, dy, iy, ty);
        const Img im{F.coeff, F.W, F.H, F.cpitch, F.pad};
        float gx, gy;
        s_r[i] = sample_cubic(im, ix, iy, tx, ty, gx, gy) - q.I1;
        s_gx[i] = gx;
        s_gy[i] = gy;
        s_ix[i] = ix;
        s_iy[i] = iy;
        s_tx[i] = tx;
        s_ty[i] = ty;
#pragma unroll
        for (int a = 0; a < 4; ++a) s_N[a][i] = q.N[a];
    }
    __syncthreads();
    for (int b = w; b < n_images; b += 8) {
        const Img dm{dcoeff + (size_t)b * coeff_stride, F.W, F.H, F.cpitch, F.pad};
        float ax[4] = {0.f, 0.f, 0.f, 0.f}, ay[4] = {0.f, 0.f, 0.f, 0.f};
        for (int i = lane; i < n; i += 32) {
            float dgx, dgy;
            const float dv = sample_cubic(dm, s_ix[i], s_iy[i], s_tx[i], s_ty[i], dgx, dgy);
            const float r = s_r[i];
            const float txv = __fmaf_rn(r, dgx, __fmul_rn(dv, s_gx[i])), tyv = __fmaf_rn(r, dgy, __fmul_rn(dv, s_gy[i]));
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                ax[a] = __fmaf_rn(s_N[a][i], txv, ax[a]);
                ay[a] = __fmaf_rn(s_N[a][i], tyv, ay[a]);
            }
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            ax[a] = warp_sum_f(ax[a]);
            ay[a] = warp_sum_f(ay[a]);
        }
        if (lane < 4) {
            const float gx = lane == 0 ? ax[0] : lane == 1 ? ax[1] : lane == 2 ? ax[2] : ax[3];
            const float gy = lane == 0 ? ay[0] : lane == 1 ? ay[1] : lane == 2 ? ay[2] : ay[3];
            slots[(size_t)b * slot_stride + (size_t)slot * F.n_nodes + nd] = make_float2(gx, gy);
        }
    }
}

// Up to 16 images the few-images form: at 1024 x 1024 with 10-px elements, coefficients included, 1 image 92 us against
// 123 us from windows, 6 images 144 and 172, 16 images 270 and 273; 24 images 372 and 337, 64 images 910 and 772.
constexpr int MIX_FEW = 17;
constexpr int MIX_SMEM = MIX_WARPS * MIX * MIX_TILE * (int)sizeof(float);
static int mixed_launch(const d2ic_frame_t *frame_dev, int n_chunks, const float *u, const float *dcoeff, float *slots,
                        size_t coeff_stride, size_t slot_stride, int n_images, cudaStream_t s) {
    if (n_images < MIX_FEW) {
        mixed_chunks_few<<<n_chunks, 256, 0, s>>>(frame_dev, (const float2 *)u, dcoeff, (float2 *)slots, coeff_stride,
                                                  slot_stride, n_images);
        D2IC_CHECK_LAUNCH("mixed_chunks_few");
        return D2IC_OK;
    }
    const cudaError_t e = cudaFuncSetAttribute(mixed_chunks, cudaFuncAttributeMaxDynamicSharedMemorySize, MIX_SMEM);
    if (e != cudaSuccess) return cuda_status(e, "mixed_chunks");
    mixed_chunks<<<n_chunks, 32 * MIX_WARPS, MIX_SMEM, s>>>(frame_dev, (const float2 *)u, dcoeff, (float2 *)slots,
                                                           coeff_stride, slot_stride, n_images);
    D2IC_CHECK_LAUNCH("mixed_chunks");
    return D2IC_OK;
}

// node sum of float2 slots, scaled; writes column k of out (node, comp, K)
__global__ void slots_to_nodes(const d2ic_frame_t *__restrict__ fp, const float2 *__restrict__ slots, float scale,
                               float *__restrict__ out, int K, int k0, size_t slot_stride) {
    const d2ic_frame_t &F = *fp;
    slots += blockIdx.y * slot_stride;                 // image blockIdx.y of a batch -> column k0 + y
    const int k = k0 + (int)blockIdx.y;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= F.n_nodes) return;
    float sx = 0.f, sy = 0.f;
    for (int s = 0; s < F.node_chunk_k; ++s) {
        const float2 v = slots[(size_t)s * F.n_nodes + n];
        sx += v.x;
        sy += v.y;
    }
    out[((size_t)n * 2) * K + k] = sx * scale;
    out[((size_t)n * 2 + 1) * K + k] = sy * scale;
}

// Adjoint of mixed for the K nodal fields of a batch, one warp per chunk: its pixels are located and
// sampled in the frame once (kept in shared memory); then per field the weights of
// lambda . (d grad_u J / dI2) on the 16 coefficient taps of every pixel are added to the field's
// coefficients with atomics.  Within a step of 32 pixels, lanes whose stencil corners follow one another
// along a row hand their taps to the lane that owns the column, so that a run of pixels adds each
// coefficient of a row once instead of four times.
//
// Bound by the L2's atomics: six fields at 777 x 901 98 us one field at a time with 16 atomics per pixel,
// 65 us now (summed in a shared-memory tile per chunk instead: 169 us, a chain of dependent reads and
// writes per tap).
constexpr int MT_WARPS = 4;
__global__ void __launch_bounds__(32 * MT_WARPS) mixed_T_chunks(const d2ic_frame_t *__restrict__ fp,
                                                                const float2 *__restrict__ u,
                                                                const float *__restrict__ lam, int K, float scale,
                                                                float *__restrict__ gcoeff, size_t stride) {
    __shared__ float s_tx[MT_WARPS][D2IC_CHUNK_MAX], s_ty[MT_WARPS][D2IC_CHUNK_MAX], s_gx[MT_WARPS][D2IC_CHUNK_MAX],
        s_gy[MT_WARPS][D2IC_CHUNK_MAX], s_r[MT_WARPS][D2IC_CHUNK_MAX], s_xi[MT_WARPS][D2IC_CHUNK_MAX],
        s_eta[MT_WARPS][D2IC_CHUNK_MAX];
    __shared__ int2 s_at[MT_WARPS][D2IC_CHUNK_MAX];     // stencil corner
    const d2ic_frame_t &F = *fp;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    if (c >= F.n_chunks) return;
    float ux[4], uy[4];
    int nd, slot;
    chunk_nodes_u(F, u, c, lane, ux, uy, nd, slot);
    const Img im{F.coeff, F.W, F.H, F.cpitch, F.pad};
    const int pb = __ldg(F.chunk_begin + c), n = min(__ldg(F.chunk_begin + c + 1) - pb, D2IC_CHUNK_MAX);
    for (int i = lane; i < n; i += 32) {
        const uint4 rec = __ldg(reinterpret_cast<const uint4 *>(F.pix) + pb + i);
        const ChunkPix q = unpack(rec);
        const float dx = q.N[0] * ux[0] + q.N[1] * ux[1] + q.N[2] * ux[2] + q.N[3] * ux[3];
        const float dy = q.N[0] * uy[0] + q.N[1] * uy[1] + q.N[2] * uy[2] + q.N[3] * uy[3];
        int ix, iy;
        float tx, ty;
        split_coord(q.x, dx, ix, tx);
        split_coord(q.y, dy, iy, ty);
        float gx, gy;
        s_r[w][i] = sample_cubic(im, ix, iy, tx, ty, gx, gy) - q.I1;
        s_gx[w][i] = gx;
        s_gy[w][i] = gy;
        s_tx[w][i] = tx;
        s_ty[w][i] = ty;
        s_xi[w][i] = __uint_as_float(rec.z);
        s_eta[w][i] = __uint_as_float(rec.w);
        s_at[w][i] = make_int2(ix - 1, iy - 1);
    }
    __syncwarp();
    for (int k = 0; k < K; ++k) {
        float2 l = make_float2(0.f, 0.f);
        if (lane < 4) l = make_float2(__ldg(lam + ((size_t)nd * 2) * K + k), __ldg(lam + ((size_t)nd * 2 + 1) * K + k));
        float lx[4], ly[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            lx[a] = __shfl_sync(0xffffffffu, l.x, a);
            ly[a] = __shfl_sync(0xffffffffu, l.y, a);
        }
        float *out = gcoeff + (size_t)k * stride;
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const bool on = i < n;
            const int2 at = on ? s_at[w][i] : make_int2(1 << 28, 1 << 28);
            float wx[4] = {0.f, 0.f, 0.f, 0.f}, dwx[4], wy[4] = {0.f, 0.f, 0.f, 0.f}, dwy[4], gl = 0.f, rlx = 0.f, rly = 0.f;
#pragma unroll
            for (int a = 0; a < 4; ++a) dwx[a] = dwy[a] = 0.f;
            if (on) {
                const float xi = s_xi[w][i], eta = s_eta[w][i];
                const float a0 = 0.5f * (1.f - xi), a1 = 0.5f * (1.f + xi), c0 = 0.5f * (1.f - eta), c1 = 0.5f * (1.f + eta);
                const float N[4] = {a0 * c0, a1 * c0, a1 * c1, a0 * c1};
                const float Lx = N[0] * lx[0] + N[1] * lx[1] + N[2] * lx[2] + N[3] * lx[3];
                const float Ly = N[0] * ly[0] + N[1] * ly[1] + N[2] * ly[2] + N[3] * ly[3];
                bspline_w(s_tx[w][i], wx, dwx);
                bspline_w(s_ty[w][i], wy, dwy);
                const float r = s_r[w][i];
                gl = (s_gx[w][i] * Lx + s_gy[w][i] * Ly) * scale;
                rlx = r * Lx * scale;
                rly = r * Ly * scale;
            }
            // taps 1 .. t of this lane go to the lanes behind it, whose corners follow this one
            const int nx = __shfl_down_sync(0xffffffffu, at.x, 1), ny = __shfl_down_sync(0xffffffffu, at.y, 1);
            const unsigned next = __ballot_sync(0xffffffffu, lane < 31 && nx == at.x + 1 && ny == at.y) >> lane;
            const int t = (next & 1u) == 0u ? 0 : (next & 2u) == 0u ? 1 : (next & 4u) == 0u ? 2 : 3;
            const int back1 = __shfl_up_sync(0xffffffffu, t, 1), back2 = __shfl_up_sync(0xffffffffu, t, 2),
                      back3 = __shfl_up_sync(0xffffffffu, t, 3);
            const int x0 = clampi(at.x, -im.pad, im.W - 1 + im.pad) + im.pad;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                float *row = out + (size_t)(clampi(at.y + a, -im.pad, im.H - 1 + im.pad) + im.pad) * im.cp;
                float v[4];
#pragma unroll
                for (int b = 0; b < 4; ++b) v[b] = wy[a] * wx[b] * gl + wy[a] * dwx[b] * rlx + dwy[a] * wx[b] * rly;
                const float v1 = __shfl_up_sync(0xffffffffu, v[1], 1), v2 = __shfl_up_sync(0xffffffffu, v[2], 2),
                            v3 = __shfl_up_sync(0xffffffffu, v[3], 3);
                if (lane >= 1 && back1 >= 1) v[0] += v1;
                if (lane >= 2 && back2 >= 2) v[0] += v2;
                if (lane >= 3 && back3 >= 3) v[0] += v3;
                if (on) {
                    atomicAdd(row + x0, v[0]);
#pragma unroll
                    for (int b = 1; b < 4; ++b)
                        if (t < b) atomicAdd(row + clampi(at.x + b, -im.pad, im.W - 1 + im.pad) + im.pad, v[b]);
                }
            }
        }
    }
}

// Transpose of one clamped FIR pass.  Forward: out[i] = sum_k h[k] in[clamp(i - pad + k, 0, n - 1)] for i in
// [0, n + 2 pad); transposed: in'[j] = sum_k h[k] out'[j + pad - k] for 0 < j < n - 1, and the two edge
// samples collect every tap that the clamp sent to them.
__device__ __forceinline__ float fir_T_low(const float *src, size_t step, int in_len, int pad) {    // taps that clamp to 0
    float acc = 0.f;
    for (int i = 0; i < in_len && i <= pad + KF_T; ++i) acc += c_cum_lo[min(pad - i, KF_T) + KF_T] * src[(size_t)i * step];
    return acc;
}
__device__ __forceinline__ float fir_T_high(const float *src, size_t step, int in_len, int pad, int n) {   // ... to n - 1
    float acc = 0.f;
    for (int i = in_len - 1; i >= 0; --i) {
        const int m = n - 1 + pad - i;                 // taps k >= m
        if (m > KF_T) break;
        const float below = m - 1 >= -KF_T ? c_cum_lo[min(m - 1, KF_T) + KF_T] : 0.f;
        acc += (c_cum_lo[2 * KF_T] - below) * src[(size_t)i * step];
    }
    return acc;
}

// Column pass, image blockIdx.z: out (n rows) from in (n + 2 pad rows), every one of the CW columns.  A block
// takes TT_W columns x TT_H rows, staged once with the 2 KF_T rows around them; a thread makes TT_R
// consecutive rows of a column from a sliding window (the layout of the forward pass; one output per
// thread along the column read with a stride of a row and took 54 us per pass at 777 x 901).
constexpr int TT_W = 32, TT_H = 128, TT_R = TT_H / 8;
__global__ void __launch_bounds__(256) prefilter_T_cols(const float *__restrict__ in, int n, int CW, int pad, int cpitch,
                                                       size_t in_stride, float *__restrict__ out, size_t out_stride) {
    __shared__ float s[TT_H + 2 * KF_T][TT_W + 1];
    in += (size_t)blockIdx.z * in_stride;
    out += (size_t)blockIdx.z * out_stride;
    const int cx = blockIdx.x * TT_W + threadIdx.x, j0 = blockIdx.y * TT_H, in_len = n + 2 * pad;
    for (int r = threadIdx.y; r < TT_H + 2 * KF_T; r += 8) {
        const int i = j0 + pad - KF_T + r;
        s[r][threadIdx.x] = cx < CW && i >= 0 && i < in_len ? in[(size_t)i * cpitch + cx] : 0.f;
    }
    __syncthreads();
    if (cx >= CW) return;
    const int r0 = threadIdx.y * TT_R;
    float acc[TT_R];
#pragma unroll
    for (int o = 0; o < TT_R; ++o) acc[o] = 0.f;
#pragma unroll
    for (int t = 0; t < TT_R + 2 * KF_T; ++t) {
        const float v = s[r0 + t][threadIdx.x];
#pragma unroll
        for (int o = 0; o < TT_R; ++o) {
            const int k = t - o;                       // h is symmetric
            if (k >= 0 && k <= 2 * KF_T) acc[o] += c_fir_t[k] * v;
        }
    }
#pragma unroll
    for (int o = 0; o < TT_R; ++o) {
        const int j = j0 + r0 + o;
        if (j > 0 && j < n - 1) out[(size_t)j * cpitch + cx] = acc[o];
        else if (j == 0) out[cx] = fir_T_low(in + cx, cpitch, in_len, pad);
        else if (j == n - 1) out[(size_t)j * cpitch + cx] = fir_T_high(in + cx, cpitch, in_len, pad, n);
    }
}

// Row pass, image blockIdx.z: out (W columns) from in (W + 2 pad columns).  A block takes an even share (at
// most TR_OUT outputs, a multiple of 4) of one row, staged with its 2 KF_T neighbours; a thread makes 4
// consecutive outputs from float4 reads.
constexpr int TR_OUT = 4096;
__global__ void __launch_bounds__(1024) prefilter_T_rows(const float *__restrict__ in, int H, int W, int pad, int cpitch,
                                                        size_t in_stride, float *__restrict__ out, size_t out_stride) {
    __shared__ __align__(16) float s[TR_OUT + 2 * KF_T + 4];
    in += (size_t)blockIdx.z * in_stride + (size_t)blockIdx.y * cpitch;
    out += (size_t)blockIdx.z * out_stride + (size_t)blockIdx.y * W;
    const int CW = W + 2 * pad, per = (((W + gridDim.x - 1) / gridDim.x) + 3) & ~3;
    const int x0 = blockIdx.x * per, n_out = min(per, W - x0);
    for (int i = threadIdx.x; i < ((n_out + 3) & ~3) + 2 * KF_T + 4; i += blockDim.x) {
        const int c = x0 + pad - KF_T + i;
        s[i] = c >= 0 && c < CW ? __ldg(in + c) : 0.f;
    }
    __syncthreads();
    const int o0 = 4 * threadIdx.x;
    if (o0 < n_out) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        const float4 *s4 = reinterpret_cast<const float4 *>(s) + threadIdx.x;
#pragma unroll
        for (int m = 0; m < (2 * KF_T + 4) / 4 + 1; ++m) {
            const float4 q = s4[m];
            const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int o = 0; o < 4; ++o) {
                    const int k = 4 * m + e - o;
                    if (k >= 0 && k <= 2 * KF_T) acc[o] += c_fir_t[k] * v[e];
                }
        }
#pragma unroll
        for (int o = 0; o < 4; ++o) {
            const int j = x0 + o0 + o;
            if (o0 + o < n_out && j > 0 && j < W - 1) out[j] = acc[o];
        }
    }
    // the edge samples, a tap per lane of the first warp
    if (threadIdx.x < 32 && x0 == 0) {
        float acc = 0.f;
        for (int i = threadIdx.x; i < CW && i <= pad + KF_T; i += 32) acc += c_cum_lo[min(pad - i, KF_T) + KF_T] * in[i];
        acc = warp_sum_f(acc);
        if (threadIdx.x == 0) out[0] = acc;
    }
    if (threadIdx.x < 32 && x0 + n_out == W) {
        float acc = 0.f;
        for (int i = max(W - 1 + pad - KF_T, 0) + threadIdx.x; i < CW; i += 32) {   // taps k >= m
            const int m = W - 1 + pad - i;
            acc += (c_cum_lo[2 * KF_T] - (m - 1 >= -KF_T ? c_cum_lo[min(m - 1, KF_T) + KF_T] : 0.f)) * in[i];
        }
        acc = warp_sum_f(acc);
        if (threadIdx.x == 0) out[W - 1] = acc;
    }
}

}  // namespace d2ic

using namespace d2ic;

extern "C" int d2ic_hessian_chunks(const d2ic_frame_t *frame_dev, int n_chunks, const float *u, int exact,
                                   float *chunk_hess, void *stream) {
    D2IC_REQUIRE(frame_dev && u && chunk_hess && n_chunks >= 0, "d2ic_hessian_chunks: bad arguments");
    if (n_chunks == 0) return D2IC_OK;
    hessian_chunks<<<(n_chunks * 32 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(frame_dev, (const float2 *)u, exact,
                                                                                  chunk_hess);
    D2IC_CHECK_LAUNCH("hessian_chunks");
    return D2IC_OK;
}

extern "C" int d2ic_hessian_matvec(const d2ic_frame_t *frame_dev, int n_chunks, int n_nodes, const float *chunk_hess,
                                   const float *V, int K, float inv_np, float alpha_reg, float *slots, float *Y,
                                   void *stream) {
    D2IC_REQUIRE(frame_dev && chunk_hess && V && slots && Y && K >= 1 && n_nodes >= 1, "d2ic_hessian_matvec: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    if (n_chunks > 0) {
        hv_chunks<<<n_chunks, K < 128 ? 32 * ((K + 31) / 32) : 128, 0, s>>>(frame_dev, chunk_hess, V, K, slots);
        D2IC_CHECK_LAUNCH("hv_chunks");
    }
    const size_t nt = (size_t)n_nodes * K;
    hv_nodes<<<(unsigned)((nt + 255) / 256), 256, 0, s>>>(frame_dev, slots, V, K, inv_np, alpha_reg, Y);
    D2IC_CHECK_LAUNCH("hv_nodes");
    return D2IC_OK;
}

extern "C" int d2ic_mixed_term(const d2ic_frame_t *frame_dev, int n_chunks, int n_nodes, const float *u,
                               const float *dcoeff, float scale, float *slots, float *out, int K, int k, void *stream) {
    D2IC_REQUIRE(frame_dev && u && dcoeff && slots && out && K >= 1 && k >= 0 && k < K && n_nodes >= 1,
                 "d2ic_mixed_term: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    if (n_chunks > 0) {
        const int st = mixed_launch(frame_dev, n_chunks, u, dcoeff, slots, 0, 0, 1, s);
        if (st) return st;
    }
    slots_to_nodes<<<(n_nodes + 255) / 256, 256, 0, s>>>(frame_dev, (const float2 *)slots, scale, out, K, k, 0);
    D2IC_CHECK_LAUNCH("slots_to_nodes");
    return D2IC_OK;
}

extern "C" int d2ic_mixed_term_batch(const d2ic_frame_t *frame_dev, int n_chunks, int n_nodes, int node_chunk_k,
                                     const float *u, const float *dcoeff, int n_images, long long coeff_stride,
                                     float scale, float *slots, float *out, int K, int k0, void *stream) {
    D2IC_REQUIRE(frame_dev && u && dcoeff && slots && out && n_nodes >= 1 && node_chunk_k >= 1 && n_images >= 1 &&
                     n_images < 65536 && k0 >= 0 && k0 + n_images <= K && coeff_stride > 0,
                 "d2ic_mixed_term_batch: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    const size_t slot_stride = (size_t)node_chunk_k * n_nodes;   // float2 per image
    if (n_chunks > 0) {
        const int st = mixed_launch(frame_dev, n_chunks, u, dcoeff, slots, (size_t)coeff_stride, slot_stride, n_images, s);
        if (st) return st;
    }
    slots_to_nodes<<<dim3((n_nodes + 255) / 256, n_images), 256, 0, s>>>(frame_dev, (const float2 *)slots, scale, out,
                                                                         K, k0, slot_stride);
    D2IC_CHECK_LAUNCH("slots_to_nodes");
    return D2IC_OK;
}

extern "C" int d2ic_mixed_term_T_batch(const d2ic_frame_t *frame_dev, int n_chunks, const float *u, const float *lam,
                                       int K, float scale, float *gcoeff, long long coeff_stride, void *stream) {
    D2IC_REQUIRE(frame_dev && u && lam && gcoeff && K >= 1 && n_chunks >= 0 && (coeff_stride > 0 || K == 1),
                 "d2ic_mixed_term_T_batch: bad arguments");
    if (n_chunks == 0) return D2IC_OK;
    mixed_T_chunks<<<(n_chunks + MT_WARPS - 1) / MT_WARPS, 32 * MT_WARPS, 0, (cudaStream_t)stream>>>(
        frame_dev, (const float2 *)u, lam, K, scale, gcoeff, (size_t)coeff_stride);
    D2IC_CHECK_LAUNCH("mixed_T_chunks");
    return D2IC_OK;
}

extern "C" int d2ic_mixed_term_T(const d2ic_frame_t *frame_dev, int n_chunks, const float *u, const float *lam,
                                 float scale, float *gcoeff, void *stream) {
    D2IC_REQUIRE(frame_dev && u && lam && gcoeff, "d2ic_mixed_term_T: bad arguments");
    return d2ic_mixed_term_T_batch(frame_dev, n_chunks, u, lam, 1, scale, gcoeff, 0, stream);
}

extern "C" int d2ic_bspline_prefilter_T_batch(const float *gcoeff, int n_images, int H, int W, int pad, int cpitch,
                                              float *tmp, float *gimg, void *stream) {
    D2IC_REQUIRE(gcoeff && tmp && gimg, "d2ic_bspline_prefilter_T_batch: null pointer");
    D2IC_REQUIRE(n_images >= 1 && n_images < 65536, "d2ic_bspline_prefilter_T_batch: bad image count %d", n_images);
    D2IC_REQUIRE(H > 1 && W > 1 && H < 65536 && pad >= KF_T && cpitch >= W + 2 * pad,
                 "d2ic_bspline_prefilter_T_batch: bad sizes");
    int st = ensure_fir_t();
    if (st) return st;
    cudaStream_t s = (cudaStream_t)stream;
    const int CW = W + 2 * pad;
    // transpose of the column pass: gcoeff (H + 2 pad rows) -> tmp (H rows), every column of the halo'd width
    prefilter_T_cols<<<dim3((CW + TT_W - 1) / TT_W, (H + TT_H - 1) / TT_H, n_images), dim3(TT_W, 8), 0, s>>>(
        gcoeff, H, CW, pad, cpitch, (size_t)(H + 2 * pad) * cpitch, tmp, (size_t)H * cpitch);
    D2IC_CHECK_LAUNCH("prefilter_T_cols");
    // transpose of the row pass: tmp (CW columns) -> gimg (W columns), every row
    const int blocks = (W + TR_OUT - 1) / TR_OUT, per = (((W + blocks - 1) / blocks) + 3) & ~3;
    prefilter_T_rows<<<dim3(blocks, H, n_images), ((per / 4 + 31) / 32) * 32, 0, s>>>(
        tmp, H, W, pad, cpitch, (size_t)H * cpitch, gimg, (size_t)H * W);
    D2IC_CHECK_LAUNCH("prefilter_T_rows");
    return D2IC_OK;
}

extern "C" int d2ic_bspline_prefilter_T(const float *gcoeff, int H, int W, int pad, int cpitch, float *tmp, float *gimg,
                                        void *stream) {
    return d2ic_bspline_prefilter_T_batch(gcoeff, 1, H, W, pad, cpitch, tmp, gimg, stream);
}
