// Initial motion: integer-translation ZNCC search at element centres and
// inverse-distance projection of the centre displacements onto the nodes.
//
// ZNCC (d2ic/solver_translation_zncc.py:89-168): one block per centre; the
// template (win x win) and the search patch ((win + 2 s)^2) are staged in
// shared memory.  The score of an offset is the mean product of the normalised
// template t and the normalised window, first maximum in row-major (ky, kx)
// order.
//
// With the patch centred once (d = patch - c), an offset needs sum d t over its
// window, and sum d and sum d^2 for its mean and variance:
//   * the products are a register-blocked correlation: a thread makes
//     2 x R offsets (two rows of R), and per template value reads two patch
//     values and one template value from shared memory for 2 R multiply-adds;
//   * the two sums come from separable running sums in double-float, rounded to
//     FP32 once per row; v = sum d^2 - (sum d)^2 / n in double-float.
// With s = sum d^2 / v = 1 + (mean - c)^2 / variance of a window, the rows' rounding is amplified s-fold in v and
// the rounding of sum d t sqrt(s)-fold; the two-pass form (mean first, then centred sums, one after the other in
// FP32) has errors that grow with the window.  Simulated RMS errors of the score, correlations 0.3 and 0.99, against
// those of the two-pass form: win 5 1.0 at s = 2, 1.3 at 5; win 11 0.95 at 5, 1.2 at 10; win 21 0.9 at 10, 1.2 at 37;
// win 41 0.9 at 17, 1.0 at 62.  Windows with s above 0.15 win^1.5 (or 65) are therefore scored in two passes, by a
// thread each, or by a warp each where they are few; so is every window of a patch with values that are not finite
// or beyond 1e15.
//
// Bound by FP32 issue and shared-memory reads.  9,216 centres at win 41,
// search 24 (2401 offsets x 1681 pixels): 14.2 ms with one offset per thread in
// the two-pass form (5 instructions and 3 shared-memory reads per pixel and
// offset), 2.39 ms blocked with scalar multiply-adds, 2.07 ms with two offsets
// per instruction (fma.rn.f32x2).  16,384 centres at win 17, search 8: 743 ->
// 365 us; staging and running sums weigh more there.
#include "common.cuh"

namespace d2ic {

// the two-pass score of one offset: window mean, then centred sums
__device__ __forceinline__ float zncc_two_pass(const float *w0, int ps, const float *tpl, int win) {
    const float n = (float)(win * win);
    float s = 0.f;
    for (int i = 0; i < win; ++i)
#pragma unroll 4
        for (int j = 0; j < win; ++j) s += w0[i * ps + j];
    const float mw = s / n;
    float v = 0.f, cr = 0.f;
    for (int i = 0; i < win; ++i)
#pragma unroll 4
        for (int j = 0; j < win; ++j) {
            const float d = w0[i * ps + j] - mw;
            v += d * d;
            cr += d * tpl[i * win + j];
        }
    return cr / (sqrtf(v / n) + 1e-12f) / n;
}

// the same by a whole warp
__device__ __forceinline__ float zncc_two_pass_warp(const float *w0, int ps, const float *tpl, int win, int lane) {
    const int n = win * win;
    auto pixels = [&](auto &&f) {
        for (int p = lane, r = 0, q = lane; p < n; p += 32, q += 32) {
            while (q >= win) {
                q -= win;
                ++r;
            }
            f(w0[r * ps + q], p);
        }
    };
    float s = 0.f;
    pixels([&](float d, int) { s += d; });
    const float mw = warp_sum_f(s) / (float)n;
    float v = 0.f, cr = 0.f;
    pixels([&](float x, int p) {
        const float d = x - mw;
        v += d * d;
        cr += d * tpl[p];
    });
    v = warp_sum_f(v);
    return warp_sum_f(cr) / (sqrtf(v / (float)n) + 1e-12f) / (float)n;
}

// The offsets of a block with var < 0, in two passes: listed over the means, then a warp each where they are fewer than
// the warps times the steps that a warp saves, else a thread each.  Updates the thread's best score and its
// offset.  (Out of line: inlined, it changes how the correlation is compiled, 6 % of the whole at win 41.)
__device__ __noinline__ void zncc_left_over(const float *pat, int ps, const float *tpl, int win, int npa, const float *var,
                                            int *list, int *count, float &best, int &bidx) {
    const int n = win * win, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    auto better = [&](float sc, int o) {                   // not visited in order
        if (sc > best || (sc == best && o < bidx)) {
            best = sc;
            bidx = o;
        }
    };
    __syncthreads();                                       // every thread has read its means
    if (threadIdx.x == 0) *count = 0;
    __syncthreads();
    for (int o = threadIdx.x; o < npa * npa; o += blockDim.x)
        if (var[o] < 0.f) list[atomicAdd(count, 1)] = o;
    __syncthreads();
    const int left = *count;
    if ((long long)left * 64 <= (long long)nw * n) {
        for (int i = wid; i < left; i += nw) {
            const int o = list[i];
            const float sc = zncc_two_pass_warp(pat + (o / npa) * ps + o % npa, ps, tpl, win, lane);
            if (lane == 0) better(sc, o);
        }
    } else {
        for (int i = threadIdx.x; i < left; i += blockDim.x) {
            const int o = list[i];
            better(zncc_two_pass(pat + (o / npa) * ps + o % npa, ps, tpl, win), o);
        }
    }
}

// a float added to a double-float whose low word collects the rounding errors
__device__ __forceinline__ void df_acc(DF &a, float x) {
    const DF s = df_two_sum(a.hi, x);
    a.hi = s.hi;
    a.lo += s.lo;
}

// Running sums along one line: out[k] = sum_{i < win} f(k + i) for k in [k0, k1), f(i) a double-float
// (or, with an exact low word of 0, a float).
template <class F, class O>
__device__ __forceinline__ void running_sums(int k0, int k1, int win, F &&f, O &&out) {
    DF a = {0.f, 0.f};
    for (int i = 0; i < win; ++i) f(k0 + i, [&](float x) { df_acc(a, x); });
    for (int k = k0;;) {
        out(k, a);
        if (++k >= k1) break;
        f(k - 1, [&](float x) { df_acc(a, -x); });
        f(k + win - 1, [&](float x) { df_acc(a, x); });
    }
}

constexpr int ZNCC_SEG = 7;   // outputs per thread of a running sum
constexpr int ZNCC_MAX_THREADS = 384, ZNCC_TPT = 2;   // column tasks per thread

template <int R>
__global__ void __launch_bounds__(ZNCC_MAX_THREADS) zncc_kernel(const float *__restrict__ ref, int Hr, int Wr,
                                                                const float *__restrict__ def, int Hd, int Wd,
                                                                const float2 *__restrict__ centers, int win,
                                                                int search, float2 *__restrict__ u_out,
                                                                float *__restrict__ score_out) {
    extern __shared__ float sm[];
    const int ps = win + 2 * search, npa = 2 * search + 1;
    const int n = win * win, np2 = npa * npa;
    float *tpl = sm;                 // win * win, normalised template
    float *pat = sm + n;             // ps * ps, centred patch (one spare row of R values for the last block's reads)
    float *row1 = pat + ps * ps + R, *row2 = row1 + ps * npa;   // row sums of d and d^2: ps x npa
    float *mean = row1, *var = row1 + np2;                      // over them: window mean and n * variance
    __shared__ float s_red[32];
    __shared__ int s_idx[32];
    const int c = blockIdx.x;
    const float2 ctr = centers[c];
    // half to even, as jnp.rint; non-finite or far-away centres fail the bounds test below
    const bool finite = fabsf(ctr.x) < 1e7f && fabsf(ctr.y) < 1e7f;
    const int x = finite ? (int)rintf(ctr.x) : -(1 << 28), y = finite ? (int)rintf(ctr.y) : -(1 << 28);
    const int r = win / 2;
    const bool tpl_ok = (y - r >= 0) && (y + r < Hr) && (x - r >= 0) && (x + r < Wr);
    const int xs = x - search, ys = y - search, xe = x + search, ye = y + search;
    const bool patch_ok = (ys - r >= 0) && (ye + r < Hd) && (xs - r >= 0) && (xe + r < Wd);
    if (!(tpl_ok && patch_ok)) {
        if (threadIdx.x == 0) {
            u_out[c] = make_float2(0.f, 0.f);
            score_out[c] = __int_as_float(0x7fc00000);
        }
        return;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    auto block_sum = [&](float a) {
        a = warp_sum_f(a);
        __syncthreads();
        if (lane == 0) s_red[wid] = a;
        __syncthreads();
        float t = 0.f;
        for (int w = 0; w < nw; ++w) t += s_red[w];
        return t;
    };
    float a = 0.f, pa = 0.f;
    bool odd = false;                // a value that the running sums cannot take
    for (int i = wid; i < win; i += nw)
        for (int j = lane; j < win; j += 32) {
            const float t = __ldg(ref + (size_t)(y - r + i) * Wr + (x - r + j));
            tpl[i * win + j] = t;
            odd |= !(fabsf(t) < 1e15f);
            a += t;
        }
    for (int i = wid; i < ps; i += nw)
        for (int j = lane; j < ps; j += 32) {
            const float t = __ldg(def + (size_t)(ys - r + i) * Wd + (xs - r + j));
            pat[i * ps + j] = t;
            odd |= !(fabsf(t) < 1e15f);
            pa += t;
        }
    odd = __syncthreads_or(odd);
    // template mean and population std (two passes)
    const float mu = block_sum(a) / (float)n;
    a = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float d = tpl[i] - mu;
        a += d * d;
    }
    const float inv = 1.0f / (sqrtf(block_sum(a) / (float)n) + 1e-12f);
    float t1 = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float t = (tpl[i] - mu) * inv;
        tpl[i] = t;
        t1 += t;
    }
    t1 = block_sum(t1);              // zero but for rounding
    float best = -INFINITY;
    int bidx = 0x7fffffff;
    auto take = [&](float sc, int o) {
        if (sc > best || (sc != sc && best == best)) {   // NaN wins, as argmax
            best = sc;
            bidx = o;
        }
    };
    if (odd) {
        __syncthreads();
        for (int o = threadIdx.x; o < np2; o += blockDim.x)
            take(zncc_two_pass(pat + (o / npa) * ps + o % npa, ps, tpl, win), o);
    } else {
        const float pc = block_sum(pa) / (float)(ps * ps);
        for (int i = threadIdx.x; i < ps * ps; i += blockDim.x) pat[i] -= pc;
        if ((int)threadIdx.x < R) pat[ps * ps + threadIdx.x] = 0.f;
        __syncthreads();
        const int segs = (npa + ZNCC_SEG - 1) / ZNCC_SEG;
        const float most = fminf(0.15f * (float)win * sqrtf((float)win), 65.f);   // of sum d^2 / v
        // rows: sums over win columns (a thread: one row, ZNCC_SEG columns; neighbouring threads take
        // neighbouring rows)
        for (int t = threadIdx.x; t < 2 * ps * segs; t += blockDim.x) {
            const bool sq = t >= ps * segs;
            const int q = sq ? t - ps * segs : t, row = q % ps, k0 = (q / ps) * ZNCC_SEG;
            const float *src = pat + row * ps;
            float *dst = (sq ? row2 : row1) + row * npa;
            if (sq)
                running_sums(k0, min(k0 + ZNCC_SEG, npa), win,
                             [&](int i, auto &&add) {
                                 const DF p = df_prod(src[i], src[i]);
                                 add(p.hi);
                                 add(p.lo);
                             },
                             [&](int k, const DF &v) { dst[k] = v.hi + v.lo; });
            else
                running_sums(k0, min(k0 + ZNCC_SEG, npa), win, [&](int i, auto &&add) { add(src[i]); },
                             [&](int k, const DF &v) { dst[k] = v.hi + v.lo; });
        }
        __syncthreads();
        // columns: the window sums, kept in registers until every thread has read its rows (mean and var
        // lie over the rows).  A task is one column, ZNCC_SEG rows; at most ZNCC_TPT per thread.
        float wm[ZNCC_TPT][ZNCC_SEG], wv[ZNCC_TPT][ZNCC_SEG];
        bool two_pass = false;
#pragma unroll
        for (int h = 0; h < ZNCC_TPT; ++h) {
            const int task = threadIdx.x + h * blockDim.x, kx = task % npa, ky0 = (task / npa) * ZNCC_SEG;
            if (task < npa * segs) {
                DF s1 = {0.f, 0.f}, s2 = {0.f, 0.f};
                for (int i = 0; i < win; ++i) {
                    df_acc(s1, row1[(ky0 + i) * npa + kx]);
                    df_acc(s2, row2[(ky0 + i) * npa + kx]);
                }
#pragma unroll
                for (int q = 0; q < ZNCC_SEG; ++q) {
                    // n * variance = sum d^2 - (sum d)^2 / n, negative where the window needs the two-pass form
                    const float hi = s1.hi + s1.lo, lo = s1.lo - (hi - s1.hi), m = hi / (float)n;
                    const float rest = __fmaf_rn(-m, (float)n, hi) + lo;        // sum d - n m
                    const DF sq = df_prod(m, hi);
                    const DF d = df_add(s2, DF{-sq.hi, -(sq.lo + m * (lo + rest))});
                    const float v = d.hi + d.lo;
                    wm[h][q] = m;
                    wv[h][q] = v * most >= s2.hi + s2.lo ? fmaxf(v, 0.f) : -1.f;
                    if (ky0 + q + 1 < npa && q + 1 < ZNCC_SEG) {
                        df_acc(s1, -row1[(ky0 + q) * npa + kx]);
                        df_acc(s1, row1[(ky0 + q + win) * npa + kx]);
                        df_acc(s2, -row2[(ky0 + q) * npa + kx]);
                        df_acc(s2, row2[(ky0 + q + win) * npa + kx]);
                    }
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < ZNCC_TPT; ++h) {
            const int task = threadIdx.x + h * blockDim.x, kx = task % npa, ky0 = (task / npa) * ZNCC_SEG;
            if (task < npa * segs)
#pragma unroll
                for (int q = 0; q < ZNCC_SEG; ++q)
                    if (ky0 + q < npa) {
                        mean[(ky0 + q) * npa + kx] = wm[h][q];
                        var[(ky0 + q) * npa + kx] = wv[h][q];
                        two_pass |= wv[h][q] < 0.f;
                    }
        }
        two_pass = __syncthreads_or(two_pass);
        // the correlation: 2 rows x R columns of offsets per thread
        const int nbx = (npa + R - 1) / R, nby = (npa + 1) / 2;
        for (int t = threadIdx.x; t < nbx * nby; t += blockDim.x) {
            // rows ky and ky + nby: neighbouring threads read neighbouring rows, an odd number of words apart
            const int ky = t % nby, kx0 = (t / nby) * R;
            const bool two = ky + nby < npa;
            const float *p0 = pat + ky * ps + kx0, *p1 = two ? p0 + nby * ps : p0;
            Pair acc[R];
#pragma unroll
            for (int q = 0; q < R; ++q) acc[q] = pair(0.f, 0.f);
            for (int i = 0; i < win; ++i, p0 += ps, p1 += ps) {
                const float *ti = tpl + i * win;
                Pair w[R];                                 // sliding window: column j + q at (j + q) % R
#pragma unroll
                for (int q = 0; q < R - 1; ++q) w[q] = pair(p0[q], p1[q]);
                auto column = [&](int j, int q) {          // q = j mod R, known at compile time
                    const Pair tv = pair(ti[j], ti[j]);
                    w[(q + R - 1) % R] = pair(p0[j + R - 1], p1[j + R - 1]);
#pragma unroll
                    for (int o = 0; o < R; ++o) acc[o] = pair_fma(w[(q + o) % R], tv, acc[o]);
                };
                int j = 0;
                // R = 7 unrolled takes 4 % more with many centres (9,216 at 41 / 24: 2.16 ms), 3 % less with 625; the
                // others take 1 to 20 % less unrolled (49 centres at 41 / 12: 49 and 60 us)
                if constexpr (R == 7) {
#pragma unroll 1
                    for (; j + R <= win; j += R)
#pragma unroll
                        for (int q = 0; q < R; ++q) column(j + q, q);
                } else {
                    for (; j + R <= win; j += R)
#pragma unroll
                        for (int q = 0; q < R; ++q) column(j + q, q);
                }
#pragma unroll
                for (int q = 0; q < R - 1; ++q)             // the last win % R columns
                    if (j + q < win) column(j + q, q);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (h == 0 || two)
#pragma unroll
                    for (int q = 0; q < R; ++q)
                        if (kx0 + q < npa) {
                            const int o = (ky + h * nby) * npa + kx0 + q;
                            const float v = var[o], cr = (h == 0 ? pair_lo(acc[q]) : pair_hi(acc[q])) - mean[o] * t1;
                            const float sc = cr / (sqrtf(v / (float)n) + 1e-12f) / (float)n;
                            if (v >= 0.f && (sc > best || (sc == best && o < bidx))) {   // not visited in order
                                best = sc;
                                bidx = o;
                            }
                        }
        }
        if (two_pass) zncc_left_over(pat, ps, tpl, win, npa, var, reinterpret_cast<int *>(mean), s_idx, best, bidx);
    }
    // block argmax: larger score, then smaller index
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bidx, off);
        if (ob > best || (ob == best && oi < bidx)) {
            best = ob;
            bidx = oi;
        }
    }
    __syncthreads();
    if (lane == 0) {
        s_red[wid] = best;
        s_idx[wid] = bidx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = s_red[0];
        int bi = s_idx[0];
        for (int w = 1; w < nw; ++w)
            if (s_red[w] > b || (s_red[w] == b && s_idx[w] < bi)) {
                b = s_red[w];
                bi = s_idx[w];
            }
        const int ky = bi / npa, kx = bi % npa;
        u_out[c] = make_float2((float)(xs + kx - x), (float)(ys + ky - y));
        score_out[c] = b;
    }
}

// Windows and search ranges beyond what zncc_kernel's row sums and tasks hold: one offset per thread.
__global__ void __launch_bounds__(1024) zncc_wide_kernel(const float *__restrict__ ref, int Hr, int Wr, const float *__restrict__ def, int Hd,
                            int Wd, const float2 *__restrict__ centers, int win, int search, float2 *__restrict__ u_out,
                            float *__restrict__ score_out) {
    extern __shared__ float sm[];
    const int ps = win + 2 * search;
    float *tpl = sm;                 // win * win, normalised template
    float *pat = sm + win * win;     // ps * ps
    __shared__ float s_red[32];
    __shared__ int s_idx[32];
    __shared__ float s_mean, s_inv;
    const int c = blockIdx.x;
    const float2 ctr = centers[c];
    // half to even, as jnp.rint; non-finite or far-away centres fail the bounds test below
    const bool finite = fabsf(ctr.x) < 1e7f && fabsf(ctr.y) < 1e7f;
    const int x = finite ? (int)rintf(ctr.x) : -(1 << 28), y = finite ? (int)rintf(ctr.y) : -(1 << 28);
    const int r = win / 2;
    const bool tpl_ok = (y - r >= 0) && (y + r < Hr) && (x - r >= 0) && (x + r < Wr);
    const int xs = x - search, ys = y - search, xe = x + search, ye = y + search;
    const bool patch_ok = (ys - r >= 0) && (ye + r < Hd) && (xs - r >= 0) && (xe + r < Wd);
    if (!(tpl_ok && patch_ok)) {
        if (threadIdx.x == 0) {
            u_out[c] = make_float2(0.f, 0.f);
            score_out[c] = __int_as_float(0x7fc00000);
        }
        return;
    }
    const int n = win * win;
    for (int i = threadIdx.x; i < n; i += blockDim.x) tpl[i] = __ldg(ref + (size_t)(y - r + i / win) * Wr + (x - r + i % win));
    for (int i = threadIdx.x; i < ps * ps; i += blockDim.x)
        pat[i] = __ldg(def + (size_t)(ys - r + i / ps) * Wd + (xs - r + i % ps));
    __syncthreads();
    // template mean and population std (two passes)
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float a = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) a += tpl[i];
    a = warp_sum_f(a);
    if (lane == 0) s_red[wid] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < nw; ++w) t += s_red[w];
        s_mean = t / (float)n;
    }
    __syncthreads();
    const float mu = s_mean;
    a = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float d = tpl[i] - mu;
        a += d * d;
    }
    a = warp_sum_f(a);
    __syncthreads();
    if (lane == 0) s_red[wid] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < nw; ++w) t += s_red[w];
        s_inv = 1.0f / (sqrtf(t / (float)n) + 1e-12f);
    }
    __syncthreads();
    const float inv = s_inv;
    for (int i = threadIdx.x; i < n; i += blockDim.x) tpl[i] = (tpl[i] - mu) * inv;
    __syncthreads();
    // score every offset
    const int npa = 2 * search + 1;
    float best = -INFINITY;
    int bidx = 0x7fffffff;
    for (int o = threadIdx.x; o < npa * npa; o += blockDim.x) {
        const int ky = o / npa, kx = o % npa;
        const float *w0 = pat + ky * ps + kx;
        float s = 0.f;
        for (int i = 0; i < win; ++i)
            for (int j = 0; j < win; ++j) s += w0[i * ps + j];
        const float mw = s / (float)n;
        float v = 0.f, cr = 0.f;
        for (int i = 0; i < win; ++i)
            for (int j = 0; j < win; ++j) {
                const float d = w0[i * ps + j] - mw;
                v += d * d;
                cr += d * tpl[i * win + j];
            }
        const float sc = cr / (sqrtf(v / (float)n) + 1e-12f) / (float)n;
        if (sc > best || (sc != sc && best == best)) {   // NaN wins, as argmax
            best = sc;
            bidx = o;
        }
    }
    // block argmax: larger score, then smaller index
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bidx, off);
        if (ob > best || (ob == best && oi < bidx)) {
            best = ob;
            bidx = oi;
        }
    }
    __syncthreads();
    if (lane == 0) {
        s_red[wid] = best;
        s_idx[wid] = bidx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = s_red[0];
        int bi = s_idx[0];
        for (int w = 1; w < nw; ++w)
            if (s_red[w] > b || (s_red[w] == b && s_idx[w] < bi)) {
                b = s_red[w];
                bi = s_idx[w];
            }
        const int ky = bi / npa, kx = bi % npa;
        u_out[c] = make_float2((float)(xs + kx - x), (float)(ys + ky - y));
        score_out[c] = b;
    }
}

// IDW (power p) of centre displacements onto nodes: one warp per NPW nodes (8 warps per block; 4
// nodes on large meshes, 1 where 4 would leave SMs idle), the centres staged in shared-memory tiles
// of 256 that the block's warps share; lane l takes centres l, l + 32, ... of each tile against all
// of the warp's nodes, so one centre read serves NPW pairs.  FP64 sqrt/divide are slow on GB300, so per-pair math is FP32 (squared
// distances of pixel-grid coordinates are exact in FP32 up to 2^24) with the reciprocal correctly
// rounded; each lane sums a tile (8 centres) in FP32 and adds that into FP64 accumulators, and the
// lanes' FP64 sums are reduced over the warp at the end.  A centre closer than 1e-6 gives the node
// its displacement: the smallest such centre index, tracked without a branch (its infinite weight
// is discarded).  Centres with a NaN displacement are dropped.
constexpr int IDW_TILE = 256;
template <int IDW_NODES>
__global__ void __launch_bounds__(256) idw_kernel(const float2 *__restrict__ nodes, int n_nodes,
                                                  const float2 *__restrict__ centers, const float2 *__restrict__ disp,
                                                  int nc, float power, float2 *__restrict__ out) {
    __shared__ float2 sc[IDW_TILE], sd[IDW_TILE];
    const int lane = threadIdx.x & 31;
    const int i0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * IDW_NODES;
    float2 p[IDW_NODES];
    double sw[IDW_NODES], sx[IDW_NODES], sy[IDW_NODES];
    int ex[IDW_NODES];
#pragma unroll
    for (int j = 0; j < IDW_NODES; ++j) {
        p[j] = (i0 + j < n_nodes) ? nodes[i0 + j] : make_float2(0.f, 0.f);
        sw[j] = sx[j] = sy[j] = 0.0;
        ex[j] = 0x7fffffff;
    }
    const bool p2 = (power == 2.0f);
    for (int base = 0; base < nc; base += IDW_TILE) {
        const int m = min(IDW_TILE, nc - base);
        __syncthreads();
        if ((int)threadIdx.x < m) {
            sc[threadIdx.x] = centers[base + threadIdx.x];
            sd[threadIdx.x] = disp[base + threadIdx.x];
        }
        __syncthreads();
        if (i0 >= n_nodes) continue;
        float tw[IDW_NODES], tx[IDW_NODES], ty[IDW_NODES];
#pragma unroll
        for (int j = 0; j < IDW_NODES; ++j) tw[j] = tx[j] = ty[j] = 0.f;
        for (int k = lane; k < m; k += 32) {
            const float2 d = sd[k];
            if (d.x != d.x || d.y != d.y) continue;      // centres with NaN displacement are dropped
            const float2 c = sc[k];
#pragma unroll
            for (int j = 0; j < IDW_NODES; ++j) {
                const float dx = c.x - p[j].x, dy = c.y - p[j].y;
                const float d2 = dx * dx + dy * dy;
                ex[j] = d2 < 1e-12f ? min(ex[j], base + k) : ex[j];   // dist < 1e-6
                const float w = p2 ? __frcp_rn(d2) : powf(sqrtf(d2), -power);
                tw[j] += w;
                tx[j] += w * d.x;
                ty[j] += w * d.y;
            }
        }
#pragma unroll
        for (int j = 0; j < IDW_NODES; ++j) {
            sw[j] += (double)tw[j];
            sx[j] += (double)tx[j];
            sy[j] += (double)ty[j];
        }
    }
    if (i0 >= n_nodes) return;
#pragma unroll
    for (int j = 0; j < IDW_NODES; ++j) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sw[j] += __shfl_xor_sync(0xffffffffu, sw[j], o);
            sx[j] += __shfl_xor_sync(0xffffffffu, sx[j], o);
            sy[j] += __shfl_xor_sync(0xffffffffu, sy[j], o);
            ex[j] = min(ex[j], __shfl_xor_sync(0xffffffffu, ex[j], o));
        }
        if (lane == j && i0 + j < n_nodes) {
            if (ex[j] != 0x7fffffff) out[i0 + j] = disp[ex[j]];
            else if (sw[j] > 0.0) out[i0 + j] = make_float2((float)(sx[j] / sw[j]), (float)(sy[j] / sw[j]));
            else out[i0 + j] = make_float2(0.f, 0.f);
        }
    }
}

}  // namespace d2ic

using namespace d2ic;

extern "C" int d2ic_zncc_match(const float *ref, int Hr, int Wr, const float *def, int Hd, int Wd,
                               const float *centers, int n_centers, int win, int search, float *u_out,
                               float *score_out, void *stream) {
    D2IC_REQUIRE(ref && def && u_out && score_out && (centers || n_centers == 0), "d2ic_zncc_match: null pointer");
    D2IC_REQUIRE(win > 0 && (win % 2) == 1, "d2ic_zncc_match: win must be odd and positive (got %d)", win);
    D2IC_REQUIRE(search >= 0 && n_centers >= 0 && Hr > 0 && Wr > 0 && Hd > 0 && Wd > 0, "d2ic_zncc_match: bad sizes");
    const size_t base = (size_t)win * win + (size_t)(win + 2 * search) * (win + 2 * search);
    D2IC_REQUIRE(sizeof(float) * base <= 200 * 1024, "d2ic_zncc_match: win/search too large for shared memory (%zu bytes)",
                 sizeof(float) * base);
    if (n_centers == 0) return D2IC_OK;
    // R columns of offsets per thread: the fewest multiply-adds on columns beyond the search range
    const int npa = 2 * search + 1, ps = win + 2 * search;
    auto blocks = [&](int R) { return (npa + R - 1) / R; };
    int R = 7;
    for (int q = 6; q >= 5; --q)
        if (blocks(q) * q < blocks(R) * R) R = q;
    const int tasks = blocks(R) * ((npa + 1) / 2);
    int threads = ((tasks + 31) / 32) * 32;
    threads = threads < 64 ? 64 : (threads > ZNCC_MAX_THREADS ? ZNCC_MAX_THREADS : threads);
    const size_t smem = sizeof(float) * (base + R + 2 * (size_t)ps * npa);
    // The register-blocked form where its row sums fit in shared memory and its column tasks in the block
    // (search <= 34 at win 41); the wide form, one offset per thread, beyond, and where there is too little to do
    // for the blocked form's running sums: below 24,000 pixels x offsets per centre (10,000 centres, win 11: search 4
    // 64 us wide, 129 us blocked; search 6 124 and 149; search 8 203 and 153), or, with fewer centres than SMs,
    // below 300,000 (49 centres, win 21: search 6 27 and 32 us, win 31: search 8 40 and 44, search 12 54 and 41); with
    // windows up to 15 pixels also for more centres, up to 300,000 per SM (speckle, 289 centres: win 11 search 12 27 and
    // 31 us, win 15 search 10 26 and 32; 625: win 11 search 8 26 and 35, search 10 28 and 37, win 15 search 10 42 and 41;
    // 1,225: win 11 search 8 34 and 36, search 10 47 and 39).
    // Windows below 9 pixels, most of which go through the two-pass form anyway: wide (speckle, 10,000 centres,
    // search 24: win 5 469 us wide, 738 us blocked; win 7 660 and 754; win 9 917 and 695).
    int dev = 0, sms = 0;
    cudaError_t de = cudaGetDevice(&dev);
    if (de == cudaSuccess) de = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (de != cudaSuccess) return cuda_status(de, "d2ic_zncc_match");
    const long long work = (long long)npa * npa * win * win;
    const bool little =
        work < 24000 || (work < 300000 && (n_centers <= sms || (win <= 15 && work * n_centers < 300000ll * sms)));
    if (win >= 9 && !little && smem <= 200 * 1024 && npa * ((npa + ZNCC_SEG - 1) / ZNCC_SEG) <= ZNCC_TPT * threads) {
        auto launch = [&](auto kernel) {
            if (smem > 48 * 1024) {
                cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                if (e != cudaSuccess) return cuda_status(e, "zncc smem attribute");
            }
            kernel<<<n_centers, threads, smem, (cudaStream_t)stream>>>(ref, Hr, Wr, def, Hd, Wd, (const float2 *)centers,
                                                                      win, search, (float2 *)u_out, score_out);
            D2IC_CHECK_LAUNCH("zncc_kernel");
            return (int)D2IC_OK;
        };
        return R == 7 ? launch(zncc_kernel<7>) : (R == 6 ? launch(zncc_kernel<6>) : launch(zncc_kernel<5>));
    }
    const size_t wide = sizeof(float) * base;
    if (wide > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(zncc_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wide);
        if (e != cudaSuccess) return cuda_status(e, "zncc smem attribute");
    }
    const int wide_threads = npa * npa >= 1024 ? 1024 : ((npa * npa + 31) / 32) * 32;
    zncc_wide_kernel<<<n_centers, wide_threads < 64 ? 64 : wide_threads, wide, (cudaStream_t)stream>>>(
        ref, Hr, Wr, def, Hd, Wd, (const float2 *)centers, win, search, (float2 *)u_out, score_out);
    D2IC_CHECK_LAUNCH("zncc_wide_kernel");
    return D2IC_OK;
}

extern "C" int d2ic_idw_project(const float *nodes, int n_nodes, const float *centers, const float *disp,
                                int n_centers, float power, float *u_out, void *stream) {
    D2IC_REQUIRE(nodes && u_out && (n_centers == 0 || (centers && disp)), "d2ic_idw_project: null pointer");
    D2IC_REQUIRE(n_nodes >= 0 && n_centers >= 0, "d2ic_idw_project: bad sizes");
    if (n_nodes == 0) return D2IC_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (n_nodes >= 4 * 8 * 912)   // at least ~2 waves of 4-node warps (3 blocks per SM on 152 SMs)
        idw_kernel<4><<<(n_nodes + 31) / 32, 256, 0, s>>>((const float2 *)nodes, n_nodes, (const float2 *)centers,
                                                          (const float2 *)disp, n_centers, power, (float2 *)u_out);
    else
        idw_kernel<1><<<(n_nodes + 7) / 8, 256, 0, s>>>((const float2 *)nodes, n_nodes, (const float2 *)centers,
                                                        (const float2 *)disp, n_centers, power, (float2 *)u_out);
    D2IC_CHECK_LAUNCH("idw_kernel");
    return D2IC_OK;
}
