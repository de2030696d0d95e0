// The Hessian of the converged frame as an assembled node operator, and the
// block-Jacobi preconditioned CG that solves H X = B for K right-hand sides in
// lock step (the linear solves of the implicit adjoint).
//
// Assembly (once per linearisation point): the per-chunk element blocks
// (d2ic_hessian_chunks: 10 symmetric 2x2 blocks per chunk) are scattered into
// per-node slots (each chunk owns one slot of each of its nodes, so no atomics),
// then one warp per node merges its slots and its springs into at most
// D2IC_HOP_MAX (column node, symmetric 2x2 block) entries, in slot order:
//     H_nj = (1/Np) sum_{chunks c at n, j} K^c_nj  +  alpha * springs.
// Apply: Y = H V, one warp per node and 32 right-hand sides (lane = column),
// V and Y laid out (node, component, k) with k fastest, so every neighbour read
// is one coalesced 128-byte row; the entries of a node are read once for all
// columns.  This replaces the chunk -> node-slot -> node pass per product (one
// write and one read of node_chunk_k * Nn * 2 * K floats per product).
//
// PCG: one cooperative launch runs all iterations of up to 64 columns with the vectors in shared memory
// (pcg_resident).  Meshes whose vectors do not fit on the chip, or only a few columns of many, keep them in memory and run five kernels
// per iteration: AP = H P with the block partials of P.AP, their column sums, the update of X, R, Z with
// the partials of R.R and R.Z, their column sums (one warp per column, blocks summed in a fixed order:
// deterministic) and the new direction; the last block of the second column sum decides convergence
// (||R|| <= rtol ||B|| for every column) into a device flag that makes the later kernels return at once,
// so the host launches iterations in batches and reads the flag once per batch.
#include <stdlib.h>
#include <string.h>

#include "common.cuh"

namespace d2ic {

constexpr int HOP = D2IC_HOP_MAX;   // operator entries per node
static_assert(HOP <= 32, "one lane per operator entry");
constexpr int PT = 256;             // threads per block of the node-range kernels

__device__ __forceinline__ int hop_pair(int a, int b) {   // a <= b: index of the pair in 0..9
    return a * 4 - (a * (a - 1)) / 2 + (b - a);
}

// operator storage inside the caller's buffer
struct HopView {
    float4 *blk;     // Nn * HOP: (xx, xy, yy, 0) of entry q of node n at n * HOP + q
    int *idx;        // Nn * HOP: column node, -1 after the last entry
    int *err;        // 1 int: set when a node has more than HOP distinct columns
    int *sids;       // assembly scratch: node_chunk_k * Nn * 4 column nodes (-1: slot not owned)
    float4 *sblk;    // node_chunk_k * Nn * 4 blocks
};

__host__ __device__ inline size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

__host__ __device__ inline size_t hop_layout(int n_nodes, int node_chunk_k, char *base, HopView *v) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off += al256(bytes);
        return p;
    };
    v->blk = (float4 *)take(sizeof(float4) * (size_t)n_nodes * HOP);
    v->idx = (int *)take(sizeof(int) * (size_t)n_nodes * HOP);
    v->err = (int *)take(sizeof(int));
    v->sids = (int *)take(sizeof(int) * (size_t)node_chunk_k * n_nodes * 4);
    v->sblk = (float4 *)take(sizeof(float4) * (size_t)node_chunk_k * n_nodes * 4);
    return off;
}

// chunk pass: thread (c, a) writes row a of chunk c's element matrix into slot rank_a(c) of node n_a
__global__ void __launch_bounds__(256) hop_scatter(const d2ic_frame_t *__restrict__ fp, const float *__restrict__ hess,
                                                   int *__restrict__ sids, float4 *__restrict__ sblk) {
    const d2ic_frame_t &F = *fp;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = t >> 2, a = t & 3;
    if (c >= F.n_chunks) return;
    const int n = __ldg(F.chunk_nodes + 4 * c + a);
    const int s = (int)(((unsigned)__ldg(F.chunk_slot + c) >> (8 * a)) & 0xffu);
    const size_t e = ((size_t)s * F.n_nodes + n) * 4;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int p = 3 * hop_pair(min(a, b), max(a, b));
        sids[e + b] = __ldg(F.chunk_nodes + 4 * c + b);
        sblk[e + b] = make_float4(__ldg(hess + 32 * (size_t)c + p), __ldg(hess + 32 * (size_t)c + p + 1),
                                  __ldg(hess + 32 * (size_t)c + p + 2), 0.f);
    }
}

// add (xx, xy, yy) to the entry of column j, appending it if new (whole warp; lane q holds entry q)
__device__ __forceinline__ void hop_add(int &my_idx, float4 &my_blk, int &count, int &overflow, int j, float xx,
                                        float xy, float yy, int lane) {
    const unsigned hit = __ballot_sync(0xffffffffu, my_idx == j);
    int q;
    if (hit) {
        q = __ffs(hit) - 1;
    } else {
        q = count;
        if (q >= HOP) {
            overflow = 1;
            return;
        }
        ++count;
        if (lane == q) my_idx = j;
    }
    if (lane == q) {
        my_blk.x += xx;
        my_blk.y += xy;
        my_blk.z += yy;
    }
}

// node pass: one warp per node merges its slots (slot order, row order) and its springs
__global__ void __launch_bounds__(256) hop_merge(const d2ic_frame_t *__restrict__ fp, const int *__restrict__ sids,
                                                 const float4 *__restrict__ sblk, float inv_np, float alpha,
                                                 int *__restrict__ idx, float4 *__restrict__ blk, int *__restrict__ err) {
    const d2ic_frame_t &F = *fp;
    const int lane = threadIdx.x & 31;
    const int n = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    if (n >= F.n_nodes) return;
    const size_t Nn = F.n_nodes;
    int my_idx = -1, count = 0, overflow = 0;
    float4 my_blk = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < F.node_chunk_k; ++s) {
        const size_t e = ((size_t)s * Nn + n) * 4;
        const int jl = lane < 4 ? __ldg(sids + e + lane) : -1;
        const float4 bl = lane < 4 ? __ldg(sblk + e + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int b = 0; b < 4; ++b) {
            const int j = __shfl_sync(0xffffffffu, jl, b);
            if (j < 0) break;   // slot not owned by a chunk (uniform)
            hop_add(my_idx, my_blk, count, overflow, j, inv_np * __shfl_sync(0xffffffffu, bl.x, b),
                    inv_np * __shfl_sync(0xffffffffu, bl.y, b), inv_np * __shfl_sync(0xffffffffu, bl.z, b), lane);
        }
    }
    for (int q = 0; q < F.max_deg; ++q) {                 // springs: alpha * w on the diagonal, -alpha * w off it
        const int j = __ldg(F.nbr_index + (size_t)q * Nn + n);
        if (j < 0) break;
        const float w = alpha * __ldg(F.nbr_weight + (size_t)q * Nn + n);
        hop_add(my_idx, my_blk, count, overflow, n, w, 0.f, w, lane);
        hop_add(my_idx, my_blk, count, overflow, j, -w, 0.f, -w, lane);
    }
    if (lane < HOP) {
        idx[(size_t)n * HOP + lane] = my_idx;
        blk[(size_t)n * HOP + lane] = my_blk;
    }
    if (overflow && lane == 0) atomicExch(err, 1);
}

// The block-Jacobi preconditioner: the inverse of each node's diagonal block (FP64, row-major 2x2), zero
// and inactive where the node has no block or one without a positive determinant.  One thread per node sums
// the block in FP64 from the node's slots and springs: the operator's merged block is an FP32 sum, whose
// rounding decides the sign of the determinant where the image varies along one direction only.  The
// determinant's products are rounded before the difference, so that equal products cancel to zero.
__global__ void hop_diagonal(const d2ic_frame_t *__restrict__ fp, const int *__restrict__ sids,
                             const float4 *__restrict__ sblk, float inv_np, float alpha, double *__restrict__ Minv,
                             unsigned char *__restrict__ active) {
    const d2ic_frame_t &F = *fp;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= F.n_nodes) return;
    const size_t Nn = F.n_nodes;
    const int K = F.node_chunk_k, md = F.max_deg;
    double xx = 0.0, xy = 0.0, yy = 0.0, w = 0.0;
    // loads of a batch in flight together
    constexpr int QS = 4, QN = 8;
    for (int s0 = 0; s0 < K; s0 += QS) {
        int4 j[QS];
#pragma unroll
        for (int t = 0; t < QS; ++t)                       // -1: slot not owned by a chunk
            j[t] = s0 + t < K ? __ldg(reinterpret_cast<const int4 *>(sids) + (size_t)(s0 + t) * Nn + n)
                              : make_int4(-1, -1, -1, -1);
#pragma unroll
        for (int t = 0; t < QS; ++t) {
            const int jj[4] = {j[t].x, j[t].y, j[t].z, j[t].w};
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if (jj[b] == n) {
                    const float4 v = __ldg(sblk + 4 * ((size_t)(s0 + t) * Nn + n) + b);
                    xx += (double)(inv_np * v.x);
                    xy += (double)(inv_np * v.y);
                    yy += (double)(inv_np * v.z);
                }
        }
    }
    bool alive = true;                                     // entries after the first -1 are padding
    for (int q0 = 0; q0 < md && alive; q0 += QN) {
        int i[QN];
        float v[QN];
#pragma unroll
        for (int t = 0; t < QN; ++t) {
            i[t] = q0 + t < md ? __ldg(F.nbr_index + (size_t)(q0 + t) * Nn + n) : -1;
            v[t] = q0 + t < md ? __ldg(F.nbr_weight + (size_t)(q0 + t) * Nn + n) : 0.f;
        }
#pragma unroll
        for (int t = 0; t < QN; ++t) {
            alive = alive && i[t] >= 0;
            if (alive) w += (double)v[t];
        }
    }
    xx += (double)alpha * w;
    yy += (double)alpha * w;
    const double det = __dsub_rn(__dmul_rn(xx, yy), __dmul_rn(xy, xy));
    const bool on = fabs(xx) + fabs(xy) + fabs(yy) > 0.0 && det > 0.0;
    double *m = Minv + 4 * (size_t)n;
    m[0] = on ? yy / det : 0.0;
    m[1] = m[2] = on ? -xy / det : 0.0;
    m[3] = on ? xx / det : 0.0;
    active[n] = on;
}

// one node (warp) x 32 columns (lanes): y = sum_q blk_q v_{idx_q}
__device__ __forceinline__ void hop_row(const int *__restrict__ idx, const float4 *__restrict__ blk, int n, int K, int k,
                                        const float *__restrict__ V, int lane, float &yx, float &yy) {
    const int my_idx = lane < HOP ? __ldg(idx + (size_t)n * HOP + lane) : -1;
    const float4 my_blk = lane < HOP ? __ldg(blk + (size_t)n * HOP + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    const unsigned live = __ballot_sync(0xffffffffu, my_idx >= 0);
    const int cnt = __popc(live);                          // entries are packed from lane 0
    yx = 0.f;
    yy = 0.f;
    constexpr int UB = 8;
    for (int q0 = 0; q0 < cnt; q0 += UB) {
        float vx[UB], vy[UB];
        int jj[UB];
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            jj[u] = __shfl_sync(0xffffffffu, my_idx, (q0 + u) & 31);
            const bool ok = q0 + u < cnt && k < K;
            vx[u] = ok ? __ldg(V + ((size_t)jj[u] * 2) * K + k) : 0.f;
            vy[u] = ok ? __ldg(V + ((size_t)jj[u] * 2 + 1) * K + k) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            const int q = (q0 + u) & 31;
            const float bx = __shfl_sync(0xffffffffu, my_blk.x, q), by = __shfl_sync(0xffffffffu, my_blk.y, q),
                        bz = __shfl_sync(0xffffffffu, my_blk.z, q);
            if (q0 + u < cnt) {
                yx = __fmaf_rn(bx, vx[u], __fmaf_rn(by, vy[u], yx));
                yy = __fmaf_rn(by, vx[u], __fmaf_rn(bz, vy[u], yy));
            }
        }
    }
}

// Y = H V: block = 8 nodes (warps) x 32 columns
__global__ void __launch_bounds__(256) hop_apply(const int *__restrict__ idx, const float4 *__restrict__ blk,
                                                 int n_nodes, const float *__restrict__ V, int K, float *__restrict__ Y) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n = blockIdx.x * 8 + w, k = blockIdx.y * 32 + lane;
    if (n >= n_nodes) return;
    float yx, yy;
    hop_row(idx, blk, n, K, k, V, lane, yx, yy);
    if (k < K) {
        Y[((size_t)n * 2) * K + k] = yx;
        Y[((size_t)n * 2 + 1) * K + k] = yy;
    }
}

// The entries of a block's 8 nodes, staged in shared memory and read as broadcasts.
struct HopTile {
    int idx[8][HOP];
    float4 blk[8][HOP];
    int cnt[8];
};

__device__ __forceinline__ void hop_stage(const int *__restrict__ idx, const float4 *__restrict__ blk, int n_nodes,
                                          HopTile &T) {
    static_assert(8 * HOP <= 256, "one thread per staged entry");
    const int t = threadIdx.x;
    if (t < 8 * HOP) {
        const int w = t / HOP, q = t % HOP, n = blockIdx.x * 8 + w;
        int j = -1;
        float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < n_nodes) {
            j = __ldg(idx + (size_t)n * HOP + q);
            b = __ldg(blk + (size_t)n * HOP + q);
        }
        T.idx[w][q] = j;
        T.blk[w][q] = b;
    }
    __syncthreads();
    if (t < 8) {
        int c = 0;
        while (c < HOP && T.idx[t][c] >= 0) ++c;   // entries are packed from the first
        T.cnt[t] = c;
    }
    __syncthreads();
}

// node w of the tile x 4 consecutive columns k0 .. k0 + 3 (K a multiple of 4): the same operations per
// column, in the same order, as hop_row
__device__ __forceinline__ void hop_row4(const HopTile &T, int w, int K, int k0, const float *__restrict__ V,
                                         float4 &yx, float4 &yy) {
    yx = make_float4(0.f, 0.f, 0.f, 0.f);
    yy = yx;
    const int cnt = T.cnt[w];
#pragma unroll 3
    for (int q = 0; q < cnt; ++q) {
        const int j = T.idx[w][q];
        const float4 b = T.blk[w][q];
        const float4 vx = __ldg(reinterpret_cast<const float4 *>(V + ((size_t)j * 2) * K + k0));
        const float4 vy = __ldg(reinterpret_cast<const float4 *>(V + ((size_t)j * 2 + 1) * K + k0));
        yx.x = __fmaf_rn(b.x, vx.x, __fmaf_rn(b.y, vy.x, yx.x));
        yx.y = __fmaf_rn(b.x, vx.y, __fmaf_rn(b.y, vy.y, yx.y));
        yx.z = __fmaf_rn(b.x, vx.z, __fmaf_rn(b.y, vy.z, yx.z));
        yx.w = __fmaf_rn(b.x, vx.w, __fmaf_rn(b.y, vy.w, yx.w));
        yy.x = __fmaf_rn(b.y, vx.x, __fmaf_rn(b.z, vy.x, yy.x));
        yy.y = __fmaf_rn(b.y, vx.y, __fmaf_rn(b.z, vy.y, yy.y));
        yy.z = __fmaf_rn(b.y, vx.z, __fmaf_rn(b.z, vy.z, yy.z));
        yy.w = __fmaf_rn(b.y, vx.w, __fmaf_rn(b.z, vy.w, yy.w));
    }
}

// Y = H V for K a multiple of 4: one warp per node (8 per block), lane l on columns 4 l .. 4 l + 3 of
// each 128-column pass over K.  The node's entries are staged once per warp in shared memory (no
// block-wide barrier) and read as broadcasts; per column the operations are those of hop_row.  At
// 32 registers 64 warps fit on an SM, so a frame's nodes (one warp each) run in a single wave on
// 152 SMs up to 9,728 nodes instead of queueing a second, mostly empty wave of blocks.
__global__ void __launch_bounds__(256, 8) hop_apply4(const int *__restrict__ idx, const float4 *__restrict__ blk,
                                                     int n_nodes, const float *__restrict__ V, int K,
                                                     float *__restrict__ Y) {
    __shared__ int s_j[8][HOP];
    __shared__ float4 s_b[8][HOP];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n = blockIdx.x * 8 + w;
    if (n >= n_nodes) return;                  // the whole warp: nothing below waits on the block
    int j = -1;
    if (lane < HOP) {
        j = __ldg(idx + (size_t)n * HOP + lane);
        s_j[w][lane] = j;
        s_b[w][lane] = __ldg(blk + (size_t)n * HOP + lane);
    }
    const int cnt = __popc(__ballot_sync(0xffffffffu, j >= 0));   // entries are packed from the first
    __syncwarp();
    // float4 offsets within 32 bits (the host checks n_nodes * 2 * K < 2^31): row 2 j at j * K / 2
    const int h = K >> 1, q4 = K >> 2;
    const float4 *V4 = reinterpret_cast<const float4 *>(V);
    float4 *Y4 = reinterpret_cast<float4 *>(Y) + n * h;
    for (int c = lane; c < q4; c += 32) {
        float4 yx = make_float4(0.f, 0.f, 0.f, 0.f), yy = yx;
#pragma unroll 1
        for (int q = 0; q < cnt; ++q) {
            const int r = s_j[w][q] * h + c;
            const float4 b = s_b[w][q];
            const float4 vx = __ldg(V4 + r);
            const float4 vy = __ldg(V4 + r + q4);
            yx.x = __fmaf_rn(b.x, vx.x, __fmaf_rn(b.y, vy.x, yx.x));
            yx.y = __fmaf_rn(b.x, vx.y, __fmaf_rn(b.y, vy.y, yx.y));
            yx.z = __fmaf_rn(b.x, vx.z, __fmaf_rn(b.y, vy.z, yx.z));
            yx.w = __fmaf_rn(b.x, vx.w, __fmaf_rn(b.y, vy.w, yx.w));
            yy.x = __fmaf_rn(b.y, vx.x, __fmaf_rn(b.z, vy.x, yy.x));
            yy.y = __fmaf_rn(b.y, vx.y, __fmaf_rn(b.z, vy.y, yy.y));
            yy.z = __fmaf_rn(b.y, vx.z, __fmaf_rn(b.z, vy.z, yy.z));
            yy.w = __fmaf_rn(b.y, vx.w, __fmaf_rn(b.z, vy.w, yy.w));
        }
        Y4[c] = yx;
        Y4[c + q4] = yy;
    }
}

// ---------------------------------------------------------------------------
// PCG
// ---------------------------------------------------------------------------
struct PcgCtl {
    int done;        // all columns converged: later kernels return at once
    int iters;       // iterations whose update ran
    int cnt_check;   // last-block counter of the convergence check (reset by the last block)
    int pad_;
};

__device__ __forceinline__ int ld_flag(const int *p) { return *(volatile const int *)p; }

// nodes [n0, n1) of block b
__device__ __forceinline__ void node_range(int n_nodes, int &n0, int &n1) {
    const int per = (n_nodes + gridDim.x - 1) / gridDim.x;
    n0 = min((int)blockIdx.x * per, n_nodes);
    n1 = min(n0 + per, n_nodes);
}

__global__ void __launch_bounds__(PT) pcg_init(int n_nodes, int K, const double *__restrict__ B,
                                               const unsigned char *__restrict__ act, const double *__restrict__ Minv,
                                               double *__restrict__ X, double *__restrict__ R, double *__restrict__ Z,
                                               double *__restrict__ P, float *__restrict__ Pf,
                                               double *__restrict__ part_rz, double *__restrict__ part_bb) {
    int n0, n1;
    node_range(n_nodes, n0, n1);
    for (int k = threadIdx.x; k < K; k += PT) {
        double srz = 0.0, sbb = 0.0;
        for (int n = n0; n < n1; ++n) {
            const double m = act[n] ? 1.0 : 0.0;
            const size_t i0 = ((size_t)n * 2) * K + k, i1 = i0 + K;
            const double b0 = B[i0] * m, b1 = B[i1] * m;
            const double *M = Minv + 4 * (size_t)n;
            const double z0 = M[0] * b0 + M[1] * b1, z1 = M[2] * b0 + M[3] * b1;
            X[i0] = 0.0;
            X[i1] = 0.0;
            R[i0] = b0;
            R[i1] = b1;
            Z[i0] = z0;
            Z[i1] = z1;
            P[i0] = z0;
            P[i1] = z1;
            Pf[i0] = (float)z0;
            Pf[i1] = (float)z1;
            srz += b0 * z0 + b1 * z1;
            sbb += b0 * b0 + b1 * b1;
        }
        part_rz[(size_t)blockIdx.x * K + k] = srz;
        part_bb[(size_t)blockIdx.x * K + k] = sbb;
    }
}

// AP = H P (masked to active dofs) and the block partials of pap[k] = P.AP: block = 8 nodes x
// 32 columns (one per lane) or, with VEC (K a multiple of 4), 128 columns (four per lane)
template <bool VEC>
__global__ void __launch_bounds__(256) pcg_apply(const int *__restrict__ idx, const float4 *__restrict__ blk,
                                                 int n_nodes, int K, const float *__restrict__ Pf,
                                                 const double *__restrict__ P, const unsigned char *__restrict__ act,
                                                 float *__restrict__ AP, double *__restrict__ part,
                                                 const PcgCtl *ctl) {
    if (ld_flag(&ctl->done)) return;
    constexpr int CW = VEC ? 4 : 1;                 // columns per lane
    __shared__ HopTile T;
    __shared__ double s_p[8][32 * CW];
    hop_stage(idx, blk, n_nodes, T);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n = blockIdx.x * 8 + w, k0 = blockIdx.y * 32 * CW + CW * lane;
    double pp[CW];
#pragma unroll
    for (int c = 0; c < CW; ++c) pp[c] = 0.0;
    if (n < n_nodes && k0 < K) {
        float y0[CW], y1[CW];
        if (VEC) {
            float4 yx, yy;
            hop_row4(T, w, K, k0, Pf, yx, yy);
            *reinterpret_cast<float4 *>(AP + ((size_t)n * 2) * K + k0) = yx;
            *reinterpret_cast<float4 *>(AP + ((size_t)n * 2 + 1) * K + k0) = yy;
            const float a0[4] = {yx.x, yx.y, yx.z, yx.w}, a1[4] = {yy.x, yy.y, yy.z, yy.w};
#pragma unroll
            for (int c = 0; c < CW; ++c) {
                y0[c] = a0[c];
                y1[c] = a1[c];
            }
        } else {
            float yx = 0.f, yy = 0.f;
            for (int q = 0; q < T.cnt[w]; ++q) {
                const int j = T.idx[w][q];
                const float4 b = T.blk[w][q];
                const float vx = __ldg(Pf + ((size_t)j * 2) * K + k0), vy = __ldg(Pf + ((size_t)j * 2 + 1) * K + k0);
                yx = __fmaf_rn(b.x, vx, __fmaf_rn(b.y, vy, yx));
                yy = __fmaf_rn(b.y, vx, __fmaf_rn(b.z, vy, yy));
            }
            AP[((size_t)n * 2) * K + k0] = yx;
            AP[((size_t)n * 2 + 1) * K + k0] = yy;
            y0[0] = yx;
            y1[0] = yy;
        }
        if (act[n]) {
#pragma unroll
            for (int c = 0; c < CW; ++c) {
                const size_t i0 = ((size_t)n * 2) * K + k0 + c;
                pp[c] = P[i0] * (double)y0[c] + P[i0 + K] * (double)y1[c];
            }
        }
    }
#pragma unroll
    for (int c = 0; c < CW; ++c) s_p[w][CW * lane + c] = pp[c];
    __syncthreads();
    for (int t = threadIdx.x; t < 32 * CW; t += blockDim.x) {
        const int k = blockIdx.y * 32 * CW + t;
        if (k >= K) continue;
        double sum = 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += s_p[i][t];
        part[(size_t)blockIdx.x * K + k] = sum;
    }
}

__global__ void __launch_bounds__(PT) pcg_step(int n_nodes, int K, const double *__restrict__ rz,
                                               const double *__restrict__ pap, const unsigned char *__restrict__ act,
                                               const double *__restrict__ Minv, double *__restrict__ X,
                                               double *__restrict__ R, double *__restrict__ Z,
                                               const double *__restrict__ P, const float *__restrict__ AP,
                                               double *__restrict__ part_rr, double *__restrict__ part_rz,
                                               const PcgCtl *ctl) {
    if (ld_flag(&ctl->done)) return;
    int n0, n1;
    node_range(n_nodes, n0, n1);
    for (int k = threadIdx.x; k < K; k += PT) {
        const double a = pap[k] > 0.0 ? rz[k] / pap[k] : 0.0;
        double srr = 0.0, srz = 0.0;
        for (int n = n0; n < n1; ++n) {
            const double m = act[n] ? 1.0 : 0.0;
            const size_t i0 = ((size_t)n * 2) * K + k, i1 = i0 + K;
            X[i0] += a * P[i0];
            X[i1] += a * P[i1];
            const double r0 = R[i0] - a * ((double)AP[i0] * m), r1 = R[i1] - a * ((double)AP[i1] * m);
            R[i0] = r0;
            R[i1] = r1;
            const double *M = Minv + 4 * (size_t)n;
            const double z0 = M[0] * r0 + M[1] * r1, z1 = M[2] * r0 + M[3] * r1;
            Z[i0] = z0;
            Z[i1] = z1;
            srr += r0 * r0 + r1 * r1;
            srz += r0 * z0 + r1 * z1;
        }
        part_rr[(size_t)blockIdx.x * K + k] = srr;
        part_rz[(size_t)blockIdx.x * K + k] = srz;
    }
}

// out_a[k] (and out_b[k]) = sum over blocks b of part_a[b][k] (part_b): one warp per column, lane l
// sums blocks l, l + 32, ... in order, then a fixed shuffle tree (deterministic).  With `check`,
// the last block to finish decides convergence (every column: sqrt(out_a) <= rtol sqrt(bb)) and
// counts the iteration.
__global__ void pcg_colsum(int nb, int K, const double *__restrict__ part_a, const double *__restrict__ part_b,
                           double *__restrict__ out_a, double *__restrict__ out_b, const double *__restrict__ bb,
                           double rtol, int check, PcgCtl *ctl) {
    if (ld_flag(&ctl->done)) return;
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k < K) {
        double sa = 0.0, sb = 0.0;
        for (int b = lane; b < nb; b += 32) {
            sa += part_a[(size_t)b * K + k];
            if (part_b) sb += part_b[(size_t)b * K + k];
        }
        sa = warp_sum_d(sa);
        sb = warp_sum_d(sb);
        if (lane == 0) {
            out_a[k] = sa;
            if (out_b) out_b[k] = sb;
        }
    }
    if (!check) return;
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(&ctl->cnt_check, 1) == (int)gridDim.x - 1;
        if (s_last) ctl->cnt_check = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    int ok = 1;
    for (int c = threadIdx.x; c < K; c += blockDim.x) {
        const double bn = fmax(sqrt(__ldcg(bb + c)), 1e-300);
        ok &= sqrt(__ldcg(out_a + c)) <= rtol * bn;
    }
    ok = __syncthreads_and(ok);
    if (threadIdx.x == 0) {
        ctl->iters += 1;
        if (ok) ctl->done = 1;
    }
}

__global__ void __launch_bounds__(PT) pcg_dir(int n_nodes, int K, const double *__restrict__ rz_old,
                                              const double *__restrict__ rz_new, const double *__restrict__ Z,
                                              double *__restrict__ P, float *__restrict__ Pf, const PcgCtl *ctl) {
    if (ld_flag(&ctl->done)) return;
    int n0, n1;
    node_range(n_nodes, n0, n1);
    for (int k = threadIdx.x; k < K; k += PT) {
        const double beta = rz_old[k] > 0.0 ? rz_new[k] / rz_old[k] : 0.0;
        for (int n = n0; n < n1; ++n) {
            const size_t i0 = ((size_t)n * 2) * K + k, i1 = i0 + K;
            const double p0 = Z[i0] + beta * P[i0], p1 = Z[i1] + beta * P[i1];
            P[i0] = p0;
            P[i1] = p1;
            Pf[i0] = (float)p0;
            Pf[i1] = (float)p1;
        }
    }
}

// ---------------------------------------------------------------------------
// PCG with the vectors on the chip
// ---------------------------------------------------------------------------
// One launch runs all iterations of up to PR_COLS columns: block b owns a range of nodes and keeps X, R,
// P and H P of its (node, column) pairs in shared memory; only P in FP32, which neighbours need, goes
// through global memory.  Per iteration: H P and P.HP; the step with R.R and R.Z; the new direction.  A
// sum over the grid is two hops of tagged records (the block's partial to the warp that owns the sum,
// the sum to every block), the exchange of P one grid barrier; a system that fits one block needs only
// block barriers.
//
// The vectors and the sums are double-floats (48 bits) instead of FP64: GB300 issues an FP64
// instruction per SM every 16 cycles, so the 12 FP64 operations per vector entry and iteration cost 20 us
// at 7,396 nodes x 64 columns, the same in double-float 3 us; the product with H is FP32 either way.
// Columns are scaled by a power of two to a largest entry in [1, 2), and the preconditioner by the one that
// halves the exponent of its largest entry, so that FP32's exponent range suffices wherever the FP32 operator's
// does: with H of size h, P is of size h^-1/2, H P of size h^1/2 and X, kept as h X, of size 1.  (CG with a scaled
// preconditioner gives the same iterates; powers of two change no bits.)  Errors against CG with FP64 products of the same operator are
// those of the FP32 products, with these vectors and with FP64 ones: 28 meshes of 330 to 4,212 nodes and 1 to
// 47 columns, 0.9 to 2.2e-7 of the solution's norm at rtol 1e-7, 0.8 to 1.2e-7 at 1e-10 and at 1e-13, each pair alike to
// three digits and with the same iteration counts.  (Against FP64 vectors with the same FP32 products the solution
// differs by 4e-13 to 1e-9 of its norm up to 3,000 nodes; CG amplifies any rounding, in 103 iterations on 22,801 nodes
// to 1e-8, and FP64 vectors with another order of the sums to 5e-9.)
//
// Bound by the hops at few columns (two sums and a barrier, about 6 us) and by the double-float
// arithmetic and the latency of the neighbours' values at many.  Per iteration, five kernels before ->
// now: 7,569 nodes x 64 columns 66 -> 26 us, 4,331 x 6 55 -> 12 us, 1,089 x 1 27 -> 11 us.
constexpr int PR_T = 512;                  // threads per block
constexpr int PR_PAIR_BYTES = 7 * 8;       // x, r, p (two components, double-float) and two floats of H P
constexpr int PR_NODE_BYTES = 4 * HOP + 32;   // the operator's column nodes and the preconditioner block
constexpr int PR_BLOCK_BYTES = 16 * HOP;       // the operator's blocks of a node
constexpr int PR_BYTES = 212 * 1024;       // dynamic shared memory per block at most
constexpr int PR_COLS = 64;                // columns per launch
constexpr int PR_POLL = 5;                 // records a lane polls at a time: 160 blocks in one round trip
// Systems of at most two pairs per thread run in one block: no grid hops, but every pair of a thread adds to the
// iteration.  One block and several, us per iteration: 529 nodes x 1 column 8.7 and 9.2, 1,024 x 1 11.2 and 11.1,
// 2,025 x 1 20.9 and 11.3; 256 x 6 9.9 and 8.9, 400 x 6 13.7 and 8.7; 25 x 64 8.1 and 8.5, 49 x 64 12.9 and 9.4.
constexpr int PR_ONE_BLOCK = 2 * PR_T;
constexpr unsigned long long PR_WAIT_NS = 5ull * 1000ull * 1000ull * 1000ull;

struct PrArgs {
    const int *idx;                        // the operator
    const float4 *blk;
    const int *overflow;                   // the assembly's error flag
    const double *Minv;                    // inverse diagonal blocks
    float2 *M;                             // the same, scaled, as 4 double-floats per node (unless staged)
    const unsigned char *act;
    const double *B;
    double *X;
    float *P;                              // exchanged direction: (node, component, column of the launch)
    uint4 *part, *tot;                     // records: partials (sum, block), totals
    unsigned *bar;                         // barrier arrivals
    int *out;                              // iterations (max over launches), status
    int n_nodes, K, k0, Kb, max_iter;      // columns k0 .. k0 + Kb of K
    int staged;                            // operator indices and preconditioner in shared memory
    double rtol;
};

__device__ __forceinline__ DF df_mul(DF a, DF b) {
    const DF p = df_prod(a.hi, b.hi);
    const float lo = p.lo + __fmaf_rn(a.hi, b.lo, a.lo * b.hi);
    const float h = p.hi + lo;
    return {h, lo - (h - p.hi)};
}
__device__ __forceinline__ DF df_mul_f(DF a, float b) {
    const DF p = df_prod(a.hi, b);
    const float lo = __fmaf_rn(a.lo, b, p.lo), h = p.hi + lo;
    return {h, lo - (h - p.hi)};
}
__device__ __forceinline__ DF df_neg(DF a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ DF df_div(DF a, DF b) {   // two quotient digits
    const float q1 = a.hi / b.hi;
    const DF r = df_add(a, df_neg(df_mul_f(b, q1)));
    return df_two_sum(q1, r.hi / b.hi);
}
__device__ __forceinline__ DF df_from(double x) {
    const float hi = (float)x;
    return {hi, (float)(x - (double)hi)};
}

// the block's shared state
struct PrShared {
    DF red[2][PR_T];
    DF tot[2 * PR_COLS];
    DF a[PR_COLS], rz[PR_COLS];
    double thr[PR_COLS];
    int scale[PR_COLS];                    // biased FP64 exponent of the column's largest entry
    int mexp;                              // exponent of the preconditioner's scale
    int stop;                              // a wait ran out somewhere
};
extern __shared__ __align__(16) unsigned char pr_dyn[];

struct PrSum {
    __device__ static DF op(DF a, DF b) { return df_add(a, b); }
};
struct PrMax {                             // non-negative integers in the first word
    __device__ static DF op(DF a, DF b) { return __float_as_int(a.hi) >= __float_as_int(b.hi) ? a : b; }
};

// whole warp: polls the records rec[lane], rec[lane + 32], ... below n, N at most per lane, until all
// carry the tag; false after an abort
template <int N>
__device__ __forceinline__ bool pr_poll(const uint4 *rec, int n, unsigned tag, uint4 (&r)[N], int *out, int lane) {
    unsigned long long t0 = 0;
    for (unsigned it = 0;; ++it) {
        bool all = true;
#pragma unroll
        for (int i = 0; i < N; ++i) r[i] = lane + 32 * i < n ? ld_record(rec + lane + 32 * i) : make_uint4(0u, 0u, tag, 0u);
#pragma unroll
        for (int i = 0; i < N; ++i) all = all && r[i].z == tag;
        if (__all_sync(0xffffffffu, all)) return true;
        if ((it & 63) == 63) {
            int go = 1;
            if (lane == 0) {
                const unsigned long long now = gtimer();
                if (t0 == 0) t0 = now;
                if (*(volatile int *)(out + 1) != 0) go = 0;
                else if (now - t0 > PR_WAIT_NS) {
                    atomicExch(out + 1, D2IC_WAIT_TIMEOUT);
                    go = 0;
                }
            }
            if (!__shfl_sync(0xffffffffu, go, 0)) return false;
        }
    }
}

// Reduces NV values per thread (thread t: column t % Kb) over the grid into S.tot[v * Kb + k], in a fixed
// order; false after an abort.  tag: unique per call.
template <int NV, class OP>
__device__ bool pr_reduce(const DF *v, const PrArgs &A, PrShared &S, int T, int rows, unsigned tag) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, Kb = A.Kb, row = tid / Kb, k = tid % Kb;
    const int G = gridDim.x;
    DF w[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) w[i] = v[i];
    int h = rows, r = row;                 // rows of Kb values left, this thread's row
    bool mine = tid < T;
    if (32 % Kb == 0) {                    // the warp's rows first, without barriers
#pragma unroll 1
        for (int o = 16; o >= Kb; o >>= 1)
#pragma unroll
            for (int i = 0; i < NV; ++i)
                w[i] = OP::op(w[i], DF{__shfl_xor_sync(0xffffffffu, w[i].hi, o), __shfl_xor_sync(0xffffffffu, w[i].lo, o)});
        h = PR_T / 32;
        r = wid;
        mine = lane < Kb;
    }
    const int at = r * Kb + k;
    __syncthreads();                       // the previous totals have been read
    if (mine)
#pragma unroll
        for (int i = 0; i < NV; ++i) S.red[i][at] = w[i];
    while (h > 1) {
        const int half = (h + 1) >> 1;
        __syncthreads();
        if (mine && r < h - half)
#pragma unroll
            for (int i = 0; i < NV; ++i) S.red[i][at] = OP::op(S.red[i][at], S.red[i][at + half * Kb]);
        h = half;
    }
    if (G == 1) {
        if (tid < Kb)
#pragma unroll
            for (int i = 0; i < NV; ++i) S.tot[i * Kb + tid] = S.red[i][tid];
        __syncthreads();
        return true;
    }
    const int items = NV * Kb;
    if (tid < Kb)
#pragma unroll
        for (int i = 0; i < NV; ++i)
            st_record(A.part + (size_t)(i * Kb + tid) * G + blockIdx.x,
                      make_uint4(__float_as_uint(S.red[i][tid].hi), __float_as_uint(S.red[i][tid].lo), tag, 0u));
    bool ok = true;
    for (int m = blockIdx.x + G * wid; m < items && ok; m += G * (PR_T / 32)) {   // sums this block owns
        DF t = {0.f, 0.f};
        for (int g0 = 0; g0 < G && ok; g0 += 32 * PR_POLL) {
            uint4 r[PR_POLL];
            ok = pr_poll<PR_POLL>(A.part + (size_t)m * G + g0, G - g0, tag, r, A.out, lane);
#pragma unroll
            for (int i = 0; i < PR_POLL; ++i)
                if (g0 + lane + 32 * i < G) {
                    const DF x = {__uint_as_float(r[i].x), __uint_as_float(r[i].y)};
                    t = g0 + i == 0 ? x : OP::op(t, x);
                }
        }
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1)
            t = OP::op(t, DF{__shfl_xor_sync(0xffffffffu, t.hi, o), __shfl_xor_sync(0xffffffffu, t.lo, o)});
        if (lane == 0 && ok)
            st_record(A.tot + m, make_uint4(__float_as_uint(t.hi), __float_as_uint(t.lo), tag, 0u));
    }
    for (int m0 = wid * 32; m0 < items && ok; m0 += PR_T) {
        uint4 r[1];
        ok = pr_poll<1>(A.tot + m0, items - m0, tag, r, A.out, lane);
        if (ok && m0 + lane < items) S.tot[m0 + lane] = DF{__uint_as_float(r[0].x), __uint_as_float(r[0].y)};
    }
    if (!ok && lane == 0) S.stop = 1;
    __syncthreads();
    return S.stop == 0;
}

// every block's writes before it are seen by every block after it; false after an abort
__device__ bool pr_barrier(const PrArgs &A, PrShared &S, unsigned phase) {
    __syncthreads();
    if (gridDim.x == 1) return true;
    if (threadIdx.x == 0) {
        fence_acq_rel();
        atomicAdd(A.bar, 1u);
        const unsigned target = phase * gridDim.x;
        unsigned long long t0 = 0;
        for (unsigned it = 0; *(volatile unsigned *)A.bar < target; ++it)
            if ((it & 63) == 63) {
                const unsigned long long now = gtimer();
                if (t0 == 0) t0 = now;
                if (*(volatile int *)(A.out + 1) != 0) {
                    S.stop = 1;
                    break;
                }
                if (now - t0 > PR_WAIT_NS) {
                    atomicExch(A.out + 1, D2IC_WAIT_TIMEOUT);
                    S.stop = 1;
                    break;
                }
            }
        fence_acq_rel();
    }
    __syncthreads();
    return S.stop == 0;
}

__global__ void __launch_bounds__(PR_T, 1) pcg_resident(const PrArgs A) {
    __shared__ PrShared S;
    const int Kb = A.Kb, tid = threadIdx.x;
    const int per = (A.n_nodes + gridDim.x - 1) / gridDim.x;
    const int n0 = min((int)blockIdx.x * per, A.n_nodes), nn = min(per, A.n_nodes - n0);
    // thread t < T has column t % Kb and the block's nodes row, row + rows, ...
    const int rows = PR_T / Kb, T = rows * Kb, k = tid % Kb, row = tid / Kb;
    const int cap = per * Kb;                            // pairs of a full block
    float2 *x = reinterpret_cast<float2 *>(pr_dyn), *r = x + 2 * cap, *p = r + 2 * cap;   // component c at c * cap
    float *ap = reinterpret_cast<float *>(p + 2 * cap);
    // with A.staged, the block's nodes' column indices (none for an inactive node) and preconditioner
    // blocks: every grid barrier empties the L1, so from global memory they cost an L2 round trip per node
    float4 *sM = reinterpret_cast<float4 *>(pr_dyn + (((size_t)cap * PR_PAIR_BYTES + 15) & ~(size_t)15));
    int *sidx = reinterpret_cast<int *>(sM + 2 * per);
    // with A.staged 2 also the operator's blocks
    float4 *sblk = reinterpret_cast<float4 *>(sidx + HOP * per);
    if (A.staged == 2)
        for (int i = tid; i < nn * HOP; i += PR_T) sblk[i] = __ldg(A.blk + (size_t)n0 * HOP + i);
    if (A.staged) {
        for (int i = tid; i < nn * HOP; i += PR_T) sidx[i] = A.act[n0 + i / HOP] ? __ldg(A.idx + (size_t)n0 * HOP + i) : -1;
    }
    if (tid == 0) S.stop = 0;
    if (*A.overflow) return;                             // every block: the host reports it
    unsigned tag = 0, phase = 0;
    auto pairs = [&](auto &&f) {
        if (tid < T)
            for (int i = row; i < nn; i += rows) f(n0 + i, i * Kb + k);
    };
    auto ld = [](float2 v) { return DF{v.x, v.y}; };
    auto st = [](DF v) { return make_float2(v.hi, v.lo); };
    auto precond = [&](int n, DF r0, DF r1, DF &z0, DF &z1) {
        // written by this block: plain loads
        const float4 m0 = A.staged ? sM[2 * (n - n0)] : reinterpret_cast<const float4 *>(A.M)[2 * (size_t)n];
        const float4 m1 = A.staged ? sM[2 * (n - n0) + 1] : reinterpret_cast<const float4 *>(A.M)[2 * (size_t)n + 1];
        z0 = df_add(df_mul(DF{m0.x, m0.y}, r0), df_mul(DF{m0.z, m0.w}, r1));
        z1 = df_add(df_mul(DF{m1.x, m1.y}, r0), df_mul(DF{m1.z, m1.w}, r1));
    };
    auto put_p = [&](int n, DF p0, DF p1) {
        float *o = A.P + (size_t)n * 2 * Kb + k;
        o[0] = p0.hi;
        o[Kb] = p1.hi;
    };
    // the columns' scales and the preconditioner's largest entry
    int e = 0, em = 0;
    if (tid < T)
        for (int i = tid; i < 4 * nn; i += T) em = max(em, (__double2hiint(A.Minv[4 * (size_t)n0 + i]) >> 20) & 0x7ff);
    pairs([&](int n, int) {
        const size_t i0 = (size_t)n * 2 * A.K + A.k0 + k;
        if (A.act[n]) {
            e = max(e, (__double2hiint(A.B[i0]) >> 20) & 0x7ff);
            e = max(e, (__double2hiint(A.B[i0 + A.K]) >> 20) & 0x7ff);
        }
    });
    DF v[2] = {DF{__int_as_float(e), 0.f}, DF{__int_as_float(em), 0.f}};
    if (!pr_reduce<2, PrMax>(v, A, S, T, rows, ++tag)) return;
    if (tid < Kb) {
        const int m = __float_as_int(S.tot[tid].hi);
        S.scale[tid] = m == 0 || m == 0x7ff ? 1023 : min(m, 2045);
    }
    if (tid == 0) {                                      // half of its exponent off the blocks (see above)
        int m = 0;
        for (int i = 0; i < Kb; ++i) m = max(m, __float_as_int(S.tot[Kb + i].hi));
        S.mexp = m == 0 || m == 0x7ff ? 0 : -min(max((m - 1023) / 2, -100), 100);
    }
    __syncthreads();
    {
        const double by = __hiloint2double((1023 + S.mexp) << 20, 0);
        float2 *M = A.staged ? reinterpret_cast<float2 *>(sM) : A.M + 4 * (size_t)n0;
        for (int i = tid; i < 4 * nn; i += PR_T) {
            const DF m = df_from(A.Minv[4 * (size_t)n0 + i] * by);
            M[i] = make_float2(m.hi, m.lo);
        }
    }
    __syncthreads();
    const double up = __hiloint2double(min(max(2046 - S.scale[k], 1), 2046) << 20, 0);   // 2^(1023 - scale)
    const float ms = __int_as_float((127 + S.mexp) << 23);   // the preconditioner's scale
    // X = 0, R = B, Z = M R, P = Z
    v[0] = v[1] = DF{0.f, 0.f};
    pairs([&](int n, int i) {
        const size_t i0 = (size_t)n * 2 * A.K + A.k0 + k;
        const bool on = A.act[n] != 0;
        const DF r0 = on ? df_from(A.B[i0] * up) : DF{0.f, 0.f}, r1 = on ? df_from(A.B[i0 + A.K] * up) : DF{0.f, 0.f};
        DF z0, z1;
        precond(n, r0, r1, z0, z1);
        x[i] = x[cap + i] = make_float2(0.f, 0.f);
        r[i] = st(r0);
        r[cap + i] = st(r1);
        p[i] = st(z0);
        p[cap + i] = st(z1);
        put_p(n, z0, z1);
        v[0] = df_add(v[0], df_add(df_mul(r0, z0), df_mul(r1, z1)));
        v[1] = df_add(v[1], df_add(df_mul(r0, r0), df_mul(r1, r1)));
    });
    if (!pr_reduce<2, PrSum>(v, A, S, T, rows, ++tag)) return;
    if (tid < Kb) {
        S.rz[tid] = S.tot[tid];
        const double bn = A.rtol * fmax(sqrt(df_to_double(S.tot[Kb + tid])), 1e-300);
        S.thr[tid] = bn * bn;
    }
    if (!pr_barrier(A, S, ++phase)) return;
    int it = 0;
    while (it < A.max_iter) {
        // AP = H P and P.AP
        v[0] = DF{0.f, 0.f};
        pairs([&](int n, int i) {
            float y0 = 0.f, y1 = 0.f;
            const float *P = A.P + k;
            if (A.staged == 2) {
                // a node couples to nine nodes on a regular grid: their values are all in flight together
                const int4 *ix = reinterpret_cast<const int4 *>(sidx + (n - n0) * HOP);
                const float4 *bl = sblk + (n - n0) * HOP;
                constexpr int Q = 12;
                for (int q0 = 0; q0 < HOP && ix[q0 / 4].x >= 0; q0 += Q) {
                    float vx[Q], vy[Q];
#pragma unroll
                    for (int q = 0; q < Q; q += 4) {
                        const int4 j4 = q0 + q < HOP ? ix[(q0 + q) / 4] : make_int4(-1, -1, -1, -1);
                        const int jj[4] = {j4.x, j4.y, j4.z, j4.w};
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            vx[q + t] = jj[t] >= 0 ? P[(size_t)jj[t] * 2 * Kb] : 0.f;
                            vy[q + t] = jj[t] >= 0 ? P[(size_t)jj[t] * 2 * Kb + Kb] : 0.f;
                        }
                    }
#pragma unroll
                    for (int q = 0; q < Q; ++q)
                        if (q0 + q < HOP) {                // blocks beyond the last entry are zero
                            const float4 b = bl[q0 + q];
                            y0 = __fmaf_rn(b.x, vx[q], __fmaf_rn(b.y, vy[q], y0));
                            y1 = __fmaf_rn(b.y, vx[q], __fmaf_rn(b.z, vy[q], y1));
                        }
                }
            } else {
                const float4 *bl = A.blk + (size_t)n * HOP;
                const bool on = A.staged || A.act[n];
                constexpr int Q = 4;                           // entries in flight together, nine on a regular grid
                int4 j4 = make_int4(-1, -1, -1, -1);
                if (on) j4 = A.staged ? *reinterpret_cast<const int4 *>(sidx + (n - n0) * HOP)
                                      : __ldg(reinterpret_cast<const int4 *>(A.idx + (size_t)n * HOP));
                for (int q0 = 0; q0 < HOP && j4.x >= 0; q0 += Q) {
                    const int jj[Q] = {j4.x, j4.y, j4.z, j4.w};
                    float4 b[Q];
                    float vx[Q], vy[Q];
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        const bool has = jj[q] >= 0;
                        const float *src = P + (size_t)(has ? jj[q] : 0) * 2 * Kb;
                        b[q] = has ? __ldg(bl + q0 + q) : make_float4(0.f, 0.f, 0.f, 0.f);
                        vx[q] = src[0];
                        vy[q] = src[Kb];
                    }
                    j4 = make_int4(-1, -1, -1, -1);
                    if (q0 + Q < HOP)
                        j4 = A.staged ? *reinterpret_cast<const int4 *>(sidx + (n - n0) * HOP + q0 + Q)
                                      : __ldg(reinterpret_cast<const int4 *>(A.idx + (size_t)n * HOP + q0 + Q));
#pragma unroll
                    for (int q = 0; q < Q; ++q)
                        if (jj[q] >= 0) {
                            y0 = __fmaf_rn(b[q].x, vx[q], __fmaf_rn(b[q].y, vy[q], y0));
                            y1 = __fmaf_rn(b[q].y, vx[q], __fmaf_rn(b[q].z, vy[q], y1));
                        }
                }
            }
            ap[i] = y0;
            ap[cap + i] = y1;
            v[0] = df_add(v[0], df_add(df_mul_f(ld(p[i]), y0), df_mul_f(ld(p[cap + i]), y1)));
        });
        if (!pr_reduce<1, PrSum>(v, A, S, T, rows, ++tag)) return;
        if (tid < Kb) S.a[tid] = S.tot[tid].hi > 0.f ? df_div(S.rz[tid], S.tot[tid]) : DF{0.f, 0.f};
        __syncthreads();
        // X += a P, R -= a AP, R.R and R.Z
        const DF a = S.a[k], ax = {a.hi * ms * ms, a.lo * ms * ms};
        v[0] = v[1] = DF{0.f, 0.f};
        pairs([&](int n, int i) {
            x[i] = st(df_add(ld(x[i]), df_mul(ax, ld(p[i]))));
            x[cap + i] = st(df_add(ld(x[cap + i]), df_mul(ax, ld(p[cap + i]))));
            const DF r0 = df_add(ld(r[i]), df_neg(df_mul_f(a, ap[i])));
            const DF r1 = df_add(ld(r[cap + i]), df_neg(df_mul_f(a, ap[cap + i])));
            r[i] = st(r0);
            r[cap + i] = st(r1);
            DF z0, z1;
            precond(n, r0, r1, z0, z1);
            v[0] = df_add(v[0], df_add(df_mul(r0, r0), df_mul(r1, r1)));
            v[1] = df_add(v[1], df_add(df_mul(r0, z0), df_mul(r1, z1)));
        });
        if (!pr_reduce<2, PrSum>(v, A, S, T, rows, ++tag)) return;
        ++it;
        const int open = tid < Kb && !(df_to_double(S.tot[tid]) <= S.thr[tid]);
        if (!__syncthreads_or(open)) break;
        if (it == A.max_iter) break;
        if (tid < Kb) {
            const DF old = S.rz[tid], now = S.tot[Kb + tid];
            S.a[tid] = old.hi > 0.f ? df_div(now, old) : DF{0.f, 0.f};
            S.rz[tid] = now;
        }
        __syncthreads();
        // P = Z + beta P
        const DF beta = S.a[k];
        pairs([&](int n, int i) {
            DF z0, z1;
            precond(n, ld(r[i]), ld(r[cap + i]), z0, z1);
            const DF p0 = df_add(z0, df_mul(beta, ld(p[i]))), p1 = df_add(z1, df_mul(beta, ld(p[cap + i])));
            p[i] = st(p0);
            p[cap + i] = st(p1);
            put_p(n, p0, p1);
        });
        if (!pr_barrier(A, S, ++phase)) return;
    }
    // 2^(scale - 1023) and the square of the preconditioner's scale
    const double down = __hiloint2double(S.scale[k] << 20, 0), msq = __hiloint2double((1023 - 2 * S.mexp) << 20, 0);
    pairs([&](int n, int i) {
        const size_t i0 = (size_t)n * 2 * A.K + A.k0 + k;
        A.X[i0] = df_to_double(ld(x[i])) * msq * down;
        A.X[i0 + A.K] = df_to_double(ld(x[cap + i])) * msq * down;
    });
    if (blockIdx.x == 0 && tid == 0) atomicMax(A.out, it);
}

// The most launches of pcg_resident for one solve.  On large meshes few columns fit on the chip at a time, and
// every launch reads the whole operator each iteration, once for its columns; the form with its vectors in memory
// reads it once for all.  Per iteration, on the chip (launches) and in memory, in us:
//     nodes     K = 16           32            48             64             96             128            256
//     131,044   123 (4) 608   239 (8) 637   358 (12) 712   494 (16) 722   714 (24) 888   953 (32) 1075  1967 (64) 1943
//     263,169   314 (8) 1209  620 (16) 1248 1005 (24) 1386 1259 (32) 1411 1911 (48) 1738 2684 (64) 2098 4894 (128) 3862
//     330,625   609 (16) 1518 1212 (32) 1560 1831 (48) 1726 2435 (64) 1749 3653 (96) 2161
//     580,644  1285 (16) 2612 2567 (32) 2693 3840 (48) 2997 5134 (64) 3046
// and at 7,569 nodes 23.5 (1) against 75.3 with 64 columns, 167 (8) against 307 with 512.
constexpr int PR_LAUNCHES = 32;

// Columns per launch and blocks of pcg_resident; 0 columns: the vectors do not fit on the chip, or its launches
// are too many.
struct PrPlan {
    int cols, blocks, staged;
    size_t smem;
};
static PrPlan pr_plan(int n_nodes, int K, int sms) {
    PrPlan p = {0, 0, 0, 0};
    if (sms < 1) return p;
    const long long pairs_max = PR_BYTES / PR_PAIR_BYTES - 1;
    int cols = K < PR_COLS ? K : PR_COLS;
    const long long per_all = (n_nodes + sms - 1) / sms;      // nodes per block on the whole chip
    if (per_all * cols > pairs_max) cols = (int)(pairs_max / per_all);
    if (cols < 1 || (K + cols - 1) / cols > PR_LAUNCHES) return p;
    const long long pairs = (long long)n_nodes * cols;
    // one block where it fits (no grid hops); else blocks of at least a pair per thread
    long long blocks = pairs <= PR_ONE_BLOCK ? 1 : (pairs + PR_T - 1) / PR_T;
    if (blocks > sms) blocks = sms;
    while (blocks < sms && ((n_nodes + blocks - 1) / blocks) * cols > pairs_max) ++blocks;
    const long long per = (n_nodes + blocks - 1) / blocks;
    p.cols = cols;
    p.blocks = (int)blocks;
    p.smem = (size_t)((per * cols * PR_PAIR_BYTES + 15) & ~15ll);
    p.staged = p.smem + (size_t)per * PR_NODE_BYTES <= (size_t)PR_BYTES;
    if (p.staged) p.smem += (size_t)per * PR_NODE_BYTES;
    if (p.staged && p.smem + (size_t)per * PR_BLOCK_BYTES <= (size_t)PR_BYTES) {
        p.staged = 2;
        p.smem += (size_t)per * PR_BLOCK_BYTES;
    }
    return p;
}

struct PrWork {
    float *P;
    float2 *M;
    uint4 *part, *tot;
    unsigned *bar;
    int *out;
    char *op;
    size_t zero;                            // bytes from part on to clear before a launch
};
static size_t pr_carve(int n_nodes, int K, int node_chunk_k, char *base, PrWork *w) {
    const int cols = K < PR_COLS ? K : PR_COLS;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off += al256(bytes);
        return p;
    };
    w->P = (float *)take(sizeof(float) * (size_t)n_nodes * 2 * cols);
    w->M = (float2 *)take(sizeof(float2) * 4 * (size_t)n_nodes);
    w->out = (int *)take(2 * sizeof(int));
    const size_t z0 = off;
    w->part = (uint4 *)take(sizeof(uint4) * 2 * (size_t)cols * 1024);   // up to 1024 blocks
    w->tot = (uint4 *)take(sizeof(uint4) * 2 * (size_t)cols);
    w->bar = (unsigned *)take(sizeof(unsigned));
    w->zero = off - z0;
    HopView hv;
    w->op = take(hop_layout(n_nodes, node_chunk_k, nullptr, &hv));
    return off;
}

struct PcgWork {
    double *R, *Z, *P, *part_a, *part_b, *rz, *rz2, *pap, *rr, *bb;
    float *Pf, *AP;
    PcgCtl *ctl;
    char *op;
};

static int pcg_blocks(int n_nodes) {
    int nb = (n_nodes + 15) / 16;                 // >= 16 nodes per block
    return nb < 1 ? 1 : (nb > 1024 ? 1024 : nb);
}

static size_t carve(int n_nodes, int K, int node_chunk_k, char *base, PcgWork *w) {
    const size_t v = (size_t)n_nodes * 2 * K;
    const int nb = pcg_blocks(n_nodes), na = (n_nodes + 7) / 8;
    const int nparts = nb > na ? nb : na;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off += al256(bytes);
        return p;
    };
    w->R = (double *)take(sizeof(double) * v);
    w->Z = (double *)take(sizeof(double) * v);
    w->P = (double *)take(sizeof(double) * v);
    w->Pf = (float *)take(sizeof(float) * v);
    w->AP = (float *)take(sizeof(float) * v);
    w->part_a = (double *)take(sizeof(double) * (size_t)nparts * K);
    w->part_b = (double *)take(sizeof(double) * (size_t)nparts * K);
    w->rz = (double *)take(sizeof(double) * K);
    w->rz2 = (double *)take(sizeof(double) * K);
    w->pap = (double *)take(sizeof(double) * K);
    w->rr = (double *)take(sizeof(double) * K);
    w->bb = (double *)take(sizeof(double) * K);
    w->ctl = (PcgCtl *)take(sizeof(PcgCtl));
    HopView hv;
    w->op = take(hop_layout(n_nodes, node_chunk_k, nullptr, &hv));
    return off;
}

static int assemble(const d2ic_frame_t *frame_dev, int n_chunks, int n_nodes, int node_chunk_k,
                    const float *chunk_hess, float inv_np, float alpha_reg, char *op, cudaStream_t s, HopView *hv) {
    hop_layout(n_nodes, node_chunk_k, op, hv);
    cudaError_t e = cudaMemsetAsync(hv->sids, 0xff, sizeof(int) * (size_t)node_chunk_k * n_nodes * 4, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(hv->err, 0, sizeof(int), s);
    if (e != cudaSuccess) return cuda_status(e, "hessian assembly scratch");
    if (n_chunks > 0) {
        hop_scatter<<<(unsigned)((4 * (size_t)n_chunks + 255) / 256), 256, 0, s>>>(frame_dev, chunk_hess, hv->sids,
                                                                                 hv->sblk);
        D2IC_CHECK_LAUNCH("hop_scatter");
    }
    hop_merge<<<(unsigned)((32 * (size_t)n_nodes + 255) / 256), 256, 0, s>>>(frame_dev, hv->sids, hv->sblk, inv_np,
                                                                           alpha_reg, hv->idx, hv->blk, hv->err);
    D2IC_CHECK_LAUNCH("hop_merge");
    return D2IC_OK;
}

static int check_overflow(const HopView &hv, cudaStream_t s) {
    int err = 0;
    cudaError_t e = cudaMemcpyAsync(&err, hv.err, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e, "hessian assembly");
    D2IC_REQUIRE(err == 0, "hessian assembly: a node couples to more than %d nodes", HOP);
    return D2IC_OK;
}

}  // namespace d2ic

using namespace d2ic;

extern "C" size_t d2ic_hessian_op_bytes(int n_nodes, int node_chunk_k) {
    HopView hv;
    if (n_nodes < 1) n_nodes = 1;
    if (node_chunk_k < 1) node_chunk_k = 1;
    return hop_layout(n_nodes, node_chunk_k, nullptr, &hv);
}

extern "C" int d2ic_hessian_assemble(const d2ic_frame_t *frame_dev, int n_chunks, int n_nodes, int node_chunk_k,
                                     const float *chunk_hess, float inv_np, float alpha_reg, void *op, size_t op_bytes,
                                     void *stream) {
    D2IC_REQUIRE(frame_dev && op && (chunk_hess || n_chunks == 0) && n_nodes >= 1 && node_chunk_k >= 1 && n_chunks >= 0,
                 "d2ic_hessian_assemble: bad arguments");
    D2IC_REQUIRE(((uintptr_t)op & 255) == 0, "d2ic_hessian_assemble: op must be 256-byte aligned");
    D2IC_REQUIRE(op_bytes >= d2ic_hessian_op_bytes(n_nodes, node_chunk_k), "d2ic_hessian_assemble: op buffer too small");
    cudaStream_t s = (cudaStream_t)stream;
    HopView hv;
    int st = assemble(frame_dev, n_chunks, n_nodes, node_chunk_k, chunk_hess, inv_np, alpha_reg, (char *)op, s, &hv);
    if (st) return st;
    return check_overflow(hv, s);
}

extern "C" int d2ic_hessian_apply(const void *op, int n_nodes, int node_chunk_k, const float *V, int K, float *Y,
                                  void *stream) {
    D2IC_REQUIRE(op && V && Y && n_nodes >= 1 && K >= 1 && node_chunk_k >= 1, "d2ic_hessian_apply: bad arguments");
    HopView hv;
    hop_layout(n_nodes, node_chunk_k, (char *)op, &hv);
    if (K % 4 == 0 && ((uintptr_t)V & 15) == 0 && ((uintptr_t)Y & 15) == 0 &&
        (long long)n_nodes * 2 * K < (1ll << 31)) {
        hop_apply4<<<(unsigned)((n_nodes + 7) / 8), 256, 0, (cudaStream_t)stream>>>(hv.idx, hv.blk, n_nodes, V, K,
                                                                                      Y);
        D2IC_CHECK_LAUNCH("hop_apply4");
    } else {
        hop_apply<<<dim3((unsigned)((n_nodes + 7) / 8), (unsigned)((K + 31) / 32)), 256, 0, (cudaStream_t)stream>>>(
            hv.idx, hv.blk, n_nodes, V, K, Y);
        D2IC_CHECK_LAUNCH("hop_apply");
    }
    return D2IC_OK;
}

extern "C" size_t d2ic_pcg_work_bytes(int n_nodes, int K, int node_chunk_k) {
    PcgWork w;
    PrWork r;
    if (n_nodes < 1) n_nodes = 1;
    if (K < 1) K = 1;
    if (node_chunk_k < 1) node_chunk_k = 1;
    const size_t a = carve(n_nodes, K, node_chunk_k, nullptr, &w), b = pr_carve(n_nodes, K, node_chunk_k, nullptr, &r);
    return a > b ? a : b;
}

extern "C" int d2ic_pcg_plan(int n_nodes, int K, int num_sms, int *blocks) {
    const PrPlan p = n_nodes >= 1 && K >= 1 ? pr_plan(n_nodes, K, num_sms < 1024 ? num_sms : 1024) : PrPlan{0, 0, 0, 0};
    if (blocks) *blocks = p.blocks;
    return p.cols;
}

// op: an assembled operator, or null: assembled from chunk_hess into the work buffer first
static int pcg_solve(const d2ic_frame_t *frame_dev, int n_chunks, int n_nodes, int node_chunk_k,
                     const float *chunk_hess, float inv_np, float alpha_reg, const void *op, const double *Minv,
                     const unsigned char *active, const double *B, double *X, int K, double rtol, int max_iter,
                     void *work, size_t work_bytes, int *iters_out, void *stream) {
    D2IC_REQUIRE(((uintptr_t)work & 255) == 0, "d2ic_pcg_solve: work must be 256-byte aligned");
    auto get_operator = [&](char *space, cudaStream_t st, HopView *hv) -> int {
        if (!op) return assemble(frame_dev, n_chunks, n_nodes, node_chunk_k, chunk_hess, inv_np, alpha_reg, space, st, hv);
        hop_layout(n_nodes, node_chunk_k, (char *)op, hv);
        return D2IC_OK;
    };
    const size_t need = d2ic_pcg_work_bytes(n_nodes, K, node_chunk_k);
    D2IC_REQUIRE(work_bytes >= need, "d2ic_pcg_solve: work %zu bytes < %zu needed", work_bytes, need);
    cudaStream_t s = (cudaStream_t)stream;
    HopView hv;
    int dev = 0, sms = 0, smem = 0, coop = 0;
    cudaError_t de = cudaGetDevice(&dev);
    if (de == cudaSuccess) de = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (de == cudaSuccess) de = cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (de == cudaSuccess) de = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (de != cudaSuccess) return cuda_status(de, "d2ic_pcg_solve: device attributes");
    const PrPlan plan = pr_plan(n_nodes, K, sms < 1024 ? sms : 1024);
    // the vectors on the chip where a column of them fits (589,000 nodes on 152 SMs) and few launches take all
    // columns (pr_plan), else in memory
    if (plan.cols > 0 && coop && (size_t)PR_BYTES + sizeof(PrShared) <= (size_t)smem) {
        PrWork r;
        pr_carve(n_nodes, K, node_chunk_k, (char *)work, &r);
        int st = get_operator(r.op, s, &hv);
        if (st) return st;
        cudaError_t e = cudaMemsetAsync(r.out, 0, 2 * sizeof(int), s);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(pcg_resident, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_BYTES);
        if (e != cudaSuccess) return cuda_status(e, "pcg set-up");
        for (int k0 = 0; k0 < K; k0 += plan.cols) {
            PrArgs A;
            A.idx = hv.idx;
            A.blk = hv.blk;
            A.overflow = hv.err;
            A.Minv = Minv;
            A.M = r.M;
            A.act = active;
            A.B = B;
            A.X = X;
            A.P = r.P;
            A.part = r.part;
            A.tot = r.tot;
            A.bar = r.bar;
            A.out = r.out;
            A.n_nodes = n_nodes;
            A.K = K;
            A.k0 = k0;
            A.Kb = K - k0 < plan.cols ? K - k0 : plan.cols;
            A.max_iter = max_iter;
            A.staged = plan.staged;
            A.rtol = rtol;
            e = cudaMemsetAsync(r.part, 0, r.zero, s);
            if (e != cudaSuccess) return cuda_status(e, "pcg records");
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(plan.blocks);
            cfg.blockDim = dim3(PR_T);
            cfg.dynamicSmemBytes = plan.smem;
            cfg.stream = s;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeCooperative;      // the blocks wait for one another
            attr[0].val.cooperative = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            e = cudaLaunchKernelEx(&cfg, pcg_resident, A);
            if (e != cudaSuccess) return cuda_status(e, "cooperative launch of pcg_resident");
        }
        int out[2] = {0, 0}, err = 0;
        e = cudaMemcpyAsync(out, r.out, sizeof(out), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&err, hv.err, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_status(e, "pcg");
        D2IC_REQUIRE(err == 0, "hessian assembly: a node couples to more than %d nodes", HOP);
        if (out[1]) {
            set_error("d2ic_pcg_solve: a wait between blocks ran out");
            return out[1];
        }
        if (iters_out) *iters_out = out[0];
        return D2IC_OK;
    }
    PcgWork w;
    carve(n_nodes, K, node_chunk_k, (char *)work, &w);
    int st = get_operator(w.op, s, &hv);
    if (st) return st;
    cudaError_t e = cudaMemsetAsync(w.ctl, 0, sizeof(PcgCtl), s);
    if (e != cudaSuccess) return cuda_status(e, "pcg control");
    const int nb = pcg_blocks(n_nodes);
    const int rb = (K + 7) / 8;                      // column sums: 8 warps (columns) per block
    pcg_init<<<nb, PT, 0, s>>>(n_nodes, K, B, active, Minv, X, w.R, w.Z, w.P, w.Pf, w.part_a, w.part_b);
    pcg_colsum<<<rb, 256, 0, s>>>(nb, K, w.part_a, w.part_b, w.rz, w.bb, nullptr, 0.0, 0, w.ctl);
    D2IC_CHECK_LAUNCH("pcg init");
    st = check_overflow(hv, s);                      // also waits for the assembly
    if (st) return st;
    const bool vec = K % 4 == 0;                     // Pf and AP are 256-byte aligned
    const int na = (n_nodes + 7) / 8;
    const dim3 ag((unsigned)na, (unsigned)(vec ? (K + 127) / 128 : (K + 31) / 32));
    constexpr int BATCH = 8;                         // iterations launched per host check of the flag
    int it = 0;
    PcgCtl host_ctl = {};
    double *rz = w.rz, *rz_new = w.rz2;
    while (it < max_iter) {
        const int nb_it = max_iter - it < BATCH ? max_iter - it : BATCH;
        for (int i = 0; i < nb_it; ++i) {
            if (vec)
                pcg_apply<true><<<ag, 256, 0, s>>>(hv.idx, hv.blk, n_nodes, K, w.Pf, w.P, active, w.AP, w.part_a, w.ctl);
            else
                pcg_apply<false><<<ag, 256, 0, s>>>(hv.idx, hv.blk, n_nodes, K, w.Pf, w.P, active, w.AP, w.part_a,
                                                    w.ctl);
            pcg_colsum<<<rb, 256, 0, s>>>(na, K, w.part_a, nullptr, w.pap, nullptr, nullptr, 0.0, 0, w.ctl);
            pcg_step<<<nb, PT, 0, s>>>(n_nodes, K, rz, w.pap, active, Minv, X, w.R, w.Z, w.P, w.AP, w.part_a,
                                       w.part_b, w.ctl);
            pcg_colsum<<<rb, 256, 0, s>>>(nb, K, w.part_a, w.part_b, w.rr, rz_new, w.bb, rtol, 1, w.ctl);
            pcg_dir<<<nb, PT, 0, s>>>(n_nodes, K, rz, rz_new, w.Z, w.P, w.Pf, w.ctl);
            double *t = rz;
            rz = rz_new;
            rz_new = t;
        }
        it += nb_it;
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(&host_ctl, w.ctl, sizeof(PcgCtl), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_status(e, "pcg iteration");
        if (host_ctl.done) break;
    }
    if (iters_out) *iters_out = host_ctl.iters;
    return D2IC_OK;
}

extern "C" int d2ic_pcg_solve(const d2ic_frame_t *frame_dev, int n_chunks, int n_nodes, int node_chunk_k,
                              const float *chunk_hess, float inv_np, float alpha_reg, const double *Minv,
                              const unsigned char *active, const double *B, double *X, int K, double rtol,
                              int max_iter, void *work, size_t work_bytes, int *iters_out, void *stream) {
    D2IC_REQUIRE(frame_dev && chunk_hess && Minv && active && B && X && work && K >= 1 && n_nodes >= 1 &&
                     node_chunk_k >= 1 && max_iter >= 0,
                 "d2ic_pcg_solve: bad arguments");
    return pcg_solve(frame_dev, n_chunks, n_nodes, node_chunk_k, chunk_hess, inv_np, alpha_reg, nullptr, Minv, active, B,
                     X, K, rtol, max_iter, work, work_bytes, iters_out, stream);
}

extern "C" int d2ic_pcg_solve_op(const void *op, int n_nodes, int node_chunk_k, const double *Minv,
                                 const unsigned char *active, const double *B, double *X, int K, double rtol,
                                 int max_iter, void *work, size_t work_bytes, int *iters_out, void *stream) {
    D2IC_REQUIRE(op && Minv && active && B && X && work && K >= 1 && n_nodes >= 1 && node_chunk_k >= 1 && max_iter >= 0,
                 "d2ic_pcg_solve_op: bad arguments");
    return pcg_solve(nullptr, 0, n_nodes, node_chunk_k, nullptr, 0.f, 0.f, op, Minv, active, B, X, K, rtol, max_iter, work,
                     work_bytes, iters_out, stream);
}

extern "C" int d2ic_hessian_prepare(const d2ic_frame_t *frame_dev, int n_chunks, int n_nodes, int node_chunk_k,
                                    const float *chunk_hess, float inv_np, float alpha_reg, void *op, size_t op_bytes,
                                    double *Minv, unsigned char *active, void *stream) {
    D2IC_REQUIRE(frame_dev && op && Minv && active && (chunk_hess || n_chunks == 0) && n_nodes >= 1 && node_chunk_k >= 1 &&
                     n_chunks >= 0,
                 "d2ic_hessian_prepare: bad arguments");
    D2IC_REQUIRE(((uintptr_t)op & 255) == 0, "d2ic_hessian_prepare: op must be 256-byte aligned");
    D2IC_REQUIRE(op_bytes >= d2ic_hessian_op_bytes(n_nodes, node_chunk_k), "d2ic_hessian_prepare: op buffer too small");
    cudaStream_t s = (cudaStream_t)stream;
    HopView hv;
    int st = assemble(frame_dev, n_chunks, n_nodes, node_chunk_k, chunk_hess, inv_np, alpha_reg, (char *)op, s, &hv);
    if (st) return st;
    // one warp per block: the FP64 sums and divisions of 7,569 nodes on every SM
    hop_diagonal<<<(n_nodes + 31) / 32, 32, 0, s>>>(frame_dev, hv.sids, hv.sblk, inv_np, alpha_reg, Minv, active);
    D2IC_CHECK_LAUNCH("hop_diagonal");
    return D2IC_OK;
}

extern "C" int d2ic_hessian_check(const void *op, int n_nodes, int node_chunk_k, void *stream) {
    D2IC_REQUIRE(op && n_nodes >= 1 && node_chunk_k >= 1, "d2ic_hessian_check: bad arguments");
    HopView hv;
    hop_layout(n_nodes, node_chunk_k, (char *)op, &hv);
    return check_overflow(hv, (cudaStream_t)stream);
}
