// Persistent cooperative nonlinear-CG engine for the global FE-DIC objective.
//
// One launch solves a batch of independent frames (the plain GlobalCGSolver
// drop-in is a batch of one, run by a one-frame instance of the kernel).  All
// frames advance in lock-step "rounds"; one round evaluates, for every active
// frame, the objective and its gradient at the frame's current candidate point:
//
//   pixel pass   each warp takes chunks (<= 256 pixels of one element) and
//                computes, for the candidate u_c = u + alpha * dir,
//                  r = I2(x + sum_a N_a u_c[a]) - I1,
//                the chunk's sum r^2 (double-float) and its 8 nodal gradient
//                partials sum r * dI2/dx * N_a (FP32), written to the chunk's
//                own node slots as 16-byte records that carry the evaluation's
//                tag.  No atomics on data, no fence.
//   node work    the warp that owns a group of 32 nodes polls (bounded) the
//                group's slots until every chunk that touches it has written
//                this evaluation's records, adds the spring gradient over the
//                neighbour table, writes the trial gradient, point and
//                direction, and reduces (fixed order) sum r^2, spring energy,
//                g.g, g.(g - g_cur), g_cur.dir; the warp that completes a
//                supergroup of 16 groups reduces it and publishes its sums as
//                tagged records.
//   control      one warp per frame waits for the supergroup records and runs
//                the CG control of d2ic/solver_global_cg.py:362-461 (stop test,
//                PR+ beta, restart on g.d >= 0, Armijo with 10 halvings and
//                the forced 2^-10 step) and publishes the frame's next candidate
//                rule as a tagged record; a block goes on when it has the records
//                of all active frames (more than FS frames: the round's last
//                frame releases the next round for all).
//
// A round of a small frame is a chain of such hand-overs.  With counters and
// fences (count the chunks of a group, poll the counter, gather; supergroup
// and frame counters; state, fence, release word, header and state read back)
// it took 17.9 us on a 512 x 512 frame with 16-px elements, 23.5 us at
// 1024 x 1024 and 41.1 us at 2048 x 2048; with tagged records, rolled and
// smaller once-per-round code and even shares of the chunks 11.6, 14.0 and
// 31.4 us, and with the pixel pass below 10.1, 14.0 and 27.0 us.  What bounds it now: the L2 round trips of the hand-overs (about
// 0.7 us each), the fences that order the node data (0.4 us each) and, from
// 2048 x 2048 on, the pixel pass.
//
// Because every partial is written to its own slot and reduced in an order
// fixed by the frame's own data layout, a frame's result does not depend on
// which warps processed it or on which other frames shared the launch.
//
// The gradient at an accepted line-search point is produced by the same pass
// that evaluated it, so an iteration costs one pixel pass per line-search
// trial (the reference's separate value_and_grad pass is not repeated).
//
// Every wait is bounded by the globaltimer (the launch's grid barrier, the group
// and round waits: WAIT_NS; the TMA/cp.async completions: TMA_WAIT_NS): a warp
// that waits longer sets D2IC_WAIT_TIMEOUT and an abort flag, drains its own
// copies and every block leaves the kernel.
#include <cuda.h>   // CUtensorMap and its enums (the encoder is fetched from the driver at run time)
#include <stddef.h>
#include <string.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"

namespace d2ic {

constexpr int NT = 512;                        // threads per block
constexpr int NWARP = NT / 32;
static_assert(NWARP == 16, "a supergroup is the warps of one block");
constexpr int GN = D2IC_NODE_GROUP;            // nodes per group: one per lane of the warp that reduces it
static_assert(GN == 32, "a node group is one warp");
// Groups per supergroup.  A frame's group range in the active list is padded to a multiple of
// SG, so when every warp owns at most one group, supergroup sg of a frame is owned by warps
// 0 .. SG-1 of one block and is reduced through that block's shared memory.
constexpr int SG = 16;
__host__ __device__ constexpr int pad_groups(int n) { return (n + SG - 1) / SG * SG; }
#ifndef D2IC_ENGINE_MINB
#define D2IC_ENGINE_MINB 1   // resident blocks per SM the register budget is sized for
#endif
constexpr unsigned long long WAIT_NS = 5ull * 1000ull * 1000ull * 1000ull;

enum { ST_EVAL = 0, ST_TRIAL = 1, ST_FORCED = 2, ST_DONE = 3 };
enum { P_JSUM = 0, P_EREG = 1, P_GG = 2, P_GDIFF = 3, P_GD = 4 };

struct FrameState {
    double J_cur, gg_cur, gg_prev, gdiff_cur, gd, J_last, gnorm;
    float alpha, beta;
    int state, k, t, restart, gd_known, nan_seen;
    int iu, igp, igc, igt, idp;
    int n_evals;
    int reported;   // outputs of a finished frame were written by an earlier launch
    int pad2_;
};

// per-frame commands written by the host between launches (control block, after the header)
enum { CMD_INIT = 0, CMD_RUN = 1, CMD_IDLE = 2, CMD_HOLD = 3 };

struct CtlHeader {
    unsigned bar_count;
    unsigned bar_gen;
    int abort;
    int err;
    int n_active;
    int total_chunks;
    int total_groups;
    int pad0_;
    int finished;           // a frame finished in this round: the active list is rebuilt before release
    int max_rounds;
    int frames_done;        // frames whose control step ran in the current round
    int slice_stop;         // the slice ends after the released round (set before the release)
    int irq;                // written by the host while a slice runs: end the slice at the next round end
    int list_buf;           // which of the two copies of the active list the current round reads
    unsigned blocks_past;   // block arrivals at round ends: every block has finished a round's list reads
    int pad_[17];
    uint4 rel;              // the release record of the last completed round, on a cache line of its own
};
static_assert(sizeof(CtlHeader) == 144 && offsetof(CtlHeader, rel) == 128, "control header layout");

// stop_flags of a slice: end it early
enum { STOP_ON_FINISH = D2IC_STOP_ON_FINISH,   // after a round in which a frame finished
       STOP_ON_IRQ = D2IC_STOP_ON_IRQ };         // after a round that ends with the header's irq word set

// The active list is double-buffered: a round reads copy h->list_buf while the warp that ends
// the round may rebuild the list into the other copy (a frame finished) and flips list_buf before
// the release.  Warps still walking the round's list -- lookups of padding groups, or the
// rebuilding warp itself after the release -- therefore never see a half-written list.  Before it
// writes, the rebuilding warp of round r waits until every block has passed the end of round r-1
// (blocks_past), so no block still reads an older round's copy either.
struct Ctl {
    CtlHeader *h;
    int *cmd;      // n_frames: CMD_INIT / CMD_RUN / CMD_IDLE / CMD_HOLD
    int *active;   // two copies of n_frames
    int *cpre;     // two copies of n_frames + 1
    int *gpre;     // two copies of n_frames + 1
    FrameState *fs;
    uint4 *rule;   // n_frames: candidate rule of the next round, as a tagged record (direct rounds)
    int n;         // n_frames
    __device__ __forceinline__ int *act(int b) const { return active + b * n; }
    __device__ __forceinline__ int *cp(int b) const { return cpre + b * (n + 1); }
    __device__ __forceinline__ int *gp(int b) const { return gpre + b * (n + 1); }
    // n_frames: tag of the evaluation of the launch's first round, constant while it runs
    __device__ __forceinline__ unsigned *tag0() const { return reinterpret_cast<unsigned *>(rule + n); }
};

__host__ __device__ inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// control block: header | cmd | active | cpre | gpre | frame states | rule records | first tags
__host__ __device__ inline size_t ctl_layout(int n, size_t *o_active, size_t *o_cpre, size_t *o_gpre, size_t *o_fs,
                                             size_t *o_rule) {
    size_t off = align256(sizeof(CtlHeader));
    off = align256(off + sizeof(int) * (size_t)n);          // cmd
    *o_active = off;                                        // two copies of each list array
    off = align256(off + 2 * sizeof(int) * (size_t)n);
    *o_cpre = off;
    off = align256(off + 2 * sizeof(int) * (size_t)(n + 1));
    *o_gpre = off;
    off = align256(off + 2 * sizeof(int) * (size_t)(n + 1));
    *o_fs = off;
    off = (off + sizeof(FrameState) * (size_t)n + 15) & ~(size_t)15;
    *o_rule = off;
    off = align256(off + (sizeof(uint4) + sizeof(unsigned)) * (size_t)n);   // Ctl::tag0 behind the records
    return off;
}

__device__ inline Ctl make_ctl(char *base, int n) {
    size_t oa, oc, og, of, orl;
    ctl_layout(n, &oa, &oc, &og, &of, &orl);
    Ctl c;
    c.h = (CtlHeader *)base;
    c.cmd = (int *)(base + align256(sizeof(CtlHeader)));
    c.active = (int *)(base + oa);
    c.cpre = (int *)(base + oc);
    c.gpre = (int *)(base + og);
    c.n = n;
    c.fs = (FrameState *)(base + of);
    c.rule = (uint4 *)(base + orl);
    return c;
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ int ld_vol(const int *p) { return *(volatile const int *)p; }

// Warp sums of five double-floats by a reduce-scatter butterfly: at the exchange distances 16, 8 and 4
// a lane keeps half of its values and adds its partner's copy of that half, so the five sums take 8
// double-float additions instead of 25; the additions of each sum are those of df_warp_sum, so the bits
// are the same.  Lane l returns sum red5_value(l), each sum in four lanes (-1: none).  (This code runs
// once per round on one warp of an SM: its instruction count is latency.)
__device__ __forceinline__ int red5_value(int lane) {
    const int k = lane >> 2;               // lanes 0-3: sum 0, 4-7: 1, 8-11: 2, 16-19: 3, 20-23: 4
    return k < 3 ? k : (k == 4 ? 3 : (k == 5 ? 4 : -1));
}
__host__ __device__ constexpr int red5_lane(int k) { return k < 3 ? 4 * k : 4 * k + 4; }
__device__ __forceinline__ DF df_shfl_xor(DF v, int o) {
    return DF{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
}
__device__ __forceinline__ DF df_reduce5(const DF q[5], int lane) {
    const DF z = {0.f, 0.f};
    const bool b4 = (lane & 16) != 0, b3 = (lane & 8) != 0, b2 = (lane & 4) != 0;
    const DF a0 = df_add(b4 ? q[3] : q[0], df_shfl_xor(b4 ? q[0] : q[3], 16));
    const DF a1 = df_add(b4 ? q[4] : q[1], df_shfl_xor(b4 ? q[1] : q[4], 16));
    const DF a2 = df_add(b4 ? z : q[2], df_shfl_xor(b4 ? q[2] : z, 16));
    const DF c0 = df_add(b3 ? a2 : a0, df_shfl_xor(b3 ? a0 : a2, 8));
    const DF c1 = df_add(b3 ? z : a1, df_shfl_xor(b3 ? a1 : z, 8));
    DF v = df_add(b2 ? c1 : c0, df_shfl_xor(b2 ? c0 : c1, 4));
    v = df_add(v, df_shfl_xor(v, 2));
    return df_add(v, df_shfl_xor(v, 1));
}

// node buffers of a frame: 0,1 = u ; 2,3,4 = g ; 5,6 = d
__device__ __forceinline__ float2 *nbuf(const d2ic_frame_t &F, int j) {
    return reinterpret_cast<float2 *>(F.node_ws) + (size_t)j * F.n_nodes;
}

// Candidate point of the current round: u (EVAL) or u + alpha * dir with
// dir = -g (restart / first iteration) or -g + beta * d_prev.  Explicit
// round-to-nearest operations so that the P and N phases produce identical bits.
// mode 0: u, 1: conjugate direction, 2: steepest descent.
__device__ __forceinline__ float2 cand_value(float2 un, float2 gn, float2 dn, float alpha, float beta, int mode,
                                             float2 &dir) {
    if (mode == 0) {
        dir = make_float2(0.f, 0.f);
        return un;
    }
    float dx = -gn.x, dy = -gn.y;
    if (mode == 1) {
        dx = __fadd_rn(dx, __fmul_rn(beta, dn.x));
        dy = __fadd_rn(dy, __fmul_rn(beta, dn.y));
    }
    dir = make_float2(dx, dy);
    return make_float2(__fadd_rn(un.x, __fmul_rn(alpha, dx)), __fadd_rn(un.y, __fmul_rn(alpha, dy)));
}

// The candidate rule of a frame for the current round, read from its state
// with L2 loads (rewritten by other blocks; not volatile, so that the reads are in flight together).
struct FInfo {
    float alpha, beta;
    int mode, iu, igc, idp, igt;
    unsigned tag;   // this evaluation's tag: the frame's evaluations so far, plus one (28 bits used)
};
constexpr unsigned TAG_MASK = 0x0fffffffu;
// Every active frame takes one evaluation per round, so its tag is that of the launch's first round plus the
// rounds completed.  It is not read from the state: a block that has no work of the frame waits for none of the
// frame's control steps and may read a state that is already an evaluation ahead.  The rest of such a rule is
// never used (a list in which the block has work of the frame is followed by another read), a tag kept from it
// would stay wrong.  With STATE_TAG it is read from the state: a launch of one frame, whose list does not change,
// so that a block without work stays without (read from the control block there, an evaluation at 2048 x 2048 takes
// 0.6 % longer: other code for the pixel pass).
__device__ __forceinline__ unsigned frame_tag(const Ctl &C, int f, int rounds) {
    return (__ldcg(C.tag0() + f) + (unsigned)rounds) & TAG_MASK;
}
template <bool STATE_TAG = false>
__device__ __forceinline__ FInfo frame_info(const Ctl &C, int f, int rounds) {
    const FrameState *S = C.fs + f;
    FInfo fi;
    fi.iu = __ldcg(&S->iu);
    fi.igc = __ldcg(&S->igc);
    fi.idp = __ldcg(&S->idp);
    fi.igt = __ldcg(&S->igt);
    const int st = __ldcg(&S->state), k = __ldcg(&S->k), rs = __ldcg(&S->restart);
    fi.alpha = __ldcg(&S->alpha);
    fi.beta = __ldcg(&S->beta);
    fi.mode = (st == ST_EVAL) ? 0 : ((rs || k == 0) ? 2 : 1);
    fi.tag = STATE_TAG ? ((unsigned)__ldcg(&S->n_evals) + 1u) & TAG_MASK : frame_tag(C, f, rounds);
    return fi;
}

// The release of a round: one record, polled by one thread of every block.  x: rounds completed in
// this launch; y: bit 0 the launch's slice ends, bit 1 the candidate rule of the only active frame
// is in the record (mode, buffer indices in bits 2-9; alpha, beta in z, w), bits 16-31 the version
// of the active list.  With several active frames the rules are read from the frame states.
//
// Several frames, up to FS of them with a control warp each ("direct" rounds): there is no common
// release.  Each control warp publishes its frame's next rule as a record of the same form (x: rounds
// completed, REL_FIN: the frame is finished), and a block goes on when it has seen the records of all
// active frames.  Only after a round in which a frame finished does everybody wait for a release record, with
// the new list.  A frame without work in a block may be ahead of that block by a round; its flags count
// only in the record of the round that the block waits for.
constexpr unsigned REL_STOP = 1u, REL_INLINE = 2u, REL_FIN = 1u << 12;
//
// 2 frames of 911 and 1,535 chunks: 19.2 -> 14.9 us per round; 12 frames of together 46,106 chunks: 85.4 ->
// 81.7 us (with the descriptors of the active frames in shared memory).
constexpr int FS = 16;         // frames with direct rounds: their descriptors fit the block's static shared memory
enum { REFRESH_NONE = 0, REFRESH_RULES = 1, REFRESH_LIST = 2 };   // what a block reads after a release
__device__ __forceinline__ unsigned rel_pack(const FInfo &fi) {
    return REL_INLINE | ((unsigned)fi.mode << 2) | ((unsigned)fi.iu << 4) | ((unsigned)fi.igc << 5) |
           ((unsigned)fi.igt << 7) | ((unsigned)fi.idp << 9);
}

// A candidate rule as a block keeps it in shared memory, 16 bytes.
struct FRule {
    float alpha, beta;
    unsigned packed, tag;   // packed: as in the release record
    __device__ __forceinline__ FInfo info() const {
        FInfo fi;
        fi.alpha = alpha;
        fi.beta = beta;
        fi.tag = tag;
        fi.mode = (int)((packed >> 2) & 3u);
        fi.iu = (int)((packed >> 4) & 1u);
        fi.igc = (int)((packed >> 5) & 3u);
        fi.igt = (int)((packed >> 7) & 3u);
        fi.idp = (int)((packed >> 9) & 1u);
        return fi;
    }
};
__device__ __forceinline__ FRule make_rule(const FInfo &fi) { return FRule{fi.alpha, fi.beta, rel_pack(fi), fi.tag}; }

struct Cand {
    const float2 *u, *g, *d;
    float alpha, beta;
    int mode;
    __device__ __forceinline__ float2 at(int n, float2 &dir) const {
        const float2 un = __ldcg(u + n);
        const float2 gn = mode != 0 ? __ldcg(g + n) : make_float2(0.f, 0.f);
        const float2 dn = mode == 1 ? __ldcg(d + n) : make_float2(0.f, 0.f);
        return cand_value(un, gn, dn, alpha, beta, mode, dir);
    }
};

__device__ __forceinline__ Cand make_cand(const d2ic_frame_t &F, const FInfo &fi) {
    Cand c;
    c.u = nbuf(F, fi.iu);
    c.g = nbuf(F, 2 + fi.igc);
    c.d = nbuf(F, 5 + fi.idp);
    c.alpha = fi.alpha;
    c.beta = fi.beta;
    c.mode = fi.mode;
    return c;
}

// ---------------------------------------------------------------------------
// grid barrier (cooperative launch guarantees co-residency)
// ---------------------------------------------------------------------------
template <class F>
__device__ bool grid_barrier(CtlHeader *H, F &&on_last) {
    __shared__ int s_last;
    __shared__ unsigned s_gen;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned gen = ld_acquire_u32(&H->bar_gen);
        __threadfence();
        const unsigned t = atomicAdd(&H->bar_count, 1u);
        s_last = (t == gridDim.x - 1);
        s_gen = gen;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        on_last();
        __syncthreads();
        if (threadIdx.x == 0) {
            H->bar_count = 0;
            __threadfence();
            atomicExch(&H->bar_gen, s_gen + 1);
        }
    } else if (threadIdx.x == 0) {
        const unsigned long long t0 = gtimer();
        while (ld_acquire_u32(&H->bar_gen) == s_gen) {
            if (ld_vol(&H->abort)) break;
            if (gtimer() - t0 > WAIT_NS) {
                H->err = D2IC_WAIT_TIMEOUT;
                atomicExch(&H->abort, 1);
                break;
            }
            __nanosleep(100);
        }
        __threadfence();
    }
    __syncthreads();
    return ld_vol(&H->abort) == 0;
}

// largest s in [0, n) with pre[s] <= x (pre ascending, pre[0] == 0)
__device__ __forceinline__ int find_slot(const int *pre, int n, int x) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldcg(pre + mid) <= x) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// the same search over a copy of the prefix sums in shared memory
__device__ __forceinline__ int find_slot_smem(const int *pre, int n, int x) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pre[mid] <= x) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Self-check of an index taken from the active list or its prefix sums: in [0, n) it is returned;
// otherwise the launch aborts with D2IC_INTERNAL and 0 is returned, so that the access it guards
// stays inside its table.
__device__ __forceinline__ int checked_index(int v, int n, CtlHeader *H) {
    if ((unsigned)v < (unsigned)n) return v;
    H->err = D2IC_INTERNAL;
    atomicExch(&H->abort, 1);
    return 0;
}

// ---------------------------------------------------------------------------
// P phase: one chunk per warp at a time
// ---------------------------------------------------------------------------
// Each warp walks its chunks (a contiguous range for one frame, c, c + W,
// c + 2W, ... for W warps in the grid with several) in batches of 32, one chunk
// per lane.  What a chunk needs besides its pixels is done for the batch at once,
// by the chunk's lane and with all loads in flight together: its metadata (pixel
// range, nodes, slots, tile origin), the nodal candidates (u + alpha dir at its
// four nodes), whether its stencils all lie inside its tile, and the tile origin
// of the next pass.  The warp then takes the chunks one by one:
//   chunk i + 1: pixel records copied into the warp's shared-memory buffer by
//                one TMA bulk copy (cp.async.bulk, completion on an mbarrier),
//                and its window of the deformed image's coefficients (tile_w x
//                tile_h floats) by a 2-D TMA copy on the same mbarrier, both
//                issued by the chunk's lane;
//   chunk i:     values broadcast from its lane, sampled and reduced.
// The window is placed from the chunk's candidate of the previous pass, with a
// margin of TILE_MARGIN pixels on every side (stored per chunk in
// chunk_tile); a pixel whose 4x4 stencil is not inside it (a larger move, the
// first pass) reads global memory with the same arithmetic.
//
// With the per-chunk work done by the whole warp and scalar pixel arithmetic a
// 256-pixel chunk took about 2,000 issue slots, 650 of them besides the pixels, and
// the pass ran at 92 % of the issue rate.  Lane batches and two pixels per
// instruction leave about 1,150: per evaluation 31.4 -> 27.4 us at 2048 x 2048 with
// 16-px elements, 62.7 -> 40.5 us with 8-px elements, 219 -> 149 us at 4096 x 4096
// with 8-px elements.  A pass without the coefficient tiles' traffic takes 0.5 us
// less at 2048 x 2048: what bounds it now is the FMA pipe (60 % busy during the pass)
// with 4 warps per scheduler to hide its latencies, not the L2.
constexpr int CHUNK_BYTES = D2IC_CHUNK_MAX * 16;            // one staged record buffer
constexpr int TILE_BYTES = D2IC_TILE_MAX_FLOATS * 4;        // one staged coefficient tile
static_assert(TILE_BYTES % 128 == 0, "tile buffers keep 128-byte alignment");
constexpr int WARP_SMEM = 2 * CHUNK_BYTES + 2 * TILE_BYTES;
constexpr int TILE_MARGIN = 2;
constexpr int TILE_NONE = (int)0x80008000u;                 // no valid origin (col = row = -32768)
constexpr unsigned long long TMA_WAIT_NS = 200ull * 1000ull * 1000ull;
constexpr int FCACHE = 64;    // active frames whose per-round lookup data is kept in shared memory

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(unsigned long long *b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
// 1-D TMA: global -> this CTA's shared memory, completion counted on mbarrier b
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(b))
                 : "memory");
}
// 2-D TMA: the tensor map's box at tensor coordinates (x, y) -> shared memory
__device__ __forceinline__ void tensor_load_2d(void *dst, const void *map, int x, int y, unsigned long long *b) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(smem_addr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_addr(b))
        : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long *b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_addr(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// false if the phase did not complete within TMA_WAIT_NS
__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity) {
    if (mbar_test(b, parity)) return true;
    const unsigned long long t0 = gtimer();
    while (!mbar_test(b, parity))
        if (gtimer() - t0 > TMA_WAIT_NS) return false;
    return true;
}

// A chunk as its lane holds it from the load to the candidates.
struct ChunkMeta {
    int f, c, pb, n;                 // frame (its key), chunk within the frame, first pixel, pixels
    int box0, box1;                  // packed pixel-box corners
    int origin, flags;               // packed tile origin (TMA column, row), CH_* bits
    int4 nd;                         // nodes
    unsigned slot;                   // slot rank of node a in byte a
};
enum { CH_STAGED = 1, CH_TILED = 2, CH_FAST = 4 };   // records / tile in shared memory; no pixel leaves the tile

// Lane's chunk c of frame f.  chunk_tile is rewritten every pass: read from L2.
template <int KIND>
__device__ __forceinline__ ChunkMeta load_meta(const d2ic_frame_t &F, int f, int c, bool tiles_ok) {
    ChunkMeta m;
    m.f = f;
    m.c = c;
    m.pb = __ldg(F.chunk_begin + c);
    m.n = max(__ldg(F.chunk_begin + c + 1) - m.pb, 0);
    m.box0 = __ldg(F.chunk_box + 2 * c);
    m.box1 = __ldg(F.chunk_box + 2 * c + 1);
    m.nd = make_int4(__ldg(F.chunk_nodes + 4 * c), __ldg(F.chunk_nodes + 4 * c + 1), __ldg(F.chunk_nodes + 4 * c + 2),
                     __ldg(F.chunk_nodes + 4 * c + 3));
    m.slot = (unsigned)__ldg(F.chunk_slot + c);
    m.flags = m.n > 0 && ((reinterpret_cast<uintptr_t>(F.pix) & 15) == 0) ? CH_STAGED : 0;
    m.origin = 0;
    if (KIND == D2IC_INTERP_CUBIC && tiles_ok && F.tile_w > 0) {
        const int tile = __ldcg(F.chunk_tile + c);
        const int tx0 = (int)(short)(tile & 0xffff) & ~3;            // TMA x: a multiple of 4 floats
        const int ty0 = (int)(short)((unsigned)tile >> 16);
        m.origin = (tx0 & 0xffff) | (int)((unsigned)ty0 << 16);
        if (tile != TILE_NONE && tx0 >= -F.pad && ty0 >= -F.pad && tx0 + F.tile_w <= F.W + F.pad &&
            ty0 + F.tile_h <= F.H + F.pad)                           // inside the halo'd array: no fill
            m.flags |= CH_TILED;
    }
    return m;
}

// Tile origin for the next pass from this pass's nodal candidates: the
// smallest tap column / row any pixel of the chunk can reach, less the margin.
__device__ __forceinline__ int tile_origin(int box0, const float ux[4], const float uy[4]) {
    const float mnx = fminf(fminf(ux[0], ux[1]), fminf(ux[2], ux[3]));
    const float mny = fminf(fminf(uy[0], uy[1]), fminf(uy[2], uy[3]));
    const int ox = (box0 & 0xffff) + (int)safe_floor(mnx) - 1 - TILE_MARGIN;
    const int oy = (int)((unsigned)box0 >> 16) + (int)safe_floor(mny) - 1 - TILE_MARGIN;
    if (ox <= -32768 || ox >= 32768 || oy <= -32768 || oy >= 32768) return TILE_NONE;   // also NaN candidates
    return (ox & 0xffff) | (int)((unsigned)oy << 16);
}

__device__ __forceinline__ int atom_acq_rel_add(int *p, int v) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// Whole chunk inside its tile: a pixel's displacement is a convex combination of its
// element's nodal candidates, so its stencil corner lies in the chunk's pixel box shifted by
// [floor(min u), floor(max u)] (taken with 0.5 px of slack).  Then no pixel needs the
// per-pixel test or the global-memory path.
__device__ __forceinline__ bool inside_tile(const d2ic_frame_t &F, const ChunkMeta &m, const float ux[4], const float uy[4]) {
    bool fin = true;
#pragma unroll
    for (int a = 0; a < 4; ++a) fin = fin && isfinite(ux[a]) && isfinite(uy[a]);
    if (!fin) return false;
    const float mnx = fminf(fminf(ux[0], ux[1]), fminf(ux[2], ux[3]));
    const float mxx = fmaxf(fmaxf(ux[0], ux[1]), fmaxf(ux[2], ux[3]));
    const float mny = fminf(fminf(uy[0], uy[1]), fminf(uy[2], uy[3]));
    const float mxy = fmaxf(fmaxf(uy[0], uy[1]), fmaxf(uy[2], uy[3]));
    const int tx0 = (int)(short)(m.origin & 0xffff), ty0 = (int)(short)((unsigned)m.origin >> 16);
    const int lx0 = (m.box0 & 0xffff) + (int)safe_floor(mnx - 0.5f) - 1 - tx0;
    const int lx1 = (m.box1 & 0xffff) + (int)safe_floor(mxx + 0.5f) - 1 - tx0;
    const int ly0 = (int)((unsigned)m.box0 >> 16) + (int)safe_floor(mny - 0.5f) - 1 - ty0;
    const int ly1 = (int)((unsigned)m.box1 >> 16) + (int)safe_floor(mxy + 0.5f) - 1 - ty0;
    return lx0 >= 0 && lx1 <= F.tile_w - 4 && ly0 >= 0 && ly1 <= F.tile_h - 4;
}

// What the chunk's lane keeps for the pixel loop
struct ChunkWork {
    int f, pb, n, origin;
    unsigned flags;              // CH_* bits; bits 4 + 4a ..: low bits of node a's record (see gather_slots)
    unsigned tag;                // the evaluation's tag
    float ux[4], uy[4];          // nodal candidates
    int rec[4];                  // node a's record among the frame's slots
};

// The sum over the warp of values v >= 0 (or NaN): the values as 54-bit fixed-point numbers relative to
// the largest, summed by integer warp reductions (a double-float butterfly takes five dependent steps of
// two shuffles and an 11-operation sum).  Error: below 2^-47 of the sum, and at most 2^-48.0 in 12,000 simulated sums
// of values of equal and very different size, where the butterfly's is up to 2^-47.0 (RMS 2^-50 to 2^-52 both).
__device__ __forceinline__ DF warp_sum_nonneg(float v) {
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(v)), e = m >> 23;
    if (e < 27u || e >= 255u) return df_warp_sum(DF{v, 0.f});          // tiny, infinite or NaN: the same for all lanes
    const float q = v * __uint_as_float((280u - e) << 23);             // < 2^27
    const unsigned hi = (unsigned)q;
    const unsigned lo = (unsigned)((q - (float)hi) * 134217728.f);     // 27 more bits
    unsigned sh = __reduce_add_sync(0xffffffffu, hi);
    const unsigned sl = __reduce_add_sync(0xffffffffu, lo);
    sh += sl >> 27;
    const float h = __uint2float_rz(sh);
    const float l = __fmaf_rn((float)(sl & 0x7ffffffu), 7.450580596923828125e-9f, (float)(sh - (unsigned)h));
    const float back = __uint_as_float((e - 26u) << 23);
    return {h * back, l * back};
}

// One chunk by the whole warp, its values broadcast from lane `src`.
template <int KIND>
__device__ __forceinline__ void chunk_compute(const d2ic_frame_t &F, const ChunkWork &w, int src, const uint4 *srec,
                                              const float *tile, int lane) {
    const unsigned flags = __shfl_sync(0xffffffffu, w.flags, src);
    const int origin = __shfl_sync(0xffffffffu, w.origin, src);
    const int n = __shfl_sync(0xffffffffu, w.n, src);
    const bool staged = (flags & CH_STAGED) != 0;
    const bool tiled = KIND == D2IC_INTERP_CUBIC && (flags & CH_TILED) != 0;
    const bool fast = KIND == D2IC_INTERP_CUBIC && (flags & CH_FAST) != 0;
    const int tw = F.tile_w, th = F.tile_h;
    const int tx0 = (int)(short)(origin & 0xffff), ty0 = (int)(short)((unsigned)origin >> 16);
    float ux[4], uy[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        ux[a] = __shfl_sync(0xffffffffu, w.ux[a], src);
        uy[a] = __shfl_sync(0xffffffffu, w.uy[a], src);
    }
    float jr = 0.f;
    float gxa[4] = {0.f, 0.f, 0.f, 0.f}, gya[4] = {0.f, 0.f, 0.f, 0.f};
    // fast path, two pixels per lane and step (p and p + 32): the arithmetic of `one`, in packed operations
    // (about 180 instead of 330 issue slots per step).
    // floor(d) is d + 1.5 * 2^23 rounded down, less 1.5 * 2^23 (exact: here |d| < 2^16), whose low bits are the
    // integer for the tap index; the index is limited to the tile only as a guard of the shared-memory
    // bounds (it is already inside).
    auto two_fast = [&](int p, const Pair ux2[4], const Pair uy2[4], unsigned corner, unsigned limit) {
        const uint4 ra = srec[min(p, n - 1)], rb = srec[min(p + 32, n - 1)];
        constexpr float MAGIC = 12582912.f;
        Pair N[4];
        shape4(pair(__uint_as_float(ra.z), __uint_as_float(rb.z)), pair(__uint_as_float(ra.w), __uint_as_float(rb.w)), N);
        const Pair dx = shape_sum(N, ux2), dy = shape_sum(N, uy2);
        const Pair mx = pair_add_down(dx, pair(MAGIC)), my = pair_add_down(dy, pair(MAGIC));
        const Pair tx = pair_add(dx, pair_fma(mx, pair(-1.f), pair(MAGIC)));
        const Pair ty = pair_add(dy, pair_fma(my, pair(-1.f), pair(MAGIC)));
        const unsigned ia = ((ra.x >> 16) + (unsigned)my) * (unsigned)tw + (ra.x & 0xffffu) + (unsigned)mx + corner;
        const unsigned ib = ((rb.x >> 16) + (unsigned)(my >> 32)) * (unsigned)tw + (rb.x & 0xffffu) + (unsigned)(mx >> 32) + corner;
        Pair gx, gy;
        const Pair v = sample_cubic_tile2(tile, tw, min(ia, limit), min(ib, limit), tx, ty, gx, gy);
        Pair r = pair_fma(pair(__uint_as_float(ra.y), __uint_as_float(rb.y)), pair(-1.f), v);
        r = pair(p < n ? pair_lo(r) : 0.f, p + 32 < n ? pair_hi(r) : 0.f);
        jr = __fmaf_rn(pair_lo(r), pair_lo(r), jr);
        jr = __fmaf_rn(pair_hi(r), pair_hi(r), jr);
        const Pair rgx = pair_mul(r, gx), rgy = pair_mul(r, gy);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            gxa[a] = __fmaf_rn(pair_hi(rgx), pair_hi(N[a]), __fmaf_rn(pair_lo(rgx), pair_lo(N[a]), gxa[a]));
            gya[a] = __fmaf_rn(pair_hi(rgy), pair_hi(N[a]), __fmaf_rn(pair_lo(rgy), pair_lo(N[a]), gya[a]));
        }
    };
    auto one = [&](const Img &im, const uint4 r4) {

        const int x = (int)(r4.x & 0xffffu), y = (int)(r4.x >> 16);
        const float I1 = __uint_as_float(r4.y);
        float N[4];
        shape4(__uint_as_float(r4.z), __uint_as_float(r4.w), N);
        int ix, iy;
        float tx, ty;
        split_coord(x, shape_sum(N, ux), ix, tx);
        split_coord(y, shape_sum(N, uy), iy, ty);
        float gx, gy, v;
        const int lx = ix - 1 - tx0, ly = iy - 1 - ty0;   // stencil corner inside the tile
        if (tiled && (unsigned)lx <= (unsigned)(tw - 4) && (unsigned)ly <= (unsigned)(th - 4))
            v = sample_cubic_tile(tile, tw, lx, ly, tx, ty, gx, gy);
        else
            v = sample<KIND>(im, ix, iy, tx, ty, gx, gy);
        const float r = v - I1;
        jr = __fmaf_rn(r, r, jr);
        const float rgx = r * gx, rgy = r * gy;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            gxa[a] = __fmaf_rn(rgx, N[a], gxa[a]);
            gya[a] = __fmaf_rn(rgy, N[a], gya[a]);
        }
    };
    if (fast) {
        Pair ux2[4], uy2[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            ux2[a] = pair(ux[a]);
            uy2[a] = pair(uy[a]);
        }
        // a pixel's tap index: (y + floor(dy) - 1 - ty0) tw + (x + floor(dx) - 1 - tx0), modulo 2^32
        const unsigned corner = 0u - (0x4b400000u + 1u + (unsigned)ty0) * (unsigned)tw - (0x4b400000u + 1u + (unsigned)tx0);
        const unsigned limit = (unsigned)((th - 4) * tw + tw - 4);
#pragma unroll 1
        for (int p = lane; p - lane < n; p += 64) two_fast(p, ux2, uy2, corner, limit);
    } else {
        // boundary chunks and the first pass: one copy of the general per-pixel code (this loop's body
        // is several times the fast one's; the instruction cache matters more here than its speed)
        const Img im{F.coeff, F.W, F.H, F.cpitch, F.pad};
        const uint4 *gpix = reinterpret_cast<const uint4 *>(F.pix) + __shfl_sync(0xffffffffu, w.pb, src);
#pragma unroll 1
        for (int p = lane; p < n; p += 32) one(im, staged && p < D2IC_CHUNK_MAX ? srec[p] : __ldg(gpix + p));
    }
    const DF js = warp_sum_nonneg(jr);
    // The 8 nodal partials summed over the warp by a reduce-scatter butterfly: at each of the
    // steps over lane bits 4, 3, 2 a lane keeps half of its values and adds its partner's copy of
    // that half (7 shuffles instead of 40); bits 1, 0 finish the sums.  Value k = (gx_0..3,
    // gy_0..3)[k] ends in lane 16 (k >> 2) + 8 ((k >> 1) & 1) + 4 (k & 1).
    float v4[4];
    {
        const bool b = (lane >> 4) & 1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float give = b ? gxa[q] : gya[q];
            const float keep = b ? gya[q] : gxa[q];
            v4[q] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
        }
    }
    float v2[2];
    {
        const bool b = (lane >> 3) & 1;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float give = b ? v4[q] : v4[q + 2];
            const float keep = b ? v4[q + 2] : v4[q];
            v2[q] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
        }
    }
    float v1;
    {
        const bool b = (lane >> 2) & 1;
        const float give = b ? v2[0] : v2[1];
        const float keep = b ? v2[1] : v2[0];
        v1 = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    }
    v1 += __shfl_xor_sync(0xffffffffu, v1, 2);
    v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
    // lane a < 4 takes gx_a (k = a) and gy_a (k = 4 + a)
    const int la = lane & 3;
    const float gxs = __shfl_sync(0xffffffffu, v1, 8 * ((la >> 1) & 1) + 4 * (la & 1));
    const float gys = __shfl_sync(0xffffffffu, v1, 16 + 8 * ((la >> 1) & 1) + 4 * (la & 1));
    // Lane a stores node a's partial in the chunk's slot of that node as one tagged record; the slots
    // of nodes 0 and 1 also carry the two words of the chunk's sum of r^2, so every chunk is counted
    // exactly once.
    int rec = __shfl_sync(0xffffffffu, w.rec[0], src);
#pragma unroll
    for (int a = 1; a < 4; ++a) {
        const int t = __shfl_sync(0xffffffffu, w.rec[a], src);
        if (lane == a) rec = t;
    }
    const unsigned tag = __shfl_sync(0xffffffffu, w.tag, src);
    if (lane < 4)
        st_record(reinterpret_cast<float4 *>(F.node_grad) + rec,
                  make_uint4(__float_as_uint(gxs), __float_as_uint(gys),
                             __float_as_uint(lane == 0 ? js.hi : (lane == 1 ? js.lo : 0.f)),
                             (tag << 4) | ((flags >> (4 + 4 * lane)) & 15u)));
    __syncwarp();                                   // every lane is done with the staged buffers
}

// ---------------------------------------------------------------------------
// N work: one group of GN = 32 nodes per warp (lane = node)
// ---------------------------------------------------------------------------
// Per node, in two parts.  node_pre needs nothing from this round's pixel pass (the
// candidate point, the trial direction, the current gradient and the spring terms), so a
// warp runs it before it waits for its group's chunks; node_post gathers the chunk
// partials from the node's K slots (slot order), writes the trial gradient, point and
// direction, and returns the node's terms of sum r^2, spring energy, g.g, g.(g - g_cur)
// and g_cur.dir in double-float.
struct NodePre {
    float2 ui, dir, gc;
    float rx, ry, en;
};

__device__ __forceinline__ NodePre node_pre(const d2ic_frame_t &F, const FInfo &fi, int n) {
    NodePre p;
    p.rx = p.ry = p.en = 0.f;
    p.ui = p.dir = p.gc = make_float2(0.f, 0.f);
    if (n >= F.n_nodes) return p;
    const Cand cd = make_cand(F, fi);
    // All loads of a batch are issued before any is consumed: a short chain of L2 round
    // trips instead of one per table entry.  Sums still run in table order.
    p.gc = __ldcg(nbuf(F, 2 + fi.igc) + n);
    p.ui = cd.at(n, p.dir);
    const int md = F.max_deg, Nn = F.n_nodes;
    const int *nbi = F.nbr_index + n;             // column-major: entry k at k * n_nodes
    const float *nbw = F.nbr_weight + n;
    bool alive = true;                               // entries after the first -1 are padding
    constexpr int NBN = 8;
    for (int kb = 0; kb < md && alive; kb += NBN) {
        int jj[NBN];
        float ww[NBN];
#pragma unroll
        for (int t = 0; t < NBN; ++t) {
            jj[t] = (kb + t < md) ? __ldg(nbi + (size_t)(kb + t) * Nn) : -1;
            ww[t] = (kb + t < md) ? __ldg(nbw + (size_t)(kb + t) * Nn) : 0.f;
        }
        float2 uj[NBN];
#pragma unroll
        for (int t = 0; t < NBN; ++t) {
            float2 dj;
            uj[t] = (jj[t] >= 0) ? cd.at(jj[t], dj) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int t = 0; t < NBN; ++t) {
            alive = alive && jj[t] >= 0;
            if (alive) {
                const float ddx = p.ui.x - uj[t].x, ddy = p.ui.y - uj[t].y;
                p.rx += ww[t] * ddx;
                p.ry += ww[t] * ddy;
                p.en += ww[t] * (ddx * ddx + ddy * ddy);
            }
        }
    }
    return p;
}

// A node's sums over its K slots (slot order).
struct SlotSums {
    float x, y;
    DF j;
};

// A bounded wait's periodic check (whole warp): false once the launch is aborted, or aborts it when
// more than WAIT_NS have passed since the first check (t0, 0 before it).
__device__ __forceinline__ bool keep_waiting(CtlHeader *H, unsigned long long &t0, int lane) {
    int go = 1;
    if (lane == 0) {
        const unsigned long long now = gtimer();
        if (t0 == 0) t0 = now;
        if (ld_vol(&H->abort)) {
            go = 0;
        } else if (now - t0 > WAIT_NS) {
            H->err = D2IC_WAIT_TIMEOUT;
            atomicExch(&H->abort, 1);
            go = 0;
        }
    }
    return __shfl_sync(0xffffffffu, go, 0) != 0;
}

// Gathers the slots of a group's nodes (lane = node n) once every chunk that touches the group has
// written this evaluation's records (whole warp; false after an abort or WAIT_NS).  The slots
// themselves are polled: a slot that no chunk owns never carries the tag, so the group is complete
// when `need` (chunks touching the group) first-node records have arrived and the records they
// announce -- their chunks' nodes in this group -- are as many as the records that arrived.
__device__ __forceinline__ bool gather_slots(const d2ic_frame_t &F, int n, int need, unsigned tag, CtlHeader *H,
                                             SlotSums &s) {
    const int K = F.node_chunk_k, Nn = F.n_nodes;
    const float4 *ng = reinterpret_cast<const float4 *>(F.node_grad) + n;
    constexpr int NB = 4;                              // K of elements that are one chunk each
    const int lane = threadIdx.x & 31;
    unsigned long long t0 = 0;
    auto add = [&](const uint4 &v) {                   // absent records add zeros
        s.x += __uint_as_float(v.x);
        s.y += __uint_as_float(v.y);
        s.j = df_add(s.j, DF{__uint_as_float(v.z), 0.f});
    };
    for (unsigned it = 0;; ++it) {
        int acc = 0;                                   // arrived - announced in the low half, firsts above
        uint4 v[NB];
        s.x = s.y = 0.f;
        s.j = DF{0.f, 0.f};
        for (int kb = 0; kb < K; kb += NB) {
#pragma unroll
            for (int t = 0; t < NB; ++t)
                v[t] = n < Nn && kb + t < K ? ld_record(ng + (size_t)(kb + t) * Nn) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int t = 0; t < NB; ++t) {
                const int x = (v[t].w & 1u) ? 0x10001 - (int)((v[t].w >> 1) & 7u) : 1;
                acc += (v[t].w >> 4) == tag ? x : 0;
            }
            if (K > NB)                                // summed along the way; else once, when complete
#pragma unroll
                for (int t = 0; t < NB; ++t) add(v[t]);
        }
        const int sum = __reduce_add_sync(0xffffffffu, acc);
        const int open = (int)(short)(sum & 0xffff), firsts = (sum - open) >> 16;
        if (open == 0 && firsts >= need) {
            if (K <= NB)
#pragma unroll
                for (int t = 0; t < NB; ++t) add(v[t]);
            return true;
        }
        if ((it & 63) == 63 && !keep_waiting(H, t0, lane)) return false;
    }
}

__device__ __forceinline__ void node_post(const d2ic_frame_t &F, const FInfo &fi, int n, const NodePre &p,
                                          const SlotSums &s, DF q[5]) {
#pragma unroll
    for (int i = 0; i < 5; ++i) q[i] = DF{0.f, 0.f};
    if (n >= F.n_nodes) return;
    const float sx = s.x, sy = s.y;
    const DF sj = s.j;
    const float inv_np = 1.0f / (float)max(F.n_pix, 1);
    const float gx = sx * inv_np + F.alpha_reg * p.rx;
    const float gy = sy * inv_np + F.alpha_reg * p.ry;
    nbuf(F, 2 + fi.igt)[n] = make_float2(gx, gy);
    nbuf(F, 1 - fi.iu)[n] = p.ui;
    nbuf(F, 5 + (1 - fi.idp))[n] = p.dir;
    // per-node terms of the inner products, exact in double-float (g - g_cur rounded
    // in FP32 as the reference's elementwise difference)
    q[P_JSUM] = sj;
    q[P_EREG] = DF{0.25f * p.en, 0.f};
    q[P_GG] = df_add(df_prod(gx, gx), df_prod(gy, gy));
    q[P_GDIFF] = df_add(df_prod(gx, gx - p.gc.x), df_prod(gy, gy - p.gc.y));
    q[P_GD] = df_add(df_prod(p.gc.x, p.dir.x), df_prod(p.gc.y, p.dir.y));
}

// ---------------------------------------------------------------------------
// Control step (one warp per frame and round)
// ---------------------------------------------------------------------------
// The descriptor scalars the control step reads, loaded once at its start.
struct FConst {
    float *hist;
    double tol, tol2_hi;   // tol2_hi: squares at or above it are certainly not below tol
    int max_iter;
};

// Values of a control step, computed for the whole warp at once (GB300's FP64 pipe is narrow, so
// each FP64 instruction is costly): the objective J of this round's point, the squared gradient norm
// of the state after accepting this point and the PR+ ratio g.(g - g_prev) / (g_prev.g_prev + 1e-16).
struct StepVals {
    double J, gg, ratio, armijo;   // armijo: 1e-4 alpha
};

// Tests on the bits of a double (an FP64 comparison costs tens of cycles on GB300).
__device__ __forceinline__ bool is_nan64(double x) {
    return ((unsigned long long)__double_as_longlong(x) << 1) > 0xffe0000000000000ull;
}
__device__ __forceinline__ bool is_neg64(double x) {   // x < 0 (not for -0 or NaN)
    const long long b = __double_as_longlong(x);
    return b < 0 && (b << 1) != 0 && !is_nan64(x);
}
__device__ __forceinline__ bool is_nonneg64(double x) {   // x >= 0 (also -0, not NaN)
    const long long b = __double_as_longlong(x);
    return (b >= 0 || (b << 1) == 0) && !is_nan64(x);
}

__device__ __forceinline__ void hist_row(const FConst &F, int k, double a, double b, double c) {
    if (F.hist && k < F.max_iter) {
        F.hist[3 * k + 0] = (float)a;
        F.hist[3 * k + 1] = (float)b;
        F.hist[3 * k + 2] = (float)c;
    }
}

__device__ __forceinline__ void accept_point(FrameState &S, double J, double gg, double gdiff) {
    S.J_cur = J;
    S.gg_prev = S.gg_cur;
    S.gg_cur = gg;
    S.gdiff_cur = gdiff;
    const int gp = S.igp;
    S.igp = S.igc;
    S.igc = S.igt;
    S.igt = gp;
    S.iu = 1 - S.iu;
    S.idp = 1 - S.idp;
}

// Called right after accept_point of this round's point, so v.gg = S.gg_cur and
// v.ratio = S.gdiff_cur / (S.gg_prev + 1e-16).  The norm sqrt(g.g) itself is needed only for the stop
// test and, later, the history: far above the tolerance the test is decided on the squares, and the
// square root is taken after the release (S.gnorm < 0 marks it as open).
__device__ __forceinline__ void start_iter(FrameState &S, const FConst &F, const StepVals &v) {
    S.gnorm = -1.0;
    if (!(v.gg >= F.tol2_hi)) {
        S.gnorm = sqrt(v.gg);
        if (S.gnorm < F.tol) {                   // stop branch: k unchanged
            hist_row(F, S.k, S.J_cur, S.gnorm, 0.0);
            S.state = ST_DONE;
            return;
        }
    }
    double beta = 0.0;
    if (S.k > 0) {
        beta = is_neg64(v.ratio) ? 0.0 : v.ratio;   // max(ratio, 0); jnp.maximum keeps NaN
    }
    S.beta = (float)beta;
    S.alpha = 1.0f;
    S.t = 0;
    S.restart = 0;
    S.gd_known = 0;
    S.state = ST_TRIAL;
}

__device__ __forceinline__ void frame_decide(FrameState &S, const FConst &F, const double *q, const StepVals &v, int eval_only) {
    const double J = v.J;
    if (is_nan64(J) || is_nan64(q[P_GG])) S.nan_seen = 1;
    S.n_evals += 1;
    // control-flow guard: an iteration takes at most 11 evaluations plus one restart
    if (S.n_evals > 12 * max(F.max_iter, 0) + 4) {
        S.state = ST_DONE;
        return;
    }
    switch (S.state) {
        case ST_EVAL:
            accept_point(S, J, q[P_GG], q[P_GDIFF]);
            if (eval_only || F.max_iter <= 0) {
                S.state = ST_DONE;
                return;
            }
            start_iter(S, F, v);
            return;
        case ST_TRIAL: {
            if (!S.gd_known) {
                S.gd_known = 1;
                S.gd = q[P_GD];
                if (is_nonneg64(S.gd)) {           // not a descent direction: restart with -g
                    S.restart = 1;
                    S.gd = -S.gg_cur;
                    S.alpha = 1.0f;
                    return;                        // re-evaluate trial 0 along -g
                }
            }
            if (J <= S.J_cur + v.armijo * S.gd) {
                hist_row(F, S.k, J, S.gnorm, (double)S.alpha);
                S.k += 1;
                accept_point(S, J, q[P_GG], q[P_GDIFF]);
                if (S.k >= F.max_iter) S.state = ST_DONE;
                else start_iter(S, F, v);
            } else {
                S.J_last = J;
                S.t += 1;
                S.alpha *= 0.5f;
                if (S.t >= 10) S.state = ST_FORCED;   // alpha == 2^-10 is applied anyway
            }
            return;
        }
        case ST_FORCED:
            hist_row(F, S.k, S.J_last, S.gnorm, (double)S.alpha);
            S.k += 1;
            accept_point(S, J, q[P_GG], q[P_GDIFF]);
            if (S.k >= F.max_iter) S.state = ST_DONE;
            else start_iter(S, F, v);
            return;
        default:
            return;
    }
}

// exclusive block-wide scan of three counters (warp shuffles + one shared pass)
__device__ __forceinline__ void block_scan3(int &a, int &b, int &c, int &ta, int &tb, int &tc) {
    __shared__ int s_w[NWARP][3];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int ia = a, ib = b, ic = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int xa = __shfl_up_sync(0xffffffffu, ia, o), xb = __shfl_up_sync(0xffffffffu, ib, o),
                  xc = __shfl_up_sync(0xffffffffu, ic, o);
        if (lane >= o) { ia += xa; ib += xb; ic += xc; }
    }
    if (lane == 31) { s_w[wid][0] = ia; s_w[wid][1] = ib; s_w[wid][2] = ic; }
    __syncthreads();
    int oa = 0, ob = 0, oc = 0;
    ta = tb = tc = 0;
    for (int w = 0; w < NWARP; ++w) {
        if (w == wid) { oa = ta; ob = tb; oc = tc; }
        ta += s_w[w][0]; tb += s_w[w][1]; tc += s_w[w][2];
    }
    a = oa + ia - a;
    b = ob + ib - b;
    c = oc + ic - c;
    __syncthreads();
}

// A frame takes part in this launch's rounds: not finished and not held (CMD_HOLD keeps an admitted
// frame's state but leaves it out of the launch).  The command words are constant once r_init ran.
__device__ __forceinline__ bool in_launch(Ctl &C, int f) {
    return ld_vol(&C.fs[f].state) != ST_DONE && ld_vol(C.cmd + f) != CMD_HOLD;
}

// rebuild the active list and prefix sums (whole block)
__device__ void rebuild_active(const d2ic_frame_t *frames, int n_frames, Ctl &C) {
    const int per = (n_frames + NT - 1) / NT;
    const int f0 = threadIdx.x * per, f1 = min(f0 + per, n_frames);
    int cnt = 0, ch = 0, gr = 0;
    for (int f = f0; f < f1; ++f)
        if (in_launch(C, f)) {
            ++cnt;
            ch += frames[f].n_chunks;
            gr += pad_groups(frames[f].n_groups);
        }
    int ta, tb, tc;
    block_scan3(cnt, ch, gr, ta, tb, tc);
    const int lb = ld_vol(&C.h->list_buf);         // start of a launch: nothing reads the list yet
    if (threadIdx.x == 0) {
        C.h->n_active = ta;
        C.h->total_chunks = tb;
        C.h->total_groups = tc;
        C.cp(lb)[ta] = tb;
        C.gp(lb)[ta] = tc;
    }
    int slot = cnt, cp = ch, gp = gr;
    for (int f = f0; f < f1; ++f)
        if (in_launch(C, f)) {
            C.act(lb)[slot] = f;
            C.cp(lb)[slot] = cp;
            C.gp(lb)[slot] = gp;
            ++slot;
            cp += frames[f].n_chunks;
            gp += pad_groups(frames[f].n_groups);
        }
    __syncthreads();
}

// Start of a launch: new frames (CMD_INIT) get a fresh CG state, idle slots are
// parked as finished-and-reported, running and held frames keep their state (held
// ones stay out of the active list); frames that finished in an earlier launch are
// marked reported (their outputs were written at the end of that launch).
__device__ void r_init(const d2ic_frame_t *frames, int n_frames, Ctl &C) {
    for (int f = threadIdx.x; f < n_frames; f += NT) {
        C.rule[f] = make_uint4(0u, 0u, 0u, 0u);
        const int cmd = ld_vol(C.cmd + f);
        if (cmd == CMD_INIT) {
            FrameState S;
            S.J_cur = S.gg_cur = S.gg_prev = S.gdiff_cur = S.gd = S.J_last = S.gnorm = 0.0;
            S.alpha = 0.f;
            S.beta = 0.f;
            S.k = S.t = S.restart = S.gd_known = S.nan_seen = S.n_evals = 0;
            S.iu = 0; S.igp = 0; S.igc = 1; S.igt = 2; S.idp = 0;
            S.state = ST_EVAL;
            S.reported = 0;
            S.pad2_ = 0;
            C.fs[f] = S;
            C.cmd[f] = CMD_RUN;
        } else if (cmd == CMD_IDLE) {
            C.fs[f].state = ST_DONE;
            C.fs[f].reported = 1;
        } else if (ld_vol(&C.fs[f].state) == ST_DONE) {
            C.fs[f].reported = 1;
        }
        C.tag0()[f] = cmd == CMD_INIT ? 1u : ((unsigned)ld_vol(&C.fs[f].n_evals) + 1u) & TAG_MASK;
    }
    __syncthreads();
    rebuild_active(frames, n_frames, C);
}

// Wait (bounded) until blocks_past reaches target; on a timeout the launch aborts and the list
// is left as it is.
__device__ __forceinline__ int wait_blocks_past(CtlHeader *H, unsigned target) {
    if (ld_acquire_u32(&H->blocks_past) >= target) return 1;
    const unsigned long long t0 = gtimer();
    while (ld_acquire_u32(&H->blocks_past) < target) {
        if (ld_vol(&H->abort)) return 0;
        if (gtimer() - t0 > WAIT_NS) {
            H->err = D2IC_WAIT_TIMEOUT;
            atomicExch(&H->abort, 1);
            return 0;
        }
        __nanosleep(32);
    }
    return 1;
}

// Active list rebuilt by one warp (the warp that ends a round): lane l scans a contiguous
// block of frames, a warp scan gives each block its slot and prefix offsets.
__device__ __forceinline__ void rebuild_active_warp(const d2ic_frame_t *frames, int n_frames, Ctl &C, int lane) {
    const int per = (n_frames + 31) / 32;
    const int f0 = min(lane * per, n_frames), f1 = min(f0 + per, n_frames);
    int cnt = 0, ch = 0, gr = 0;
    for (int f = f0; f < f1; ++f)
        if (in_launch(C, f)) {
            ++cnt;
            ch += frames[f].n_chunks;
            gr += pad_groups(frames[f].n_groups);
        }
    int ic = cnt, ih = ch, ig = gr;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, ic, o), b = __shfl_up_sync(0xffffffffu, ih, o),
                  c = __shfl_up_sync(0xffffffffu, ig, o);
        if (lane >= o) {
            ic += a;
            ih += b;
            ig += c;
        }
    }
    const int ta = __shfl_sync(0xffffffffu, ic, 31), tb = __shfl_sync(0xffffffffu, ih, 31),
              tc = __shfl_sync(0xffffffffu, ig, 31);
    // the copy no block reads (see Ctl); read once, before lane 0 flips it below
    const int nb = 1 - __shfl_sync(0xffffffffu, lane == 0 ? ld_vol(&C.h->list_buf) : 0, 0);
    int slot = ic - cnt, cp = ih - ch, gp = ig - gr;
    for (int f = f0; f < f1; ++f)
        if (in_launch(C, f)) {
            C.act(nb)[slot] = f;
            C.cp(nb)[slot] = cp;
            C.gp(nb)[slot] = gp;
            ++slot;
            cp += frames[f].n_chunks;
            gp += pad_groups(frames[f].n_groups);
        }
    if (lane == 0) {
        C.h->n_active = ta;
        C.h->total_chunks = tb;
        C.h->total_groups = tc;
        C.cp(nb)[ta] = tb;
        C.gp(nb)[ta] = tc;
        C.h->list_buf = nb;                          // published by the round's release
    }
    __syncwarp();
}

// Supergroup records of a frame, behind its group partials: one tagged 16-byte record per sum.
constexpr int SG_RECORDS = D2IC_NPART;
__host__ __device__ inline size_t sg_record_offset(int n_groups) {
    return ((size_t)n_groups * D2IC_NPART * sizeof(float2) + 15) & ~(size_t)15;
}
__device__ __forceinline__ uint4 *sg_records(const d2ic_frame_t &F) {
    return reinterpret_cast<uint4 *>(reinterpret_cast<char *>(F.group_part) + sg_record_offset(F.n_groups));
}

// The control step of one frame: waits (bounded) for the frame's supergroup records of this
// evaluation, reduces them (lane-strided, then a warp sum) and advances the CG state, which lane 0
// returns in S (shared memory of the block with SHARED, else registers); false after an abort.  Everything that does not need the sums -- the state, one word per
// lane, and the reciprocals of the two divisions -- is read and computed before the wait, and the
// square root is left for after the release, so that the path from the last supergroup to the
// release holds about ten FP64 operations.
template <bool SHARED>
__device__ __forceinline__ bool frame_r(const d2ic_frame_t &F, int f, Ctl &C, int eval_only, int lane, unsigned tag,
                                        FrameState &S) {
    constexpr int WORDS = sizeof(FrameState) / 8;
    constexpr int L_HIST = WORDS, L_TOL = WORDS + 1, L_PAR = WORDS + 2;   // lanes of the descriptor's words
    static_assert(L_PAR < 32, "one word of the state or the descriptor per lane");
    static_assert(offsetof(d2ic_frame_t, alpha_reg) % 8 == 0 &&
                      offsetof(d2ic_frame_t, max_iter) == offsetof(d2ic_frame_t, alpha_reg) + 4,
                  "alpha_reg and max_iter are one word");
    DF q[5] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(C.fs + f) + lane;
    if (lane == L_HIST) src = reinterpret_cast<const unsigned long long *>(&F.hist);
    if (lane == L_TOL) src = reinterpret_cast<const unsigned long long *>(&F.tol);
    if (lane == L_PAR) src = reinterpret_cast<const unsigned long long *>(&F.alpha_reg);
    unsigned long long word = 0;
    if (lane < WORDS) word = __ldcg(src);
    else if (lane <= L_PAR) word = *src;
    // lane 0: 0.5 / n_pix; lane 1: 1 / (g.g + 1e-16); lane 2: squares at or above it are certainly not below
    // tol; lane 3: the Armijo factor
    const double gg_old = __longlong_as_double(
        (long long)__shfl_sync(0xffffffffu, word, (int)(offsetof(FrameState, gg_cur) / 8)));
    const double tol = __longlong_as_double((long long)__shfl_sync(0xffffffffu, word, L_TOL));
    double inv = (lane == 0 ? 0.5 : 1.0) / (lane == 0 ? (double)max(F.n_pix, 1) : gg_old + 1e-16);
    const float alpha_old = __uint_as_float((unsigned)(__shfl_sync(0xffffffffu, word, (int)(offsetof(FrameState, alpha) / 8)) >>
                                                       (8 * (offsetof(FrameState, alpha) % 8))));
    if (lane == 3) inv = 1e-4 * (double)alpha_old;
    if (lane == 2) inv = tol > 0.0 ? fmax(tol * tol * (1.0 + 1e-12), 1e-290) : 0.0;
    const int nsg = (F.n_groups + SG - 1) / SG;
    const uint4 *rec = sg_records(F);
    // Every branch of the wait is taken by the whole warp: lanes that left a polling loop one by one
    // stayed split after it, and the sums below then ran lane by lane (6 us instead of 0.3 us).
    // Batches of 32 supergroups, D in flight, added in the same order (above 32 supergroups two in flight: 1.4 % of a
    // round at 2048 x 2048 and 4096 x 4096; four spill).
    auto gather = [&](auto depth) {
        constexpr int D = decltype(depth)::value;
        for (int g0 = 0; g0 < nsg; g0 += 32 * D) {
            uint4 r[D][SG_RECORDS];
            unsigned long long t0 = 0;
            for (unsigned it = 0;; ++it) {
                bool all = true;
#pragma unroll
                for (int d = 0; d < D; ++d)
#pragma unroll
                    for (int k = 0; k < SG_RECORDS; ++k) {
                        const int g = g0 + 32 * d + lane;
                        r[d][k] = g < nsg ? ld_record(rec + (size_t)g * SG_RECORDS + k) : make_uint4(0u, 0u, tag, 0u);
                    }
#pragma unroll
                for (int d = 0; d < D; ++d)
#pragma unroll
                    for (int k = 0; k < SG_RECORDS; ++k) all = all && r[d][k].z == tag;
                if (__all_sync(0xffffffffu, all)) break;
                if ((it & 63) == 63 && !keep_waiting(C.h, t0, lane)) return false;
            }
#pragma unroll
            for (int d = 0; d < D; ++d)
#pragma unroll
                for (int k = 0; k < SG_RECORDS; ++k)
                    q[k] = df_add(q[k], DF{__uint_as_float(r[d][k].x), __uint_as_float(r[d][k].y)});
        }
        return true;
    };
    if (!(nsg <= 32 ? gather(std::integral_constant<int, 1>{}) : gather(std::integral_constant<int, 2>{}))) return false;
    fence_acq_rel();                                   // the groups' node data before this frame's release
    // the lanes that hold a sum convert it to FP64: one conversion for all five
    const double mine = df_to_double(df_reduce5(q, lane));
    double qd[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) qd[i] = __shfl_sync(0xffffffffu, mine, red5_lane(i));
    StepVals v;
    v.gg = qd[P_GG];
    v.ratio = qd[P_GDIFF] * __shfl_sync(0xffffffffu, inv, 1);
    v.armijo = __shfl_sync(0xffffffffu, inv, 3);
    const unsigned long long par = __shfl_sync(0xffffffffu, word, L_PAR);
    v.J = qd[P_JSUM] * __shfl_sync(0xffffffffu, inv, 0) + (double)__uint_as_float((unsigned)par) * qd[P_EREG];
    FConst fc;
    fc.hist = reinterpret_cast<float *>(__shfl_sync(0xffffffffu, word, L_HIST));
    fc.tol = __longlong_as_double((long long)__shfl_sync(0xffffffffu, word, L_TOL));
    fc.tol2_hi = __shfl_sync(0xffffffffu, inv, 2);
    fc.max_iter = (int)(par >> 32);
    unsigned long long *sw = reinterpret_cast<unsigned long long *>(&S);
    if (SHARED) {
        if (lane < WORDS) sw[lane] = word;
        __syncwarp();
    } else {
#pragma unroll
        for (int i = 0; i < WORDS; ++i) sw[i] = __shfl_sync(0xffffffffu, word, i);
    }
    if (lane == 0) frame_decide(S, fc, qd, v, eval_only);
    __syncwarp();
    return true;
}

// The rest of a control step (whole warp): the gradient norm if it is still open, and the state.
template <bool SHARED>
__device__ __forceinline__ void frame_store(FrameState &S, FrameState *dst, int lane) {
    if (lane == 0 && S.gnorm < 0.0) S.gnorm = sqrt(S.gg_cur);
    if (SHARED) {
        __syncwarp();
        if (lane < (int)(sizeof(FrameState) / 8))
            reinterpret_cast<unsigned long long *>(dst)[lane] = reinterpret_cast<const unsigned long long *>(&S)[lane];
        __syncwarp();
    } else if (lane == 0) {
        *dst = S;
    }
}

// The candidate rule that follows from a state (as frame_info reads it back).
__device__ __forceinline__ FInfo info_of(const FrameState &S) {
    FInfo fi;
    fi.iu = S.iu;
    fi.igc = S.igc;
    fi.idp = S.idp;
    fi.igt = S.igt;
    fi.alpha = S.alpha;
    fi.beta = S.beta;
    fi.mode = (S.state == ST_EVAL) ? 0 : ((S.restart || S.k == 0) ? 2 : 1);
    fi.tag = 0;
    return fi;
}

// The round's frames have all run their control step and one has finished: the active list is rebuilt
// (whole warp).  Returns the release word.
__device__ __forceinline__ unsigned rebuild_for_release(const d2ic_frame_t *frames, int n_frames, Ctl &C, int round,
                                                        int list_version, int stop_flags, int lane) {
    // no block still reads the list copy of an earlier round (bounded)
    int past = 1;
    if (lane == 0) past = wait_blocks_past(C.h, gridDim.x * (unsigned)round);
    if (__shfl_sync(0xffffffffu, past, 0)) rebuild_active_warp(frames, n_frames, C, lane);
    return ((unsigned)((list_version + 1) & 0xffff) << 16) | ((stop_flags & STOP_ON_FINISH) ? REL_STOP : 0u);
}

// Control step of frame f (one warp), and the round's release if it is the round's last frame.
// direct: f is in slot `slot` of the na active frames `act`.
template <bool SHARED>
__device__ __forceinline__ void control_step(const d2ic_frame_t *frames, const d2ic_frame_t &F, int n_frames, Ctl &C, int f, unsigned tag,
                                             int na, bool blockred, bool direct, int slot, const int *act, int round,
                                             int list_version, int eval_only, int stop_flags, unsigned long long *trace,
                                             int trace_rounds, int lane, FrameState &S) {
    const bool rt = trace != nullptr && lane == 0 && round < trace_rounds;
    const int irq = direct && slot == 0 && (stop_flags & STOP_ON_IRQ) ? ld_vol(&C.h->irq) : 0;
    if (!frame_r<SHARED>(F, f, C, eval_only, lane, tag, S)) return;
    if (rt) trace[7 * round + 3] = gtimer();
    // With one active frame whose control stays on this warp the release carries the next candidate
    // rule, and the state is stored after it.  (A finished frame's state is read by every block after
    // the release, so it is stored before.)
    const bool done = SHARED ? S.state == ST_DONE : __shfl_sync(0xffffffffu, lane == 0 ? (S.state == ST_DONE) : 0, 0);
    if (!SHARED && direct) {
        if (done) frame_store<SHARED>(S, C.fs + f, lane);
        if (lane == 0) {
            const FInfo nx = info_of(S);
            if (done) fence_acq_rel();
            st_record(C.rule + f, make_uint4((unsigned)(round + 1), rel_pack(nx) | (done ? REL_FIN : 0u) | (irq ? REL_STOP : 0u),
                                             __float_as_uint(nx.alpha), __float_as_uint(nx.beta)));
        }
        if (rt) trace[7 * round + 4] = gtimer();
        if (!done) {
            frame_store<SHARED>(S, C.fs + f, lane);
            return;
        }
        // the first of the frames that finished in this round waits for the others' records and rebuilds the list
        const uint4 *mine = C.rule + (lane < na ? act[lane] : f);
        uint4 r;
        unsigned long long t0 = 0;
        for (unsigned it = 0;; ++it) {
            r = ld_record(mine);
            if (__all_sync(0xffffffffu, r.x > (unsigned)round)) break;
            if ((it & 63) == 63 && !keep_waiting(C.h, t0, lane)) return;
        }
        fence_acq_rel();
        const unsigned fin = __ballot_sync(0xffffffffu, lane < na && r.x == (unsigned)(round + 1) && (r.y & REL_FIN));
        if (__ffs((int)fin) - 1 != slot) return;
        const unsigned rel = rebuild_for_release(frames, n_frames, C, round, list_version, stop_flags, lane);
        if (lane == 0) {
            fence_acq_rel();
            st_record(&C.h->rel, make_uint4((unsigned)(round + 1), rel, 0u, 0u));
        }
        return;
    }
    const bool inlined = na == 1 && blockred && !done;
    int last_frame = 1;
    if (!inlined) frame_store<SHARED>(S, C.fs + f, lane);
    if (lane == 0 && !inlined) {
        if (done) atomicExch(&C.h->finished, 1);
        __threadfence();
        if (na > 1) last_frame = atom_acq_rel_add(&C.h->frames_done, 1) == na - 1;
    }
    __syncwarp();
    if (__shfl_sync(0xffffffffu, last_frame, 0)) {
        // every frame of the round has run its control step, so every block's work of the round is
        // done: rebuild the active list if a frame finished, and release the round
        unsigned rel = (unsigned)list_version << 16;
        if (!inlined) {
            if (lane == 0 && na > 1) C.h->frames_done = 0;
            if (ld_vol(&C.h->finished)) {
                rel = rebuild_for_release(frames, n_frames, C, round, list_version, stop_flags, lane);
                if (lane == 0) C.h->finished = 0;
            }
        }
        if (lane == 0) {
            if ((stop_flags & STOP_ON_IRQ) && ld_vol(&C.h->irq)) rel |= REL_STOP;
            uint4 r = make_uint4((unsigned)(round + 1), rel, 0u, 0u);
            if (inlined) {
                const FInfo nx = info_of(S);
                r.y |= rel_pack(nx);
                r.z = __float_as_uint(nx.alpha);
                r.w = __float_as_uint(nx.beta);
            } else {
                fence_acq_rel();
            }
            st_record(&C.h->rel, r);
        }
    }
    if (rt) trace[7 * round + 4] = gtimer();
    if (inlined) frame_store<SHARED>(S, C.fs + f, lane);
}

// The active list (n_active = na <= FCACHE) with its prefix sums and each frame's candidate
// rule after `rounds` completed rounds, copied into the block's shared memory (whole block).
template <bool STATE_TAG>
__device__ __forceinline__ void load_list(Ctl &C, int lb, int na, int rounds, int *s_cpre, int *s_gpre, int *s_act,
                                          FRule *s_fi) {
    if (na > FCACHE) return;
    for (int s = threadIdx.x; s <= na; s += NT) {
        s_cpre[s] = __ldcg(C.cp(lb) + s);
        s_gpre[s] = __ldcg(C.gp(lb) + s);
    }
    for (int s = threadIdx.x; s < na; s += NT) {
        const int f = checked_index(__ldcg(C.act(lb) + s), C.n, C.h);
        s_act[s] = f;
        s_fi[s] = make_rule(frame_info<STATE_TAG>(C, f, rounds));
    }
}

// The chunk range of warp wid when one frame is active.  Every block takes a contiguous share of the
// chunks (neighbouring elements share coefficient rows in cache), split evenly over its warps, so that
// no SM has more chunks than the others (shares dealt out warp by warp left 49 of 152 SMs with all of
// a 512 x 512 frame, and 80 against 64 chunks per SM at 2048 x 2048).  Blocks whose warps reduce node
// groups (group gi: warp gi), and the last block, which runs the control step, take LEAD_PIXELS pixels
// less than the others: a block's pixel work of about 2.5 us, the time of the node work that comes
// before the wait for a group's chunks.  (Without it an evaluation at 512 x 512 takes 12.2 instead of 10.2 us, at
// 1024 x 1024 15.6 instead of 14.0, at 2048 x 2048 28.3 instead of 27.0; half of it: 11.6, 14.2 and 27.6.)
constexpr int LEAD_PIXELS = 2304;
__device__ __forceinline__ int2 chunk_share(const d2ic_frame_t &F, int total, int tg, int wid) {
    const int nb = (int)gridDim.x, b = (int)blockIdx.x, rb = (tg + NWARP - 1) / NWARP, full = nb - rb - 1;
    int b0, n;
    if (full > 0) {
        const int lead = (int)((long long)LEAD_PIXELS * total / max(F.n_pix, 1));   // in chunks
        const int light = (int)max(((long long)total - (long long)lead * full) / nb, 0ll);
        const int rest = total - (rb + 1) * light;
        if (b < rb) {
            b0 = b * light;
            n = light;
        } else if (b == nb - 1) {
            b0 = total - light;
            n = light;
        } else {
            b0 = rb * light + (int)((long long)rest * (b - rb) / full);
            n = rb * light + (int)((long long)rest * (b - rb + 1) / full) - b0;
        }
    } else {
        b0 = (int)((long long)total * b / nb);
        n = (int)((long long)total * (b + 1) / nb) - b0;
    }
    const int base = n / NWARP, extra = n - base * NWARP;   // spare chunks to the last warps
    const int c0 = b0 + wid * base + max(wid - (NWARP - extra), 0);
    return make_int2(c0, c0 + base + (wid >= NWARP - extra ? 1 : 0));
}

// ---------------------------------------------------------------------------
// the persistent kernel
// ---------------------------------------------------------------------------
// ONE: a launch of exactly one frame; the pixel pass then reads that frame's descriptor at a
// fixed address, so its fields are loop invariants (loaded once, not per chunk; measured 2-5%
// faster per round).
constexpr int FRAME_BEGIN = (int)offsetof(d2ic_frame_t, coeff), FRAME_END = (int)offsetof(d2ic_frame_t, reserved_);
static_assert(FRAME_BEGIN % 8 == 0 && FRAME_END % 8 == 0, "the kept part of a descriptor is whole words");

template <int KIND, bool ONE = false>
__global__ void __launch_bounds__(NT, D2IC_ENGINE_MINB) cg_engine(const d2ic_frame_t *__restrict__ frames, int n_frames_arg,
                                                   char *ctl_base, int eval_only, const float *u_eval,
                                                   double *J_out, float *grad_out, unsigned long long *trace,
                                                   int trace_rounds, int max_rounds, int stop_flags) {
    __shared__ unsigned long long s_bar[NWARP][2];   // per-warp mbarriers of the two record buffers
    const int n_frames = ONE ? 1 : n_frames_arg;     // ONE: the control block's offsets are constants
    constexpr int FC = ONE ? 1 : FCACHE;
    __shared__ int s_cpre[FC + 1];                   // per-round copies of the active list (na <= FCACHE)
    __shared__ int s_gpre[FC + 1];
    __shared__ int s_act[FC];
    __shared__ FRule s_fi[FC];
    // descriptors of the active frames (na <= FS) without their tensor maps and reserved words
    constexpr int FS_N = ONE ? 1 : FS, FS_WORDS = (FRAME_END - FRAME_BEGIN) / 8;
    __shared__ __align__(16) unsigned long long s_frame[FS_N * FS_WORDS];
    __shared__ unsigned s_tag0[FS_N];                // direct rounds: a frame's tag in the launch's first round
    __shared__ FrameState s_state;                   // ONE: the state in the control step (one warp of the grid)
    __shared__ int2 s_range[NWARP];                  // each warp's chunk range (one active frame)
    __shared__ int s_hdr[10];                         // n_active, total_chunks, total_groups, abort, slice stop,
                                                     // what to refresh, rounds completed, list_buf, list version
    __shared__ DF s_gq[NWARP][D2IC_NPART];           // group partials of this block's supergroup
    __shared__ int s_sgcnt;                          // groups of this block's supergroup reduced this round
    // per warp: two record buffers, then two coefficient-tile buffers (all 128-byte aligned)
    extern __shared__ __align__(128) unsigned char s_dyn[];
    Ctl C = make_ctl(ctl_base, n_frames);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char *wbuf = s_dyn + (size_t)wid * WARP_SMEM;
    unsigned pipe_i = 0;   // chunks this warp has staged: buffer i & 1, completion parity (i >> 1) & 1
    if (lane == 0) {
        mbar_init(&s_bar[wid][0], 1);            // the issuing lane's expect_tx
        mbar_init(&s_bar[wid][1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // descriptors (and their tensor maps) may have been rewritten since the previous launch
    for (int f = threadIdx.x; f < n_frames; f += NT)
        if (frames[f].tile_w > 0)
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(frames[f].coeff_map) : "memory");
    const bool tiles_ok = (smem_addr(s_dyn) & 127) == 0;   // tile buffers need 128-byte alignment
    // The block's copies of the descriptors.  Every round begins with an acquire that empties the L1,
    // so fields read from global memory cost an L2 round trip at each step of the round.
    auto keep_frames = [&](int n) {                  // the frames of s_act[0..n), n <= FS
        for (int i = threadIdx.x; i < n * FS_WORDS; i += NT)
            s_frame[i] = reinterpret_cast<const unsigned long long *>(frames + (ONE ? 0 : s_act[i / FS_WORDS]))[FRAME_BEGIN / 8 + i % FS_WORDS];
    };
    if (ONE) keep_frames(1);
    // a frame by its key: the active slot if the descriptors are kept, else its index
    bool kept = ONE;
    auto frame = [&](int key) -> const d2ic_frame_t & {
        const char *own = reinterpret_cast<const char *>(s_frame) - FRAME_BEGIN;
        if (ONE) return *reinterpret_cast<const d2ic_frame_t *>(own);
        return kept ? *reinterpret_cast<const d2ic_frame_t *>(own + key * (FS_WORDS * 8)) : frames[key];
    };
    __syncthreads();
    // optional phase trace per round: warp 0 of block 0 stamps [0] round start, [1] end of its pixel
    // work, [2] end of its group work, [5] after the barrier; the warp that runs a frame's control
    // stamps [3] and [4] around it
    const bool tr = trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0;
    int round = 0;
    if (threadIdx.x == 0) s_sgcnt = 0;
    // A warp's first batch of the next round, loaded before the round's release, with its first chunk
    // staged (neither depends on the control step); used if the active list is unchanged, else drained.
    bool pf = false;
    int pf_na = 0, pf_total = 0;
    ChunkMeta pf_m{};

    // ---- init of newly admitted frames: u <- u0, zero g/d buffers and gradient slots, NaN history ----
    for (int f = 0; f < n_frames; ++f) {
        if (ld_vol(C.cmd + f) != CMD_INIT) continue;
        const d2ic_frame_t &F = frames[f];
        const int nn = F.n_nodes;
        const float2 *u0 = reinterpret_cast<const float2 *>((eval_only && u_eval && f == 0) ? u_eval : F.u0);
        for (int i = blockIdx.x * NT + threadIdx.x; i < nn; i += gridDim.x * NT) {
            nbuf(F, 0)[i] = u0 ? u0[i] : make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 1; j < 7; ++j) nbuf(F, j)[i] = make_float2(0.f, 0.f);
        }
        // gradient slots that no chunk owns must read as 0 (and never carry a tag); counters start at 0
        float4 *ng = reinterpret_cast<float4 *>(F.node_grad);
        for (size_t i = blockIdx.x * NT + threadIdx.x; i < (size_t)F.node_chunk_k * nn; i += (size_t)gridDim.x * NT)
            ng[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int n_sg = (F.n_groups + SG - 1) / SG;
        for (int i = blockIdx.x * NT + threadIdx.x; i < n_sg + 1; i += gridDim.x * NT) F.group_cnt[i] = 0;
        uint4 *sr = sg_records(F);
        for (int i = blockIdx.x * NT + threadIdx.x; i < n_sg * SG_RECORDS; i += gridDim.x * NT)
            sr[i] = make_uint4(0u, 0u, 0u, 0u);        // tag 0: evaluations start at 1
        if (F.hist)
            for (int i = blockIdx.x * NT + threadIdx.x; i < 3 * F.max_iter; i += gridDim.x * NT)
                F.hist[i] = __int_as_float(0x7fc00000);
        // first-pass tile origins from u0 (the first pass evaluates u0 itself)
        if (F.tile_w > 0)
            for (int c = blockIdx.x * NT + threadIdx.x; c < F.n_chunks; c += gridDim.x * NT) {
                float ux[4], uy[4];
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const int nd = __ldg(F.chunk_nodes + 4 * c + a);
                    const float2 v = u0 ? u0[nd] : make_float2(0.f, 0.f);
                    ux[a] = v.x;
                    uy[a] = v.y;
                }
                F.chunk_tile[c] = tile_origin(__ldg(F.chunk_box + 2 * c), ux, uy);
            }
    }
    if (!grid_barrier(C.h, [&] { r_init(frames, n_frames, C); })) goto finish;
    // The block's copy of the round state: the header, and for up to FCACHE active frames the
    // active list with its prefix sums and each frame's candidate rule.
    if (threadIdx.x == 0) {
        s_hdr[0] = ld_vol(&C.h->n_active);
        s_hdr[1] = ld_vol(&C.h->total_chunks);
        s_hdr[2] = ld_vol(&C.h->total_groups);
        s_hdr[3] = ld_vol(&C.h->abort);
        s_hdr[4] = 0;
        s_hdr[5] = 0;
        s_hdr[6] = 0;
        s_hdr[7] = ld_vol(&C.h->list_buf);
        s_hdr[8] = 0;
    }
    __syncthreads();
    load_list<ONE>(C, s_hdr[7], s_hdr[0], 0, s_cpre, s_gpre, s_act, s_fi);
    __syncthreads();
    if (!ONE && s_hdr[0] <= FS) {
        keep_frames(s_hdr[0]);
        if ((int)threadIdx.x < s_hdr[0]) s_tag0[threadIdx.x] = __ldcg(C.tag0() + s_act[threadIdx.x]);
        __syncthreads();
    }
    if (!ONE) kept = s_hdr[0] <= FS;
    if (lane == 0 && s_hdr[0] == 1) s_range[wid] = chunk_share(frame(0), s_hdr[1], s_hdr[2], wid);
    __syncthreads();

    while (round < max_rounds) {                    // a slice: at most max_rounds rounds, state kept in HBM
        const int na = ONE ? min(s_hdr[0], 1) : s_hdr[0];
        const int total = s_hdr[1];
        const int tg = s_hdr[2];
        const int lb = s_hdr[7];
        if (na == 0 || s_hdr[3] || s_hdr[4]) break;
        const bool direct = !ONE && na >= 2 && na <= FS && tg <= (int)(gridDim.x * NWARP);
        const bool trr = tr && round < trace_rounds;
        if (trr) trace[7 * round + 0] = gtimer();
        // the active list only shrinks within a launch: the same count means the same list
        const bool pf_use = pf && na == pf_na && total == pf_total;
        if (pf && !pf_use) {
            if (!mbar_wait(&s_bar[wid][pipe_i & 1], (pipe_i >> 1) & 1u) && lane == 0) {   // bounded
                C.h->err = D2IC_WAIT_TIMEOUT;
                atomicExch(&C.h->abort, 1);
            }
            ++pipe_i;
        }
        pf = false;
        const ChunkMeta pm = pf_m;
        pf_m = ChunkMeta{};    // constants while the round runs (nothing to keep in registers)
        // ---- P phase: chunks of the active list spread over the warps (see below) ----
        {
            const bool cached = ONE || na <= FCACHE;
            const int gw = (int)((blockIdx.x * NT + threadIdx.x) >> 5);
            const int nw = (int)((gridDim.x * NT) >> 5);
            auto slot_of = [&](int g) {
                return ONE ? 0 : cached ? find_slot_smem(s_cpre, na, g) : find_slot(C.cp(lb), na, g);
            };
            // lane's chunk g of the active list (nothing if g >= end)
            auto fetch_meta = [&](int g, int end) {
                ChunkMeta m{};
                if (g < end) {
                    const int s = slot_of(g);
                    const int f = ONE ? 0 : cached ? s_act[s] : checked_index(__ldcg(C.act(lb) + s), n_frames, C.h);
                    const int base = ONE ? 0 : cached ? s_cpre[s] : __ldcg(C.cp(lb) + s);
                    const int key = kept ? s : f;
                    m = load_meta<KIND>(frame(key), key, checked_index(g - base, frame(key).n_chunks, C.h), tiles_ok);
                }
                return m;
            };
            // stage the chunk of lane `src` in buffer i & 1: TMA bulk copy of its records, 2-D TMA copy of its tile
            auto stage = [&](int src, int f, int pb, int n, int flags, int origin, unsigned i) {
                if (lane == src) {
                    const d2ic_frame_t &F = frame(f);
                    unsigned long long *bar = &s_bar[wid][i & 1];
                    const unsigned bytes = (flags & CH_STAGED) ? (unsigned)min(n, D2IC_CHUNK_MAX) * 16u : 0u;
                    const unsigned tbytes = (flags & CH_TILED) ? (unsigned)(F.tile_w * F.tile_h) * 4u : 0u;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // after the buffers' generic reads
                    mbar_arrive_tx(bar, bytes + tbytes);
                    if (bytes)
                        bulk_load(wbuf + (i & 1) * CHUNK_BYTES, reinterpret_cast<const uint4 *>(F.pix) + pb, bytes, bar);
                    if (tbytes)
                        tensor_load_2d(wbuf + 2 * CHUNK_BYTES + (i & 1) * TILE_BYTES, frames[ONE ? 0 : kept ? s_act[f] : f].coeff_map,
                                       (int)(short)(origin & 0xffff) + F.pad,
                                       (int)(short)((unsigned)origin >> 16) + F.pad, bar);
                }
                __syncwarp();
            };
            bool p_ok = true;
            // One frame: the warp's contiguous share (chunk_share).  Several frames: chunk g goes to warp
            // g mod (warps), warps counted across the blocks, so that every step of the pass spans few
            // frames (measured faster for batches of small frames); blocks that reduce node groups come last,
            // so that the warps with a chunk more than the others are not theirs.
            const bool contiguous = ONE || na == 1;
            const int reducers = min((tg + NWARP - 1) / NWARP, (int)gridDim.x);
            const int order = (int)blockIdx.x - reducers + ((int)blockIdx.x < reducers ? (int)gridDim.x : 0);
            const int2 range = contiguous ? s_range[wid] : make_int2(wid * (int)gridDim.x + order, total);
            const int cb = range.x, ce = range.y;
            const int cs = contiguous ? 1 : nw;
            for (int g0 = cb; g0 < ce && p_ok; g0 += 32 * cs) {
                const int cnt = min(32, (ce - g0 + cs - 1) / cs);
                ChunkWork w{};
                {
                    const bool have = pf_use && g0 == cb;
                    ChunkMeta m = pm;
                    if (!have) {
                        m = fetch_meta(g0 + lane * cs, ce);
                        stage(0, m.f, m.pb, m.n, m.flags, m.origin, pipe_i);
                    }
                    w.f = m.f;
                    w.pb = m.pb;
                    w.n = m.n;
                    w.origin = m.origin;
                    w.flags = (unsigned)m.flags;
                    if (lane < cnt) {
                        const d2ic_frame_t &F = frame(m.f);
                        const FInfo fi = kept ? s_fi[m.f].info() : cached ? s_fi[slot_of(g0 + lane * cs)].info() : frame_info(C, m.f, round);
                        const Cand cand = make_cand(F, fi);
                        w.tag = fi.tag;
                        const int nd[4] = {m.nd.x, m.nd.y, m.nd.z, m.nd.w};
#pragma unroll
                        for (int a = 0; a < 4; ++a) {
                            float2 dir;
                            const float2 v = cand.at(nd[a], dir);
                            w.ux[a] = v.x;
                            w.uy[a] = v.y;
                            w.rec[a] = (int)((m.slot >> (8 * a)) & 0xffu) * F.n_nodes + nd[a];
                            // for the waiting group: the chunk's first node there, and how many it has there
                            unsigned c2 = 0, first = 1;
#pragma unroll
                            for (int b = 0; b < 4; ++b) {
                                const unsigned same = nd[b] / GN == nd[a] / GN;
                                c2 += same;
                                if (b < a) first &= same ^ 1u;
                            }
                            w.flags |= ((c2 << 1) | first) << (4 + 4 * a);
                        }
                        if (F.tile_w > 0) F.chunk_tile[m.c] = tile_origin(m.box0, w.ux, w.uy);
                        if ((m.flags & (CH_STAGED | CH_TILED)) == (CH_STAGED | CH_TILED) && m.n <= D2IC_CHUNK_MAX &&
                            inside_tile(F, m, w.ux, w.uy))
                            w.flags |= CH_FAST;
                    }
                    __syncwarp();
                }
#pragma unroll 1
                for (int i = 0; i < cnt; ++i) {
                    const bool more = i + 1 < cnt;
                    if (more) stage(i + 1, w.f, w.pb, w.n, (int)w.flags, w.origin, pipe_i + 1);
                    const bool got = mbar_wait(&s_bar[wid][pipe_i & 1], (pipe_i >> 1) & 1u);
                    if (!__all_sync(0xffffffffu, got)) {
                        if (lane == 0) {
                            C.h->err = D2IC_WAIT_TIMEOUT;
                            atomicExch(&C.h->abort, 1);
                        }
                        if (more) mbar_wait(&s_bar[wid][(pipe_i + 1) & 1], ((pipe_i + 1) >> 1) & 1u);   // bounded
                        p_ok = false;
                        break;
                    }
                    chunk_compute<KIND>(frame(ONE ? 0 : __shfl_sync(0xffffffffu, w.f, i)), w, i,
                                        reinterpret_cast<const uint4 *>(wbuf + (pipe_i & 1) * CHUNK_BYTES),
                                        reinterpret_cast<const float *>(wbuf + 2 * CHUNK_BYTES + (pipe_i & 1) * TILE_BYTES),
                                        lane);
                    ++pipe_i;
                }
            }
            if (trr) trace[7 * round + 1] = gtimer();
            // ---- N work: group gi of the active list goes to global warp gi mod (warps in grid); the
            // warp waits until every chunk with a node in the group has written its slots.  With
            // at most one group per warp, a supergroup is the warps of one block and is reduced
            // in shared memory, and frame s's control step runs on warp (warps) - 1 - s, which waits
            // for the supergroup records themselves; otherwise groups go through the frame's global
            // partials and the warp that completes the last supergroup runs the control step. ----
            const bool blockred = tg <= nw;
            int gcur = 0;
            for (int gi = gw, cslot = nw - 1 - gw;;) {
                int cf = -1, cs_slot = 0;
                unsigned ctag = 0;
                if (gi < tg) {
                    int s = 0, f = 0, base = 0;
                    if (ONE) {
                    } else if (cached) {
                        while (gcur + 1 < na && s_gpre[gcur + 1] <= gi) ++gcur;
                        s = gcur;
                        f = s_act[s];
                        base = s_gpre[s];
                    } else {
                        s = find_slot(C.gp(lb), na, gi);
                        f = checked_index(__ldcg(C.act(lb) + s), n_frames, C.h);
                        base = __ldcg(C.gp(lb) + s);
                    }
                    const d2ic_frame_t &F = frame(kept ? s : f);
                    const int g = gi - base;
                    gi += nw;
                    if (g >= F.n_groups) continue;         // padding of the frame's group range
                    if (g < 0) {                           // self-check: the prefix sums are ascending
                        checked_index(g, 0, C.h);
                        continue;
                    }
                    const FInfo fi = cached ? s_fi[s].info() : frame_info(C, f, round);
                    const NodePre pre = node_pre(F, fi, g * GN + lane);   // independent of the pixel pass
                    SlotSums slots;
                    if (!gather_slots(F, g * GN + lane, __ldg(F.group_need + g), fi.tag, C.h, slots)) break;
                    DF q[5];
                    node_post(F, fi, g * GN + lane, pre, slots, q);
                    DF sum = df_reduce5(q, lane);
                    const int which = red5_value(lane);
                    const bool holds = which >= 0 && (lane & 3) == 0;
                    // group -> supergroup (SG groups) -> frame: the warp that completes a supergroup reduces
                    // it; a supergroup's sum is the same lane-ordered warp sum on both paths
                    const int ngr = F.n_groups, nsg = (ngr + SG - 1) / SG, sg = g / SG;
                    const int members = min(SG, ngr - sg * SG);
                    float2 *gp = reinterpret_cast<float2 *>(F.group_part);
                    int last = 0;
                    __syncwarp();
                    if (blockred) {                        // members are warps 0 .. members-1 here
                        if (holds) s_gq[wid][which] = sum;
                        __syncwarp();
                        if (lane == 0) {
                            __threadfence_block();
                            last = atomicAdd(&s_sgcnt, 1) == members - 1;
                            if (last) {
                                s_sgcnt = 0;
                                __threadfence_block();
                            }
                        }
                    } else {
                        if (holds) gp[(size_t)g * D2IC_NPART + which] = make_float2(sum.hi, sum.lo);
                        __syncwarp();
                        if (lane == 0) {
                            last = atom_acq_rel_add(F.group_cnt + sg, 1) == members - 1;
                            if (last) F.group_cnt[sg] = 0;
                        }
                    }
                    __syncwarp();
                    if (__shfl_sync(0xffffffffu, last, 0)) {
                        const int gg = sg * SG + lane;
#pragma unroll
                        for (int i = 0; i < 5; ++i) {
                            q[i] = DF{0.f, 0.f};
                            if (lane < members) {
                                if (blockred) {
                                    q[i] = s_gq[lane][i];
                                } else {
                                    const float2 t2 = __ldcg(gp + (size_t)gg * D2IC_NPART + i);
                                    q[i] = DF{t2.x, t2.y};
                                }
                            }
                        }
                        sum = df_reduce5(q, lane);
                        fence_acq_rel();                   // the supergroup's node data before its records
                        if (holds)
                            st_record(sg_records(F) + (size_t)sg * SG_RECORDS + which,
                                      make_uint4(__float_as_uint(sum.hi), __float_as_uint(sum.lo), fi.tag, 0u));
                        if (!blockred) {
                            int lastf = 0;
                            __syncwarp();
                            if (lane == 0) {
                                lastf = atom_acq_rel_add(F.group_cnt + nsg, 1) == nsg - 1;
                                if (lastf) F.group_cnt[nsg] = 0;
                            }
                            __syncwarp();
                            if (__shfl_sync(0xffffffffu, lastf, 0)) {   // the frame's last supergroup
                                cf = f;
                                cs_slot = s;
                                ctag = fi.tag;
                            }
                        }
                    }
                } else if (blockred && cslot < na) {
                    cf = ONE ? 0 : cached ? s_act[cslot] : checked_index(__ldcg(C.act(lb) + cslot), n_frames, C.h);
                    ctag = cached ? s_fi[cslot].tag : frame_tag(C, cf, round);
                    cs_slot = cslot;
                    cslot += nw;
                } else {
                    break;
                }
                if (cf >= 0) {
                    FrameState local;
                    control_step<ONE>(frames, frame(kept ? cs_slot : cf), n_frames, C, cf, ctag, ONE ? 1 : na, blockred, direct,
                                      cs_slot, s_act, round, s_hdr[8], eval_only, stop_flags, trace, trace_rounds, lane,
                                      ONE ? s_state : local);
                }
            }
            if (trr) trace[7 * round + 2] = gtimer();
            // load the next round's first batch (same ranges if the active list is unchanged).  Only
            // from the shared-memory copy of the list: the global one may be rebuilt meanwhile.
            if (cached && p_ok && cb < ce && round + 1 < max_rounds && !ld_vol(&C.h->abort)) {
                pf_m = fetch_meta(cb + lane * cs, ce);
                stage(0, pf_m.f, pf_m.pb, pf_m.n, pf_m.flags, pf_m.origin, pipe_i);
                pf = true;
                pf_na = na;
                pf_total = total;
            }
        }
        // ---- end of round: one thread per block polls the release record (direct rounds: one warp the
        // rule records).  Records only move forward; a block that had no work in a round may find a later one. ----
        __syncthreads();
        auto wait_release = [&](unsigned target) {       // one thread
            uint4 r = ld_record(&C.h->rel);
            unsigned long long t0 = 0;
            int dead = 0;
            for (unsigned it = 0; r.x < target; ++it) {
                if ((it & 63) == 63) {
                    const unsigned long long now = gtimer();
                    if (t0 == 0) t0 = now;
                    if (ld_vol(&C.h->abort)) dead = 1;
                    else if (now - t0 > WAIT_NS) {
                        C.h->err = D2IC_WAIT_TIMEOUT;
                        atomicExch(&C.h->abort, 1);
                        dead = 1;
                    }
                    if (dead) break;
                }
                r = ld_record(&C.h->rel);
            }
            fence_acq_rel();
            s_hdr[3] = dead;
            if (!dead) {
                s_hdr[4] = (int)(r.y & REL_STOP);
                s_hdr[6] = (int)r.x;
                if ((r.y & REL_INLINE) && (int)(r.y >> 16) == s_hdr[8]) {   // na == 1 and the list unchanged
                    s_fi[0] = FRule{__uint_as_float(r.z), __uint_as_float(r.w), r.y,
                                    (s_fi[0].tag + (r.x - (unsigned)round)) & TAG_MASK};
                    s_hdr[5] = REFRESH_NONE;
                } else {
                    if ((int)(r.y >> 16) != s_hdr[8]) {   // the list changed: the header of the round released last
                        for (int t = 0; t < 64; ++t) {
                            s_hdr[0] = ld_vol(&C.h->n_active);
                            s_hdr[1] = ld_vol(&C.h->total_chunks);
                            s_hdr[2] = ld_vol(&C.h->total_groups);
                            s_hdr[7] = ld_vol(&C.h->list_buf);
                            fence_acq_rel();
                            const uint4 r2 = ld_record(&C.h->rel);
                            if (r2.x == r.x) break;
                            r = r2;
                        }
                        s_hdr[4] = (int)(r.y & REL_STOP);
                        s_hdr[6] = (int)r.x;
                        s_hdr[8] = (int)(r.y >> 16);
                        s_hdr[5] = REFRESH_LIST;
                    } else {
                        s_hdr[5] = REFRESH_RULES;
                    }
                }
                // rounds passed over: their list reads are done as well
                if (r.x > target) atomicAdd(&C.h->blocks_past, r.x - target);
            }
        };
        const unsigned target = (unsigned)(round + 1);
        if (threadIdx.x == 0) atomicAdd(&C.h->blocks_past, 1u);   // this block's list reads of the round are done
        if (!direct) {
            if (threadIdx.x == 0) wait_release(target);
        } else if (wid == 0) {
            const uint4 *mine = C.rule + s_act[min(lane, na - 1)];
            uint4 r;
            unsigned long long t0 = 0;
            bool dead = false;
            for (unsigned it = 0;; ++it) {
                r = ld_record(mine);
                if (__all_sync(0xffffffffu, r.x >= target)) break;
                if ((it & 63) == 63 && !keep_waiting(C.h, t0, lane)) {
                    dead = true;
                    break;
                }
            }
            fence_acq_rel();
            const bool now = r.x == target;
            const bool fin = __any_sync(0xffffffffu, now && (r.y & REL_FIN)), stop = __any_sync(0xffffffffu, now && (r.y & REL_STOP));
            if (!dead && lane < na)
                s_fi[lane] = FRule{__uint_as_float(r.z), __uint_as_float(r.w), r.y, (s_tag0[lane] + r.x) & TAG_MASK};
            if (lane == 0) {
                s_hdr[3] = dead;
                s_hdr[4] = 0;
                s_hdr[5] = REFRESH_NONE;
                s_hdr[6] = (int)target;
                if (fin && !dead) wait_release(target);
                if (stop) s_hdr[4] = 1;
            }
        }
        __syncthreads();
        if (s_hdr[5] != REFRESH_NONE && !s_hdr[3]) {    // rules from the frame states; a changed list is reloaded
            if (s_hdr[5] == REFRESH_RULES) {
                if (na <= FCACHE)
                    for (int s = threadIdx.x; s < na; s += NT) s_fi[s] = make_rule(frame_info<ONE>(C, s_act[s], s_hdr[6]));
            } else if (s_hdr[0] > 0) {
                // after direct rounds the rules are the records' (the states may still be on their way); the
                // new list's frames are among the old one's
                const int n2 = s_hdr[0], t = (int)threadIdx.x;
                FRule rule{};
                const bool have = direct && t < n2;
                if (have) {
                    const int f = checked_index(__ldcg(C.act(s_hdr[7]) + t), C.n, C.h);
                    const uint4 r = ld_record(C.rule + f);
                    rule = FRule{__uint_as_float(r.z), __uint_as_float(r.w), r.y, frame_tag(C, f, (int)r.x)};
                }
                __syncthreads();
                load_list<ONE>(C, s_hdr[7], n2, s_hdr[6], s_cpre, s_gpre, s_act, s_fi);
                if (have) s_fi[t] = rule;                // written by this thread in load_list, too
                __syncthreads();
                if (!ONE && n2 <= FS) {
                    keep_frames(n2);
                    if (t < n2) s_tag0[t] = __ldcg(C.tag0() + s_act[t]);
                    __syncthreads();
                }
                if (!ONE) kept = n2 <= FS;
                if (lane == 0 && n2 == 1) s_range[wid] = chunk_share(frame(0), s_hdr[1], s_hdr[2], wid);
            }
            __syncthreads();
        }
        const int next_round = s_hdr[3] ? round + 1 : s_hdr[6];
        if (trr) trace[7 * round + 5] = gtimer();
        round = next_round;
    }

    if (pf) {                                       // no copy in flight at exit (bounded wait)
        mbar_wait(&s_bar[wid][pipe_i & 1], (pipe_i >> 1) & 1u);
    }

finish:
    // ---- outputs of frames that finished in this launch; running frames report D2IC_RUNNING ----
    const bool aborted = ld_vol(&C.h->abort) != 0;
    for (int f = 0; f < n_frames; ++f) {
        const d2ic_frame_t &F = frames[f];
        const FrameState *S = C.fs + f;
        const bool done = ld_vol(&S->state) == ST_DONE;
        if (!(aborted || eval_only || (done && !ld_vol(&S->reported)))) {
            if (!done && blockIdx.x == 0 && threadIdx.x == 0 && F.status) *F.status = D2IC_RUNNING;
            continue;
        }
        const int iu = ld_vol(&S->iu), igc = ld_vol(&S->igc);
        const int nn = F.n_nodes;
        float2 *uo = reinterpret_cast<float2 *>(F.u_out);
        for (int i = blockIdx.x * NT + threadIdx.x; i < nn; i += gridDim.x * NT) {
            if (uo) uo[i] = __ldcg(nbuf(F, iu) + i);
            if (eval_only && grad_out && f == 0) reinterpret_cast<float2 *>(grad_out)[i] = __ldcg(nbuf(F, 2 + igc) + i);
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            if (F.n_iters) *F.n_iters = ld_vol(&S->k);
            if (F.n_evals) *F.n_evals = ld_vol(&S->n_evals);
            int st = D2IC_OK;
            if (aborted) st = ld_vol(&C.h->err);
            else if (ld_vol(&S->nan_seen)) st = D2IC_NAN_DETECTED;
            else if (ld_vol(&S->k) >= F.max_iter && F.max_iter > 0) st = D2IC_MAX_ITERS;
            if (F.status) *F.status = st;
            if (eval_only && J_out && f == 0) *J_out = *(volatile const double *)&S->J_cur;
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
constexpr size_t ENGINE_SMEM = (size_t)NWARP * WARP_SMEM;   // per warp: 2 record + 2 tile buffers

template <int KIND>
static cudaError_t occupancy(int *blocks_per_sm) {
    cudaError_t e = cudaFuncSetAttribute(cg_engine<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ENGINE_SMEM);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(cg_engine<KIND, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ENGINE_SMEM);
    if (e != cudaSuccess) return e;
    int one = 0;   // the one-frame instance must fit as many blocks as the general one
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&one, cg_engine<KIND, true>, NT, ENGINE_SMEM);
    if (e != cudaSuccess) return e;
    int many = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&many, cg_engine<KIND>, NT, ENGINE_SMEM);
    *blocks_per_sm = one < many ? one : many;
    return e;
}

struct DevInfo {
    int sms = 0, bps[2] = {0, 0};
};
static DevInfo g_dev[64];

static int dev_info(int dev, DevInfo **out) {
    if (dev < 0 || dev >= 64) {
        set_error("device index %d out of range", dev);
        return D2IC_BAD_ARG;
    }
    DevInfo &d = g_dev[dev];
    if (d.sms == 0) {
        cudaError_t e = cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return cuda_status(e, "cudaDeviceGetAttribute");
        e = occupancy<D2IC_INTERP_CUBIC>(&d.bps[0]);
        if (e != cudaSuccess) return cuda_status(e, "occupancy");
        e = occupancy<D2IC_INTERP_LINEAR>(&d.bps[1]);
        if (e != cudaSuccess) return cuda_status(e, "occupancy");
    }
    *out = &d;
    return D2IC_OK;
}

static int launch_engine(const d2ic_frame_t *frames, int n_frames, void *control, size_t control_bytes, int kind,
                         int grid_blocks, int eval_only, const float *u_eval, double *J_out, float *grad_out,
                         unsigned long long *trace, int trace_rounds, cudaStream_t s, int max_rounds = 0x7fffffff,
                         bool new_batch = true, int stop_flags = 0) {
    D2IC_REQUIRE(frames && control, "cg engine: null pointer");
    D2IC_REQUIRE(n_frames >= 1 && n_frames <= D2IC_MAX_FRAMES, "cg engine: n_frames %d out of [1, %d]", n_frames,
                 D2IC_MAX_FRAMES);
    D2IC_REQUIRE(kind == D2IC_INTERP_CUBIC || kind == D2IC_INTERP_LINEAR, "cg engine: unknown interpolation %d", kind);
    D2IC_REQUIRE(((uintptr_t)control & 255) == 0, "cg engine: control scratch must be 256-byte aligned");
    const size_t need = d2ic_cg_control_bytes(n_frames);
    D2IC_REQUIRE(control_bytes >= need, "cg engine: control scratch %zu bytes < %zu needed", control_bytes, need);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e, "cudaGetDevice");
    DevInfo *di = nullptr;
    int st = dev_info(dev, &di);
    if (st) return st;
    const int maxb = di->sms * di->bps[kind == D2IC_INTERP_LINEAR];
    D2IC_REQUIRE(maxb > 0, "cg engine: kernel cannot be resident on this device");
    int blocks = grid_blocks > 0 ? (grid_blocks < maxb ? grid_blocks : maxb) : maxb;
    // header always; with new_batch also the command words (all frames CMD_INIT == 0)
    const size_t clear = new_batch ? align256(sizeof(CtlHeader)) + sizeof(int) * (size_t)n_frames : sizeof(CtlHeader);
    e = cudaMemsetAsync(control, 0, clear, s);
    if (e != cudaSuccess) return cuda_status(e, "control reset");
    char *cb = (char *)control;
    // cooperative launch through cudaLaunchKernelEx (co-residency checked by the driver; capturable)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = ENGINE_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const bool one = n_frames == 1;
    if (kind == D2IC_INTERP_CUBIC)
        e = one ? cudaLaunchKernelEx(&cfg, cg_engine<D2IC_INTERP_CUBIC, true>, frames, n_frames, cb, eval_only, u_eval,
                                     J_out, grad_out, trace, trace_rounds, max_rounds, stop_flags)
                : cudaLaunchKernelEx(&cfg, cg_engine<D2IC_INTERP_CUBIC>, frames, n_frames, cb, eval_only, u_eval, J_out,
                                     grad_out, trace, trace_rounds, max_rounds, stop_flags);
    else
        e = one ? cudaLaunchKernelEx(&cfg, cg_engine<D2IC_INTERP_LINEAR, true>, frames, n_frames, cb, eval_only,
                                     u_eval, J_out, grad_out, trace, trace_rounds, max_rounds, stop_flags)
                : cudaLaunchKernelEx(&cfg, cg_engine<D2IC_INTERP_LINEAR>, frames, n_frames, cb, eval_only, u_eval,
                                     J_out, grad_out, trace, trace_rounds, max_rounds, stop_flags);
    if (e != cudaSuccess) return cuda_status(e, "cooperative launch of cg_engine");
    return D2IC_OK;
}

}  // namespace d2ic

using namespace d2ic;

extern "C" size_t d2ic_cg_control_bytes(int n_frames) {
    if (n_frames < 1) n_frames = 1;
    size_t a, b, c, d, e;
    return ctl_layout(n_frames, &a, &b, &c, &d, &e);
}

// Workspace of one frame: 7 node buffers (u x2, g x3, dir x2), the K gradient
// slots per node (tagged 16-byte records: gx, gy, a word of the chunk's r^2 sum, the tag),
// the partials (D2IC_NPART double-float pairs) of every group and the tagged
// records of every supergroup of SG groups, the completion counters (supergroups
// and the frame's count of them), and the tile origins (4 bytes per chunk).
static size_t ws_layout(int n_nodes, int n_chunks, int node_chunk_k, size_t off[5]) {
    const size_t ng = (size_t)(n_nodes + GN - 1) / GN;
    size_t o = 0;
    off[0] = o;                                               // node_ws
    o += align256(sizeof(float) * 14 * (size_t)n_nodes);
    off[1] = o;                                               // node_grad
    o += align256(sizeof(float) * 4 * (size_t)node_chunk_k * n_nodes);
    off[2] = o;                                               // group_part
    const size_t ns = (ng + SG - 1) / SG;                     // supergroups of SG groups
    o += align256(sg_record_offset((int)ng) + sizeof(uint4) * SG_RECORDS * ns);
    off[3] = o;                                               // group_cnt
    o += align256(sizeof(int) * (ns + 1));
    // no less than for double-float partials of the groups and supergroups and a counter for each: the size
    // of a frame that the fixed scratch array takes does not depend on how the sums are handed over
    const size_t least = off[2] + align256(sizeof(float) * 2 * D2IC_NPART * (ng + ns)) + align256(sizeof(int) * (ng + ns + 1));
    if (o < least) o = least;
    off[4] = o;                                               // chunk_tile
    o += align256(sizeof(int) * (size_t)(n_chunks > 0 ? n_chunks : 1));
    return o;
}

extern "C" size_t d2ic_frame_workspace_bytes(int n_nodes, int n_chunks, int node_chunk_k) {
    size_t off[5];
    if (node_chunk_k < 1) node_chunk_k = 1;
    if (n_nodes < 1) n_nodes = 1;
    return ws_layout(n_nodes, n_chunks, node_chunk_k, off);
}

extern "C" int d2ic_frame_bind_workspace(d2ic_frame_t *f, void *ws) {
    D2IC_REQUIRE(f && ws, "d2ic_frame_bind_workspace: null pointer");
    D2IC_REQUIRE(((uintptr_t)ws & 255) == 0, "d2ic_frame_bind_workspace: workspace must be 256-byte aligned");
    D2IC_REQUIRE(f->n_nodes >= 1 && f->n_chunks >= 0 && f->node_chunk_k >= 1 && f->node_chunk_k <= 255,
                 "d2ic_frame_bind_workspace: bad sizes");
    size_t off[5];
    ws_layout(f->n_nodes, f->n_chunks, f->node_chunk_k, off);
    char *p = (char *)ws;
    f->node_ws = (float *)(p + off[0]);
    f->node_grad = (float *)(p + off[1]);
    f->group_part = (float *)(p + off[2]);
    f->group_cnt = (int *)(p + off[3]);
    f->chunk_tile = (int *)(p + off[4]);
    f->n_groups = (f->n_nodes + GN - 1) / GN;
    return D2IC_OK;
}

// Tensor-map encoding comes from the driver through the runtime's entry-point
// query, so the library does not link libcuda directly.
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

extern "C" int d2ic_frame_encode_tiles(d2ic_frame_t *f, int tile_w, int tile_h) {
    static_assert(sizeof(d2ic_frame_t) % 64 == 0, "descriptor arrays keep every tensor map 64-byte aligned");
    static_assert(offsetof(d2ic_frame_t, coeff_map) == 0 && sizeof(f->coeff_map) == sizeof(CUtensorMap),
                  "tensor map first in the descriptor");
    D2IC_REQUIRE(f, "d2ic_frame_encode_tiles: null frame");
    memset(f->coeff_map, 0, sizeof(f->coeff_map));
    f->tile_w = 0;
    f->tile_h = 0;
    if (tile_w == 0) return D2IC_OK;
    D2IC_REQUIRE(tile_w >= 4 && tile_w % 4 == 0 && tile_h >= 4 && tile_w <= 256 && tile_h <= 256 &&
                     tile_w * tile_h <= D2IC_TILE_MAX_FLOATS,
                 "d2ic_frame_encode_tiles: tile %d x %d (width a multiple of 4, at most %d floats)", tile_w, tile_h,
                 D2IC_TILE_MAX_FLOATS);
    D2IC_REQUIRE(f->coeff && ((uintptr_t)f->coeff & 15) == 0, "d2ic_frame_encode_tiles: coeff must be 16-byte aligned");
    D2IC_REQUIRE(f->pad % 4 == 0 && f->cpitch % 4 == 0 && f->W >= 1 && f->H >= 1 && f->cpitch >= f->W + 2 * f->pad,
                 "d2ic_frame_encode_tiles: pad and cpitch must be multiples of 4 (pad %d, cpitch %d)", f->pad,
                 f->cpitch);
    D2IC_REQUIRE(f->W + 2 * f->pad < 32768 && f->H + 2 * f->pad < 32768,
                 "d2ic_frame_encode_tiles: image %d x %d too large for tile origins", f->W, f->H);
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) {
        set_error("d2ic_frame_encode_tiles: the driver provides no cuTensorMapEncodeTiled");
        return D2IC_UNSUPPORTED;
    }
    alignas(64) CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)(f->W + 2 * f->pad), (cuuint64_t)(f->H + 2 * f->pad)};
    const cuuint64_t strides[1] = {(cuuint64_t)f->cpitch * sizeof(float)};
    const cuuint32_t box[2] = {(cuuint32_t)tile_w, (cuuint32_t)tile_h};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void *)f->coeff, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("d2ic_frame_encode_tiles: cuTensorMapEncodeTiled failed (%d)", (int)r);
        return D2IC_CUDA_ERROR;
    }
    memcpy(f->coeff_map, &map, sizeof(map));
    f->tile_w = tile_w;
    f->tile_h = tile_h;
    return D2IC_OK;
}

extern "C" int d2ic_device_info(int device, int *num_sms, int *engine_blocks_per_sm) {
    DevInfo *di = nullptr;
    int st = dev_info(device, &di);
    if (st) return st;
    if (num_sms) *num_sms = di->sms;
    if (engine_blocks_per_sm) *engine_blocks_per_sm = di->bps[0];
    return D2IC_OK;
}

extern "C" int d2ic_cg_solve_batched(const d2ic_frame_t *frames, int n_frames, void *control, size_t control_bytes,
                                     int interp_kind, int grid_blocks, void *stream) {
    return launch_engine(frames, n_frames, control, control_bytes, interp_kind, grid_blocks, 0, nullptr, nullptr,
                         nullptr, nullptr, 0, (cudaStream_t)stream);
}

extern "C" size_t d2ic_cg_command_offset(void) { return align256(sizeof(CtlHeader)); }

extern "C" int d2ic_cg_slice(const d2ic_frame_t *frames, int n_frames, void *control, size_t control_bytes,
                             int interp_kind, int grid_blocks, int max_rounds, void *stream) {
    D2IC_REQUIRE(max_rounds >= 1, "d2ic_cg_slice: max_rounds must be >= 1 (got %d)", max_rounds);
    return launch_engine(frames, n_frames, control, control_bytes, interp_kind, grid_blocks, 0, nullptr, nullptr,
                         nullptr, nullptr, 0, (cudaStream_t)stream, max_rounds, false);
}

extern "C" int d2ic_cg_slice_ex(const d2ic_frame_t *frames, int n_frames, void *control, size_t control_bytes,
                                int interp_kind, int grid_blocks, int max_rounds, int stop_flags, void *stream) {
    D2IC_REQUIRE(max_rounds >= 1, "d2ic_cg_slice_ex: max_rounds must be >= 1 (got %d)", max_rounds);
    D2IC_REQUIRE((stop_flags & ~(D2IC_STOP_ON_FINISH | D2IC_STOP_ON_IRQ)) == 0, "d2ic_cg_slice_ex: unknown stop flags %d",
                 stop_flags);
    return launch_engine(frames, n_frames, control, control_bytes, interp_kind, grid_blocks, 0, nullptr, nullptr,
                         nullptr, nullptr, 0, (cudaStream_t)stream, max_rounds, false, stop_flags);
}

extern "C" size_t d2ic_cg_irq_offset(void) { return offsetof(CtlHeader, irq); }

extern "C" int d2ic_cg_solve_traced(const d2ic_frame_t *frames, int n_frames, void *control, size_t control_bytes,
                                    int interp_kind, int grid_blocks, unsigned long long *trace, int trace_rounds,
                                    void *stream) {
    D2IC_REQUIRE(trace && trace_rounds > 0, "d2ic_cg_solve_traced: need a trace buffer");
    return launch_engine(frames, n_frames, control, control_bytes, interp_kind, grid_blocks, 0, nullptr, nullptr,
                         nullptr, trace, trace_rounds, (cudaStream_t)stream);
}

extern "C" int d2ic_eval_objective(const d2ic_frame_t *frame, const float *u, void *control, size_t control_bytes,
                                   int interp_kind, double *J_out, float *grad_out, void *stream) {
    D2IC_REQUIRE(u && J_out && grad_out, "d2ic_eval_objective: null pointer");
    return launch_engine(frame, 1, control, control_bytes, interp_kind, 0, 1, u, J_out, grad_out, nullptr, 0,
                         (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Solve without allocating: scratch in a fixed device array
// ---------------------------------------------------------------------------
// For callers that cannot call cudaMalloc (an allocator-less runtime, a
// plugin host that owns all device memory, code running where allocation is
// forbidden): the engine's scratch -- the frame descriptor copy, the control
// block and the per-frame workspace -- is carved from this file-scope device
// array instead of caller memory.  Every GPU that loads the library holds the
// array until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[D2IC_NOALLOC_SCRATCH_BYTES];
// device address of the array, per device (the host-side name is a stand-in, not a device address);
// atomic so that threads making their first call on a device at the same time do not race
static std::atomic<void *> g_noalloc_addr[64];

// Writes a frame descriptor into the scratch array.  The descriptor travels as a kernel argument,
// copied at launch, so no host buffer has to outlive the call and the host does not wait.
__global__ void noalloc_put_descriptor(const d2ic_frame_t f, d2ic_frame_t *dst) {
    static_assert(sizeof(d2ic_frame_t) % 8 == 0, "descriptor copied in 8-byte words");
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(&f);
    unsigned long long *d = reinterpret_cast<unsigned long long *>(dst);
    for (int i = threadIdx.x; i < (int)(sizeof(d2ic_frame_t) / 8); i += blockDim.x) d[i] = src[i];
}

extern "C" int d2ic_cg_solve_noalloc(const d2ic_frame_t *frame, int interp_kind, void *stream) {
    D2IC_REQUIRE(frame, "d2ic_cg_solve_noalloc: null frame");
    D2IC_REQUIRE(frame->n_nodes >= 1 && frame->n_chunks >= 0, "d2ic_cg_solve_noalloc: bad sizes");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e, "cudaGetDevice");
    D2IC_REQUIRE(dev >= 0 && dev < 64, "d2ic_cg_solve_noalloc: device index %d out of range", dev);
    const size_t desc_bytes = align256(sizeof(d2ic_frame_t));
    const size_t ctl_bytes = d2ic_cg_control_bytes(1);
    D2IC_REQUIRE(frame->node_chunk_k >= 1 && frame->node_chunk_k <= 255, "d2ic_cg_solve_noalloc: bad node_chunk_k");
    const size_t ws_bytes = d2ic_frame_workspace_bytes(frame->n_nodes, frame->n_chunks, frame->node_chunk_k);
    const size_t need = desc_bytes + ctl_bytes + ws_bytes;
    D2IC_REQUIRE(need <= (size_t)D2IC_NOALLOC_SCRATCH_BYTES,
                 "d2ic_cg_solve_noalloc: frame needs %zu bytes of scratch (%d nodes, %d chunks), more than the "
                 "fixed %zu-byte array; use d2ic_cg_solve_batched with caller-allocated scratch",
                 need, frame->n_nodes, frame->n_chunks, (size_t)D2IC_NOALLOC_SCRATCH_BYTES);
    void *addr = g_noalloc_addr[dev].load(std::memory_order_relaxed);
    if (addr == nullptr) {                     // set-up, once per device, with that device current
        e = cudaGetSymbolAddress(&addr, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_status(e, "cudaGetSymbolAddress(noalloc scratch)");
        g_noalloc_addr[dev].store(addr, std::memory_order_relaxed);
    }
    char *base = (char *)addr;
    d2ic_frame_t f = *frame;                   // caller's inputs/outputs, workspace from the array
    int st = d2ic_frame_bind_workspace(&f, base + desc_bytes + ctl_bytes);
    if (st) return st;
    cudaStream_t s = (cudaStream_t)stream;
    noalloc_put_descriptor<<<1, 64, 0, s>>>(f, (d2ic_frame_t *)base);
    D2IC_CHECK_LAUNCH("noalloc descriptor write");
    // the launch clears the control header on `s`; the kernel initialises every workspace word it reads
    return launch_engine((const d2ic_frame_t *)base, 1, base + desc_bytes, ctl_bytes, interp_kind, 0, 0, nullptr,
                         nullptr, nullptr, nullptr, 0, s);
}
