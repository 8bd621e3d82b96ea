// Grouped matrix product of many rows a group on the fifth-generation tensor cores with CTA PAIRS: the prompt-sized form of
// grouped_mma.cu, for the experts of a routed feed-forward (rows sorted by expert, known only on the device):
//     C[c_row(r), n] = sum_k A[r, k] * W[g][n, k],   or   silu(gate) * up of two row blocks of W[g],   r in offsets[g] .. offsets[g+1]-1.
//
// The machinery is gemm_tc2.cu's: transposed, 256 WEIGHT rows a pair on the instruction's M side, a tile of the group's rows on its N
// side, each CTA staging half of both operands by TMA, accumulators in tensor memory, persistent pairs with one warp for the
// copies, one for the MMAs and four for the epilogue.  What differs is the list of tiles: every pair works it out from the
// offsets, a group's rows cut into as few tiles of at most `tok_cap` as they need, all of about the same size, and the
// instruction's N is that size (a multiple of 32), so a group of 200 rows costs 224 columns and not 256.  A group's weight is
// read once for every one of its row tiles, which is why they go up to 256 rows, as many as leave room for two accumulators.  For the
// gated form a CTA's 128 weight rows are 64 gate rows above the 64 up rows of the same outputs, and two epilogue warps exchange
// halves of what they read (128 gate and 128 up rows in two accumulators of 256 columns would leave tensor memory no second pair).
// The epilogue has to keep up with a tile's products (10 us at 2,048 elements of K): with a branch per value in it, the full
// quotient's among them, it took three times that, and gate/up 285 us in place of 168.
//
// At 2,048 tokens, 64 experts of 1,408, six chosen (192 rows an expert, width 2,048): 168 us for gate/up (142 GFLOP, 845 TFLOP/s; tensor
// pipe 61 % busy, DRAM 62 %), 30 for gathering its rows, half of it beside other kernels, 108 for down; the mma.sync kernel (grouped_mma.cu) takes 617 and 379.
// The weights alone are 1.1 GB, 170 us of memory time.  Which kernel takes a product: kernels/grouped.py, pair_pays.
//
// Every mbarrier wait is bounded (error flag, then everybody falls through to the common end); the two cluster barriers
// (after set-up, before exit) are reached on every path.
#include "common.cuh"

#include <cooperative_groups.h>
#include <cuda.h>
#include <cstdlib>

using namespace mlb;

MLB_DEFINE_LAST_ERROR()

namespace {

constexpr int BLOCK_W = 128;                 // weight rows per CTA
constexpr int PAIR_W = 256;                  // weight rows per pair (MMA M)
constexpr int HALF_W = 64;                   // weight rows of one copy
constexpr int BLOCK_K = 64;                  // bf16 per stage row: 128 bytes, one swizzle span
constexpr int UMMA_K = 16;
constexpr int A_TILE_BYTES = BLOCK_W * BLOCK_K * 2;
constexpr int MAX_STAGES = 8;
constexpr int THREADS = 192;
constexpr int SPIN_LIMIT = 1 << 21;          // polls of up to 2 us each
constexpr int TMEM_COLS = 512;
#ifndef WAIT_HINT_NS
#define WAIT_HINT_NS 2000
#endif

constexpr int MAX_GROUPS = 1024;

struct GroupedParams {
    void* out;                 // fp32 or bf16, rows of pitch ldo
    const int* offsets;        // [G + 1]
    const int* c_rows;         // the row written for a place (null: the place itself; negative: none)
    const float* row_scale;    // dual: both products times row_scale[scale_rows[place]] in front of the activation (null: 1)
    const int* scale_rows;
    int* error_flag;
    long long ldo;
    int M, N, G;               // places in the list, outputs (with dual: gate rows), groups
    int w_rows;                // weight rows of a group
    int up_offset;             // dual: the up rows start this many rows behind the gate rows
    int tok_cap;               // rows of a tile at most: 32 or a multiple of 64
    int k_blocks, stages, n_tiles;
    int out_bf16, dual, act;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// the address, in the cluster's shared window, of `addr` in the CTA of rank `rank`
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// One poll.  The hint lets the hardware park the thread until the phase completes or the time (ns) is up,
// so that waiting threads do not hammer shared memory while the tensor core reads its operands from it.
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"((uint32_t)WAIT_HINT_NS) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* error_flag, int code) {
    for (int i = 0; i < SPIN_LIMIT; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    if (error_flag) atomicExch(error_flag, code);
    return false;
}
// a whole warp waits: one lane polls, the others sleep at the warp barrier
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, int* error_flag, int code) {
    bool ok = true;
    if ((threadIdx.x & 31) == 0) ok = mbar_wait(bar, parity, error_flag, code);
    return __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
}
// true in exactly one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(pred));
    return pred != 0;
}
// this CTA's half of an operand tile; the bytes are counted on `cluster_bar`, which may live in the peer CTA
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t cluster_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(cluster_bar) : "memory");
}
// K-major operand tile, 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// kind::f16: fp32 accumulator, bf16 A and B, both K-major, M = 256 over the pair
__device__ __forceinline__ uint32_t umma_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(PAIR_W >> 4) << 24);
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives, once the pair's MMAs so far have completed, on the barrier at this offset in BOTH CTAs
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t addr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// a / y, rounded as a division is, for y in [1, QUOTIENT_MAX] and |a| <= QUOTIENT_MAX, without a branch (the values a thread holds are
// then divided side by side and not one behind another): the reciprocal refined by one Newton step, the quotient corrected by its
// remainder (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).  Above 2^126 the
// reciprocal would be flushed to zero.  Of all fp32 gates within the limits, g / (1 + e^-g) and 1 / (1 + e^(-1.702 g)) have the bits of
// the division, every one compared on a B200.
constexpr float QUOTIENT_MAX = 0x1p125f;
__device__ __forceinline__ float quotient(float a, float y) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    r = fmaf(r, fmaf(-y, r, 1.0f), r);
    const float q = a * r;
    return fmaf(-fmaf(y, q, -a), r, q);               // (this sign of the remainder keeps the sign of a zero)
}
// g <- the gated values.  silu(g) * u, or the clamped form with its limit L: g = min(g, L), u = clamp(u, -L, L), g sigmoid(1.702 g) (u + 1);
// grouped_mma.cu's bits.  A warp with a gate beyond the quotient's range (about -87 and -51, or not finite) divides one by one.
template <bool CLAMPED>
__device__ __forceinline__ void gated_values(float (&g)[16], const float (&u)[16], float limit) {
    float y[16];
    bool near = true;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        if (CLAMPED) g[j] = fminf(g[j], limit);
        y[j] = 1.0f + expf(CLAMPED ? -1.702f * g[j] : -g[j]);
        near = near && y[j] <= QUOTIENT_MAX && fabsf(g[j]) <= QUOTIENT_MAX;
    }
    if (__all_sync(0xffffffffu, near)) {
#pragma unroll
        for (int j = 0; j < 16; ++j) y[j] = quotient(CLAMPED ? 1.0f : g[j], y[j]);
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) y[j] = (CLAMPED ? 1.0f : g[j]) / y[j];
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) g[j] = CLAMPED ? g[j] * y[j] * (fminf(fmaxf(u[j], -limit), limit) + 1.0f) : y[j] * u[j];
}

// The tiles of the list, walked in increasing order by every role of a pair.
struct Tiles {
    const int *offsets, *starts;          // rows of the groups; first tile of the groups (both in shared memory)
    int n_tiles, tok_cap, tile_outputs, group = 0;
    int n0, row0, rows, cols;             // the tile: first output, first place, places, the instruction's N
    __device__ __forceinline__ static int row_tiles(int rows, int cap) { return (rows + cap - 1) / cap; }
    __device__ __forceinline__ void seek(int tile) {
        while (tile >= starts[group + 1]) ++group;
        const int first = offsets[group], count = offsets[group + 1] - first, m_tiles = row_tiles(count, tok_cap);
        const int each = ((count + m_tiles - 1) / m_tiles + 31) & ~31, at = tile - starts[group];
        n0 = (at / m_tiles) * tile_outputs;
        row0 = first + (at % m_tiles) * each;
        rows = min(each, first + count - row0);          // (at least one: each <= tok_cap, and m_tiles - 1 full tiles hold fewer than count)
        cols = each;
    }
};

__global__ void __launch_bounds__(THREADS, 1)
grouped_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, GroupedParams p) {
    pdl_launch_dependents();
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long full_bar[MAX_STAGES], empty_bar[MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int offsets_s[MAX_GROUPS + 1], starts_s[MAX_GROUPS + 1], sums_s[THREADS / 32];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster.block_rank();                       // 0: leader (issues the MMAs)
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
    const int box_rows = p.tok_cap / 2;                               // rows of A that a CTA stages; the instruction reads the first cols / 2
    const uint32_t ring = (smem_u32(smem_dyn) + 1023u) & ~1023u;      // same offset in both CTAs
    const uint32_t stage_bytes = A_TILE_BYTES + (uint32_t)box_rows * BLOCK_K * 2;
    const uint32_t exchange = ring + (uint32_t)p.stages * stage_bytes;      // dual: gate and up rows meet here (see the epilogue)
    const uint32_t acc_cols = TMEM_COLS / 2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);             // the leader's expect_tx arrival
            mbar_init(smem_u32(&empty_bar[s]), 1);            // the leader's multicast commit
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full[b]), 1);             // multicast commit
            mbar_init(smem_u32(&acc_empty[b]), 8);            // leader's copy: 4 epilogue warps of each CTA
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {                                          // the same warp of both CTAs allocates for the pair
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_s)), "r"((uint32_t)TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    // the groups' first rows, and their first tiles: a running sum over the groups, THREADS of them at a time
    for (int g = threadIdx.x; g <= p.G; g += THREADS) offsets_s[g] = min(max(p.offsets[g], 0), p.M);
    __syncthreads();
    int tiles_before = 0;
    for (int g0 = 0; g0 < p.G; g0 += THREADS) {
        const int g = g0 + threadIdx.x;
        const int own = g < p.G ? p.n_tiles * Tiles::row_tiles(max(0, offsets_s[g + 1] - offsets_s[g]), p.tok_cap) : 0;
        int inc = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += n;
        }
        if (lane == 31) sums_s[warp] = inc;
        __syncthreads();
        int before = tiles_before;
        for (int w = 0; w < THREADS / 32; ++w) {
            if (w < warp) before += sums_s[w];
            tiles_before += sums_s[w];
        }
        if (g < p.G) starts_s[g] = before + inc - own;
        __syncthreads();
    }
    if (threadIdx.x == 0) starts_s[p.G] = tiles_before;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster.sync();                                           // both CTAs' barriers exist before anything is signalled
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    const int num_tiles = starts_s[p.G];
    // outputs of a CTA's 128 weight rows: all of them, or 64 gate rows above the 64 up rows of the same outputs
    const int outputs = p.dual ? HALF_W : BLOCK_W;
    Tiles t{offsets_s, starts_s, p.n_tiles, p.tok_cap, 2 * outputs};

    if (warp == 0) {
        // ---------------------------------------------------------------- producer (both CTAs)
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
                t.seek(tile);
                const int w0 = t.group * p.w_rows + t.n0 + (int)rank * outputs, w1 = p.dual ? w0 + p.up_offset : w0 + HALF_W;
                const int row0 = t.row0 + (int)rank * (t.cols / 2);
                for (int kb = 0; kb < p.k_blocks; ++kb, ++it) {
                    lag_point();
                    const int s = it % p.stages;
                    const uint32_t round = it / p.stages;
                    if (round > 0 && !mbar_wait(smem_u32(&empty_bar[s]), (round - 1) & 1, p.error_flag, 61)) { ok = false; break; }
                    const uint32_t dst = ring + (uint32_t)s * stage_bytes;
                    const uint32_t leader_full = cluster_addr(smem_u32(&full_bar[s]), 0);
                    if (rank == 0) mbar_expect_tx(smem_u32(&full_bar[s]), 2 * stage_bytes);
                    const int k = kb * BLOCK_K;
                    tma_load_2d_pair(dst, &map_w, k, w0, leader_full);
                    tma_load_2d_pair(dst + A_TILE_BYTES / 2, &map_w, k, w1, leader_full);
                    tma_load_2d_pair(dst + A_TILE_BYTES, &map_x, k, row0, leader_full);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issue (leader only; the warp stays converged)
        if (rank == 0) {
            uint32_t it = 0, local = 0;
            bool ok = true;
            for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++local) {
                t.seek(tile);
                const uint32_t idesc = umma_idesc(t.cols);
                const uint32_t buf = local & 1, use = local >> 1;
                // both epilogues must have drained this buffer (the first use of each buffer passes at once)
                if (!mbar_wait_warp(smem_u32(&acc_empty[buf]), (use & 1) ^ 1, p.error_flag, 62)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem_base + buf * acc_cols;
                for (int kb = 0; kb < p.k_blocks; ++kb, ++it) {
                    lag_point();
                    const int s = it % p.stages;
                    if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&full_bar[s]), (it / p.stages) & 1, p.error_flag, 63))) { ok = false; break; }
                    const uint32_t a_addr = ring + (uint32_t)s * stage_bytes;
                    // descriptors of the stage; a K step of 16 elements moves the start address (16-byte units) by 2
                    const uint64_t adesc = umma_desc(a_addr), bdesc = umma_desc(a_addr + A_TILE_BYTES);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
                            umma_pair(acc, adesc + 2 * k, bdesc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                        umma_commit_pair(smem_u32(&empty_bar[s]));  // the stage is free in both CTAs once these MMAs have read it
                    }
                    __syncwarp();
                }
                if (ok && elect_one()) umma_commit_pair(smem_u32(&acc_full[buf]));
                __syncwarp();
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue (both CTAs, own 128 weight rows)
        // dual: warp `quarter` holds 32 gate rows, warp `quarter + 2` the up rows of the same outputs.  Of 32 places each of the two
        // finishes 16: it hands the other one its own values of the other 16 through shared memory (two turns of 2 KB each way, so
        // that one meeting a turn is enough).  A warp whose bounded wait ran out goes on meeting its partner, without values.
        const int quarter = warp & 3;
        const bool upper = p.dual && quarter >= 2;
        const int first_col = upper ? 16 : 0;                // the places of 32 that this warp finishes (dual)
        const uint32_t give = exchange + (uint32_t)((quarter & 1) * 2 + (upper ? 1 : 0)) * 2 * 2048 + lane * 4;
        const uint32_t take = exchange + (uint32_t)((quarter & 1) * 2 + (upper ? 0 : 1)) * 2 * 2048 + lane * 4;
        uint32_t local = 0, turn = 0;
        bool ok = true;
        for (int tile = pair; tile < num_tiles; tile += num_pairs, ++local) {
            lag_point();
            t.seek(tile);
            const uint32_t buf = local & 1, use = local >> 1;
            const int out_col = t.n0 + (int)rank * outputs + (p.dual ? quarter & 1 : quarter) * 32 + lane;
            ok = ok && mbar_wait_warp(smem_u32(&acc_full[buf]), use & 1, p.error_flag, 64);
            if (!ok && !p.dual) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t lane_addr = tmem_base + buf * acc_cols + ((uint32_t)(quarter * 32) << 16);
            for (int c = 0; c < t.rows; c += 32) {
                // lane j: the row that place c + j is written to, and its scale
                const int place = t.row0 + min(c + lane, t.rows - 1);
                const int to = p.c_rows ? p.c_rows[place] : place;
                const int scaled = p.scale_rows ? p.scale_rows[place] : place;
                const float scale = p.row_scale && scaled >= 0 ? p.row_scale[scaled] : 1.0f;       // (a negative one: a row of zeros)
                const unsigned there = __ballot_sync(0xffffffffu, to >= 0);       // (a test of each row behind its shuffle: down 127 us, so 108)
                uint32_t raw[32];
                if (ok) {
                    tmem_ld32_nowait(lane_addr + (uint32_t)c, raw);
                    tmem_wait();
                }
                if (p.dual) {
                    const uint32_t at = (turn++ & 1) * 2048;
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(give + at + j * 128), "r"(upper ? raw[j] : raw[j + 16]) : "memory");
                    asm volatile("bar.sync %0, 64;" ::"r"(1 + (quarter & 1)) : "memory");
                    float g[16], u[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float weight = __shfl_sync(0xffffffffu, scale, first_col + j);
                        uint32_t other;
                        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(other) : "r"(take + at + j * 128) : "memory");
                        const float mine = __uint_as_float(upper ? raw[j + 16] : raw[j]) * weight, theirs = __uint_as_float(other) * weight;
                        g[j] = upper ? theirs : mine;
                        u[j] = upper ? mine : theirs;
                    }
                    if (p.act > 1) gated_values<true>(g, u, __int_as_float(p.act));
                    else gated_values<false>(g, u, 0.0f);
                    const int here = ok && out_col < p.N ? t.rows - c - first_col : 0;      // places of these 16 that exist
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int row = __shfl_sync(0xffffffffu, to, first_col + j);
                        const size_t o = (size_t)row * p.ldo + out_col;
                        if (j < here && ((there >> (first_col + j)) & 1u)) {
                            if (p.out_bf16) ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(g[j]);
                            else ((float*)p.out)[o] = g[j];
                        }
                    }
                    continue;
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) {                         // (plain stores: nothing to set side by side, and no address kept for later)
                    if (c + j >= t.rows) break;                        // (uniform)
                    const int row = __shfl_sync(0xffffffffu, to, j);
                    if (out_col >= p.N || !((there >> j) & 1u)) continue;
                    if (p.out_bf16) ((__nv_bfloat16*)p.out)[(size_t)row * p.ldo + out_col] = __float2bfloat16_rn(__uint_as_float(raw[j]));
                    else ((float*)p.out)[(size_t)row * p.ldo + out_col] = __uint_as_float(raw[j]);
                }
            }
            // this warp is done reading the buffer: tell the leader's MMA warp
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_addr(smem_u32(&acc_empty[buf]), 0));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster.sync();                      // nobody leaves while the peer may still signal its barriers or read its operands
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
    }
}

// rows of A in the order of the list: out[place] = A[a_rows[place] / div], 16 bytes a thread; a negative row is one of zeros, as in
// grouped_mma.cu
__global__ void __launch_bounds__(256) gather_rows_kernel(const uint4* __restrict__ a, long long lda, const int* __restrict__ a_rows, int div,
                                                          const int* __restrict__ offsets, int G, uint4* __restrict__ out, int rows, int pieces) {
    pdl_prologue();
    const int listed = min(offsets[G], rows);                // places that belong to a group
    const long long total = (long long)listed * pieces;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
        const int place = (int)(i / pieces), piece = (int)(i % pieces);
        const int row = a_rows[place] / div;
        out[i] = row >= 0 ? a[(size_t)row * lda + piece] : make_uint4(0u, 0u, 0u, 0u);
    }
}

// --------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &res) == cudaSuccess &&
            res == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)sym;
    }
    return fn;
}

int make_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(MLB_CUDA_ERROR, "grouped_pair: cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)BLOCK_K, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(MLB_CUDA_ERROR, "grouped_pair: cuTensorMapEncodeTiled failed with %d", (int)r);
    return MLB_OK;
}

}  // namespace

// C rows [places, ldo] (fp32 or bf16) from A [places, K] bf16 (sorted by group, pitch lda) and W [G, w_rows, K] bf16.  dual: W[g] holds
// N gate rows and, up_offset rows further down, N up rows; act as in gated_value.  K and the pitches are multiples of 8 elements, the
// bases 16-byte aligned.  tok_cap: rows of a tile at most (32, or 64 .. 256 in steps of 64).
MLB_EXPORT int mlb_grouped_pair(const void* a, long long lda, const void* w, void* out, long long ldo, const int* offsets, const int* c_rows,
                                const float* row_scale, const int* scale_rows, int out_bf16, int dual, int act, int up_offset, int M, int N, int K,
                                int G, int w_rows, int tok_cap, int sm_count, int* error_flag, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || G <= 0 || w_rows < N) return fail(MLB_INVALID_ARGUMENT, "grouped_pair: bad sizes M=%d N=%d K=%d G=%d", M, N, K, G);
    if (G > MAX_GROUPS) return fail(MLB_UNSUPPORTED_SIZE, "grouped_pair: %d groups are more than %d", G, MAX_GROUPS);
    if (K % 8 != 0 || lda % 8 != 0 || lda < K || ((uintptr_t)a & 15) || ((uintptr_t)w & 15))
        return fail(MLB_UNSUPPORTED_SIZE, "grouped_pair: K=%d and the pitch %lld must be multiples of 8, the operands 16-byte aligned", K, lda);
    if (dual && (up_offset < 0 || up_offset + N > w_rows)) return fail(MLB_INVALID_ARGUMENT, "grouped_pair: up rows outside the weight");
    if (act < 0 || act == 1) return fail(MLB_INVALID_ARGUMENT, "grouped_pair: unknown activation %d", act);
    if (row_scale && !dual) return fail(MLB_INVALID_ARGUMENT, "grouped_pair: a factor per row goes with the two-block product");
    if (tok_cap != 32 && (tok_cap < 64 || tok_cap > 256 || tok_cap % 64 != 0)) return fail(MLB_INVALID_ARGUMENT, "grouped_pair: tiles of %d rows", tok_cap);
    if ((long long)G * w_rows >= (1ll << 31)) return fail(MLB_UNSUPPORTED_SIZE, "grouped_pair: too many weight rows");
    if (!offsets || sm_count < 2 || sm_count % 2 != 0) return fail(MLB_INVALID_ARGUMENT, "grouped_pair: bad arguments");
    if (M == 0) return MLB_OK;
    GroupedParams p{};
    p.out = out; p.offsets = offsets; p.c_rows = c_rows; p.row_scale = row_scale; p.scale_rows = scale_rows; p.error_flag = error_flag;
    p.ldo = ldo; p.M = M; p.N = N; p.G = G; p.w_rows = w_rows; p.up_offset = up_offset; p.tok_cap = tok_cap;
    p.k_blocks = (K + BLOCK_K - 1) / BLOCK_K;
    p.n_tiles = (N + (dual ? PAIR_W / 2 : PAIR_W) - 1) / (dual ? PAIR_W / 2 : PAIR_W);
    p.out_bf16 = out_bf16; p.dual = dual; p.act = act;
    const int stage_bytes = A_TILE_BYTES + (tok_cap / 2) * BLOCK_K * 2, exchange_bytes = dual ? 16 * 1024 : 0;
    p.stages = (208 * 1024 - exchange_bytes) / stage_bytes;
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    const size_t smem = (size_t)p.stages * stage_bytes + exchange_bytes + 1024;

    CUtensorMap map_w, map_x;
    int status = make_map(&map_w, w, (long long)G * w_rows, K, K, HALF_W);
    if (status != MLB_OK) return status;
    status = make_map(&map_x, a, M, K, lda, tok_cap / 2);
    if (status != MLB_OK) return status;
    static bool configured[MAX_DEVICES] = {false};            // the attribute belongs to the device
    const int d = device_index();
    if (!configured[d]) {
        cudaError_t e = cudaFuncSetAttribute(grouped_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(212 * 1024));
        if (e != cudaSuccess) return fail(MLB_CUDA_ERROR, "grouped_pair: cannot reserve shared memory: %s", cudaGetErrorString(e));
        configured[d] = true;
    }
    // no more pairs than there can be tiles: a group has at most one partly filled row tile
    const long long most = (long long)p.n_tiles * (M / tok_cap + (M < G ? M : G));
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)(2 * most < sm_count ? 2 * most : sm_count));
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = 2;
    attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // (behind the small kernels of a decode step the set-up is hidden)
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&config, grouped_pair_kernel, map_w, map_x, p);
    return check_launch("grouped_pair");
}

// out[place] = a[a_rows[place] / div] for the places in front of offsets[G]; K bf16 a row, K and lda multiples of 8, 16-byte aligned
MLB_EXPORT int mlb_gather_rows(const void* a, long long lda, const int* a_rows, int div, const int* offsets, int G, void* out, int rows, int K,
                               cudaStream_t stream) {
    if (rows < 0 || K <= 0 || K % 8 != 0 || lda % 8 != 0 || div <= 0 || G < 0 || !a_rows || !offsets || ((uintptr_t)a & 15) || ((uintptr_t)out & 15))
        return fail(MLB_INVALID_ARGUMENT, "gather_rows: bad arguments");
    if (rows == 0) return MLB_OK;
    const int pieces = K / 8;
    const long long blocks = ((long long)rows * pieces + 255) / 256, most = 16ll * sm_count();
    launch_kernel(gather_rows_kernel, (unsigned)(blocks < most ? blocks : most), 256, 0, stream, (const uint4*)a, lda / 8, a_rows, div, offsets, G,
                  (uint4*)out, rows, pieces);
    return check_launch("gather_rows");
}
