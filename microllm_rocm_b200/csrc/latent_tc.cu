// Latent attention of prompts on the fifth-generation tensor cores (see latent.cu): all heads read the same cache rows, a query row is one
// (token, head) pair, q [T*H, R + DR], out [T*H, R].  Compiled per model: -DLAT_R (latent width) -DLAT_DR (rotated width).
//
// THE BITS of latent_mma.cu's unsplit form: a score is four partial sums over every fourth 16-wide step of the contraction, added in order; keys go
// by in tiles of 32, after each of which a row's maximum, sum and accumulator move on; exponentials, the sum's order and the roundings
// of weights and result are the same.  tcgen05.mma adds a chain of products as mma.sync does (grouped_tc2.cu rests on it too).
//
// A CTA owns 128 consecutive query rows of one sequence and HALF of the output columns: 128 x 512 fp32 would fill tensor memory and leave no
// room for scores.  Both halves make the scores.  A tile's row is R / 64 + DR / 64 spans of 64 columns; the spans of this half's
// columns serve both products (as K, rows times contraction, and as V, the same bytes read contraction first) and stay in one of three
// buffers from the scores of a tile to its P V, the others stream through a ring, all in the order of the contraction.
//     warps 0, 6, 7  TMA, a lane a box of a span: one lane for all took longer than the tile (copies of 2 KB, about 110 cycles each)
//     warp 1         tcgen05.mma: the four partial scores of tile j + 1 while the softmax warps work on tile j, then P V of tile j
//     warps 2-5      softmax, one thread a row: four partial scores out of tensor memory, weights back into it as the A operand of P V, the
//                    accumulator in tensor memory rescaled where any row of the warp has a new maximum
// The last three spans of the queries lie in tensor memory (an A operand may), which leaves shared memory for a ring of four tiles.
//
// 2,048 tokens of 16 heads, 512 + 64 wide: 242 us, latent_mma.cu 427; 512 tokens behind 2,000 152 and 356.  What bounds it is a tile's chain:
// nine dependent steps of four MMAs of 32 columns (the order of the sums asks for them; each takes its 4 KB of queries from shared
// memory), the scores' way through the softmax, and the accumulator's through registers where a maximum grew.  Measured and no faster:
// two tiles' scores in tensor memory with weights in their place (251 us: the ring was two tiles short), two threads a row (264).
//
// Every wait on an mbarrier is bounded; when a bound is hit the error flag is raised, the CTA waits (bounded) for the copies and products it
// still has in flight, frees its tensor memory and returns.
#include "common.cuh"

#include <cuda.h>

#if !defined(LAT_R) || !defined(LAT_DR)
#error "compile with -DLAT_R and -DLAT_DR"
#endif

using namespace mlb;

MLB_DEFINE_LAST_ERROR()

namespace {

constexpr int R = LAT_R, DR = LAT_DR, DK = R + DR;
static_assert(R % 128 == 0 && R <= 512 && DR % 64 == 0 && DR >= 64, "a latent of two halves of whole spans, a rotated part of whole spans");
constexpr int BM = 128;                                      // query rows per CTA (MMA M)
constexpr int ROW_BYTES = 128;                               // one swizzle span: 64 bf16
constexpr int KEYS = 32;                                     // keys per tile
constexpr int PARTS = 4;                                     // partial scores: the four 16-wide steps of a span
constexpr int HALF = R / 2;                                  // output columns of a CTA
constexpr int SPANS = DK / 64, OWN = HALF / 64, OTHERS = SPANS - OWN;
constexpr int Q_SPAN_BYTES = BM * ROW_BYTES, K_SPAN_BYTES = KEYS * ROW_BYTES;
constexpr int Q_TMEM = 3, Q_SMEM = SPANS - Q_TMEM;      // spans of the queries in tensor memory (an A operand may lie there) and in shared memory
constexpr int Q_BYTES = Q_SMEM * Q_SPAN_BYTES, V_BYTES = OWN * K_SPAN_BYTES, V_BUFS = 3;
constexpr int SLOTS_FIT = (226 * 1024 - 1024 - Q_BYTES - V_BUFS * V_BYTES) / K_SPAN_BYTES;
constexpr int SLOTS = SLOTS_FIT > 4 * OTHERS ? 4 * OTHERS : SLOTS_FIT;
static_assert(SLOTS >= OTHERS && SLOTS % OTHERS == 0, "the ring holds whole tiles' other spans");
constexpr int SMEM_BYTES = Q_BYTES + V_BUFS * V_BYTES + SLOTS * K_SPAN_BYTES + 1024;
// A CTA takes all of its multiprocessor's tensor memory ahead of its wait for the kernel in front.  Were there room for another CTA, one of the launch
// behind could get the memory that one of this launch is still to get, and wait for this launch: neither would end.
static_assert(Q_SMEM > 0 && SMEM_BYTES > 200 * 1024, "a CTA has its multiprocessor to itself");
constexpr int THREADS = 256;
constexpr int PRODUCERS = 3, EACH = (SPANS + PRODUCERS - 1) / PRODUCERS;      // warps that copy, spans of each
// Tensor memory: O [0, HALF), a tile's partial scores, two tiles' weights, the last spans of the queries
constexpr int TMEM_COLS = 512, S_COL = 256, P_COL = S_COL + PARTS * KEYS, Q_COL = P_COL + KEYS;
static_assert(HALF <= S_COL && Q_COL + 32 * Q_TMEM <= TMEM_COLS, "room in tensor memory");
constexpr int MAX_PAGES_PER_TILE = 4;
constexpr int PARTLY = BM;                   // keys that only some of 128 rows see: fewer than 128 at either end of a window
#ifndef MLB_SPIN_LIMIT                       // (the tests build objects whose waits run out at once)
#define MLB_SPIN_LIMIT (1 << 21)
#endif
constexpr int SPIN_LIMIT = MLB_SPIN_LIMIT;   // polls of up to 2 us each
constexpr int DRAIN_LIMIT = 1 << 14;         // the same for what is in flight when a wait has run out: microseconds, or never

struct LatentTcParams {
    const __nv_bfloat16* q;         // [rows, DK]
    const __nv_bfloat16* pages;     // [num_pages, page_size, DK]
    __nv_bfloat16* out;             // [rows, R]
    const int* seq_starts;          // [A+1]
    const int* seq_pos0;            // [A]
    const int* block_table;         // [A, max_blocks]
    const int* work;                // [num_work, 2]: sequence, first of 128 of its query rows
    int heads, max_blocks, num_pages, page_size, box_rows, window;
    float scale;
    const float* sink;              // [H] or null: exp(sink[head]) joins the head's denominator (no key, no value)
    int* error_flag;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(2000u) : "memory");
    return ok != 0;
}
// false when the bound was hit (the caller gives up and the flag tells the host)
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* error_flag, int code) {
    for (int i = 0; i < SPIN_LIMIT; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    if (error_flag) atomicCAS(error_flag, 0, code);          // the first failure is the one worth reporting
    return false;
}
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < DRAIN_LIMIT; ++i)
        if (mbar_try_wait(bar, parity)) return;
}
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
// shared-memory operands, 128-byte swizzle (see attention_tc.cu): K-major, and MN-major with the next 64 columns `lead_bytes` further on
__device__ __forceinline__ uint64_t desc_mn_major(uint32_t addr, uint32_t lead_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lead_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ uint64_t desc_k_major(uint32_t addr) { return desc_mn_major(addr, 16); }
// kind::f16 instruction descriptor: fp32 accumulator, bf16 A (K-major) and B
__device__ __forceinline__ uint32_t idesc(int n, bool b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn_major ? (1u << 16) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(a), "l"(b), "r"(id), "r"(accumulate) : "memory");
}
// the same with the A operand in tensor memory (lane = row, a 32-bit column = two neighbouring bf16 of the contraction)
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t id, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(b), "r"(id), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
#define MLB_LIST32(x) x(0), x(1), x(2), x(3), x(4), x(5), x(6), x(7), x(8), x(9), x(10), x(11), x(12), x(13), x(14), x(15), x(16), x(17), x(18), x(19), x(20), \
                      x(21), x(22), x(23), x(24), x(25), x(26), x(27), x(28), x(29), x(30), x(31)
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t* r) {
#define MLB_OUT(i) "=r"(r[i])
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : MLB_LIST32(MLB_OUT) : "r"(addr));
#undef MLB_OUT
}
__device__ __forceinline__ void tmem_st32(uint32_t addr, const uint32_t* r) {
#define MLB_IN(i) "r"(r[i])
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(addr), MLB_LIST32(MLB_IN) : "memory");
#undef MLB_IN
}
#undef MLB_LIST32
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// two fp32 values in one instruction, each rounded as always
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(uint32_t lo, uint32_t hi) { return ((f32x2)hi << 32) | lo; }
__device__ __forceinline__ float low(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float high(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}

__global__ void __launch_bounds__(THREADS, 1)
latent_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv, LatentTcParams p) {
    pdl_launch_dependents();
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long q_full, v_full[V_BUFS], v_empty[V_BUFS], slot_full[SLOTS], slot_empty[SLOTS], q_there, s_full, s_empty, p_full[2], pv_done[2],
        looked, finished, stopped;
    __shared__ uint32_t tmem_base_s;
    __shared__ unsigned bad_s[2 * PARTLY / 32];            // keys that some rows see and others do not, whose values are not finite

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t q_s = (smem_u32(smem_dyn) + 1023u) & ~1023u;      // the swizzle pattern wants 1024-byte alignment
    const uint32_t v_s = q_s + Q_BYTES, ring_s = v_s + V_BUFS * V_BYTES;

    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&q_full), 1);
        for (int s = 0; s < SLOTS; ++s) {
            mbar_init(smem_u32(&slot_full[s]), 1);
            mbar_init(smem_u32(&slot_empty[s]), 1);
        }
        for (int s = 0; s < V_BUFS; ++s) {
            mbar_init(smem_u32(&v_full[s]), 1);
            mbar_init(smem_u32(&v_empty[s]), 1);
        }
        mbar_init(smem_u32(&q_there), 4);                 // one arrival per softmax warp, here and below
        mbar_init(smem_u32(&s_full), 1);
        mbar_init(smem_u32(&s_empty), 4);
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&p_full[s]), 4);           // one barrier per buffer: a warp may be a tile ahead of another
            mbar_init(smem_u32(&pv_done[s]), 1);          // P V of the even tiles, and of the odd ones
        }
        mbar_init(smem_u32(&looked), 4);                  // the softmax warps, about values that are not finite
        mbar_init(smem_u32(&finished), 1);                // every product is done,
        mbar_init(smem_u32(&stopped), 1);                 // or those issued before a wait ran out are
        for (int i = 0; i < 2 * PARTLY / 32; ++i) bad_s[i] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_s)), "r"((uint32_t)TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // ---- the tile's geometry (uniform over the CTA; the lists are older than the step's kernels)
    const int half = blockIdx.x, item = blockIdx.y;
    const int seq = p.work[2 * item], row_first = p.work[2 * item + 1];
    const int start = p.seq_starts[seq], pos0 = p.seq_pos0[seq];
    const int rows = min(BM, (p.seq_starts[seq + 1] - start) * p.heads - row_first);
    const size_t row0 = (size_t)start * p.heads + row_first;          // among all query rows
    const int qpos_first = pos0 + row_first / p.heads, qpos_last = pos0 + (row_first + rows - 1) / p.heads;
    const int lo = first_visible_key(qpos_first, p.window, 0);
    const int tile_first = lo / KEYS, n_tiles = qpos_last / KEYS - tile_first + 1;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    pdl_wait();                  // queries and this step's cache rows were written by the kernels before
    const int own_first = half * OWN;        // this half's spans: own_first .. own_first + OWN - 1

    if (warp == 0 || warp >= 6) {
        // ------------------------------------------------------------------ producers: a lane a box of a span, so that a tile's waits, announcements and
        // copies go side by side (one behind another in one lane they took longer than the tile; in one warp its 18 copies out of pages of 16 did)
        const int producer = warp == 0 ? 0 : warp - 5, boxes = KEYS / p.box_rows;          // (boxes: copies of a span)
        const int span = producer + PRODUCERS * (lane % EACH), box = lane / EACH;
        const bool own = span >= own_first && span < own_first + OWN, works = span < SPANS && box < boxes;
        if (warp == 0) {
            if (lane == 0) mbar_expect_tx(smem_u32(&q_full), Q_BYTES);
            __syncwarp();
            if (lane < Q_SMEM) tma_load_2d(q_s + lane * Q_SPAN_BYTES, &map_q, lane * 64, (int)row0, smem_u32(&q_full));
        }
        const int* table = p.block_table + (size_t)seq * p.max_blocks;
        auto lookup = [&](int j) {                        // the page that holds this lane's box of tile j
            const int block = ((tile_first + j) * KEYS + box * p.box_rows) / p.page_size;
            return works && j < n_tiles && block < p.max_blocks ? __ldg(table + block) : -1;
        };
        auto full_of = [&](int j, int item) { return own ? smem_u32(&v_full[j % V_BUFS]) : smem_u32(&slot_full[item % SLOTS]); };
        const int item0 = span - (span >= own_first ? OWN : 0);              // this lane's span among the ring's items
        int loaded = 0, page_next = lookup(0);            // tiles issued
        for (int j = 0; j < n_tiles; ++j) {
            lag_point();
            const int item = item0 + j * OTHERS, slot = item % SLOTS, buf = j % V_BUFS;
            const uint32_t empty = own ? smem_u32(&v_empty[buf]) : smem_u32(&slot_empty[slot]), full = full_of(j, item);
            const bool ok = !works || (own ? j < V_BUFS : item < SLOTS) || mbar_wait(empty, (own ? j / V_BUFS - 1 : item / SLOTS - 1) & 1, p.error_flag, own ? 62 : 61);
            if (!__all_sync(0xffffffffu, ok)) break;
            // (the other producers' copies of the same buffer may land in front of this: the phase waits for it)
            if (works && box == 0 && (!own || span == own_first)) mbar_expect_tx(full, own ? V_BYTES : K_SPAN_BYTES);
            int page = page_next;
            page_next = lookup(j + 1);
            const int first_key = (tile_first + j) * KEYS + box * p.box_rows;
            if (page < 0 || page >= p.num_pages) {
                // a page that holds a key some row must see has to exist; the others are masked
                if (works && first_key <= qpos_last && first_key + p.box_rows - 1 >= lo && p.error_flag) atomicExch(p.error_flag, 2);
                page = 0;
            }
            const uint32_t dst = own ? v_s + buf * V_BYTES + (span - own_first) * K_SPAN_BYTES : ring_s + slot * K_SPAN_BYTES;
            __syncwarp();
            if (works) tma_load_2d(dst + box * p.box_rows * ROW_BYTES, &map_kv, span * 64, page * p.page_size + first_key % p.page_size, full);
            loaded = j + 1;
        }
        // Products that are done have had their copies.  Where they never are, or a wait above ran out, the copies in flight get a bounded chance to
        // land before the CTA's memory goes away: of each buffer the last one (behind it the parity of an earlier one would say the opposite).
        if (works && !(loaded == n_tiles && mbar_wait(smem_u32(&finished), 0, nullptr, 0))) {
            if (warp == 0 && lane == 0) mbar_drain(smem_u32(&q_full), 0);
            for (int j = max(0, loaded - (own ? V_BUFS : SLOTS / OTHERS)); j < loaded; ++j)
                mbar_drain(full_of(j, item0 + j * OTHERS), (own ? j / V_BUFS : (item0 + j * OTHERS) / SLOTS) & 1);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issue: one lane, the descriptors made once (a step of 16 bytes
        // is one of their units; put together for each of a tile's 38 instructions they were what bounded it)
        if (elect_one()) {
            const uint32_t idesc_qk = idesc(KEYS, false), idesc_pv = idesc(HALF, true);
            const uint64_t q_desc = desc_k_major(q_s), ring_desc = desc_k_major(ring_s), k_desc = desc_k_major(v_s), v_desc = desc_mn_major(v_s, K_SPAN_BYTES);
            auto wait = [&](unsigned long long* bar, uint32_t parity, int code) { return mbar_wait(smem_u32(bar), parity, p.error_flag, code); };
            int slot = 0, buf_qk = 0, buf_pv = 0;              // ring items are consumed in the order they were loaded
            uint32_t slot_parity = 0, buf_parity = 0;
            auto issue_qk = [&] {
#pragma unroll
                for (int span = 0; span < SPANS; ++span) {
                    const bool own = span >= own_first && span < own_first + OWN;
                    if (span == own_first && !wait(&v_full[buf_qk], buf_parity, 65)) return false;
                    if (!own && !wait(&slot_full[slot], slot_parity, 64)) return false;
                    const uint64_t k = own ? k_desc + (uint64_t)(buf_qk * (V_BYTES / 16) + (span - own_first) * (K_SPAN_BYTES / 16))
                                           : ring_desc + (uint64_t)(slot * (K_SPAN_BYTES / 16));
#pragma unroll
                    for (int w = 0; w < PARTS; ++w)          // a span's four 16-wide steps, each to its own partial scores
                        if (span < Q_SMEM)
                            umma(tmem_base + (uint32_t)(S_COL + w * KEYS), q_desc + (uint64_t)(span * (Q_SPAN_BYTES / 16) + w * 2), k + (uint64_t)(w * 2), idesc_qk, span > 0 ? 1u : 0u);
                        else
                            umma_ts(tmem_base + (uint32_t)(S_COL + w * KEYS), tmem_base + (uint32_t)(Q_COL + (span - Q_SMEM) * 32 + w * 8), k + (uint64_t)(w * 2), idesc_qk, 1u);
                    if (own) continue;
                    umma_commit(smem_u32(&slot_empty[slot]));
                    if (++slot == SLOTS) { slot = 0; slot_parity ^= 1; }
                }
                umma_commit(smem_u32(&s_full));
                if (++buf_qk == V_BUFS) { buf_qk = 0; buf_parity ^= 1; }
                return true;
            };
            bool ok = wait(&q_full, 0, 63) && wait(&q_there, 0, 70);
            tc_fence_after();
            ok = ok && issue_qk();
            for (int j = 0; j < n_tiles && ok; ++j) {
                lag_point();
                if (j + 1 < n_tiles) {
                    ok = wait(&s_empty, j & 1, 67);
                    if (!ok) break;
                    tc_fence_after();                      // the softmax warps have read tile j's scores
                    ok = issue_qk();
                    if (!ok) break;
                }
                ok = wait(&p_full[j & 1], (j >> 1) & 1, 66);
                if (!ok) break;
                tc_fence_after();                          // P and the rescaled accumulator were written by the softmax warps
#pragma unroll
                for (int ks = 0; ks < KEYS / 16; ++ks)        // 16 keys = 8 columns of P; the keys are here since this tile's scores
                    umma_ts(tmem_base, tmem_base + (uint32_t)(P_COL + (j & 1) * (KEYS / 2) + ks * 8),
                            v_desc + (uint64_t)(buf_pv * (V_BYTES / 16) + ks * ROW_BYTES), idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
                umma_commit(smem_u32(&v_empty[buf_pv]));
                umma_commit(smem_u32(&pv_done[j & 1]));
                if (++buf_pv == V_BUFS) buf_pv = 0;
            }
            umma_commit(smem_u32(ok ? &finished : &stopped));
            if (!ok) mbar_drain(smem_u32(&stopped), 0);      // products in flight read shared and write tensor memory
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ softmax, one thread per row
        const int quarter = warp & 3;                     // the tensor-memory lanes this warp may touch
        const int r = quarter * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const bool exists = r < rows;
        const int qpos = exists ? pos0 + (row_first + r) / p.heads : -1;             // -1: sees nothing
        const int lo_r = first_visible_key(qpos, p.window, 0), lo_last = first_visible_key(qpos_last, p.window, 0);
        const bool own_sink = p.sink != nullptr && exists;
        float m_run = own_sink ? p.sink[(row_first + r) % p.heads] : -INFINITY, l_run = own_sink ? 1.0f : 0.0f;
        const f32x2 scale2 = pair(__float_as_uint(p.scale), __float_as_uint(p.scale));
        int looks = 0;
        bool ok = true;
        // the tensor-memory instructions below are warp-wide: a wait gives up for the whole warp or not at all
        auto wait_all = [&](unsigned long long* bar, uint32_t parity, int code) {
            return __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity, p.error_flag, code)) != 0;
        };
        // the last spans of the thread's query row, to tensor memory
        {
            const uint4* q = reinterpret_cast<const uint4*>(p.q + (row0 + r) * DK + Q_SMEM * 64);
#pragma unroll
            for (int span = 0; span < Q_TMEM; ++span) {
                uint32_t v[32];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint4 u = exists ? q[span * 8 + i] : make_uint4(0u, 0u, 0u, 0u);
                    v[4 * i] = u.x; v[4 * i + 1] = u.y; v[4 * i + 2] = u.z; v[4 * i + 3] = u.w;
                }
                tmem_st32(lane_base + (uint32_t)(Q_COL + span * 32), v);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&q_there));
        }
        for (int j = 0; j < n_tiles; ++j) {
            const int buf = j & 1;
            lag_point();
            ok = wait_all(&s_full, j & 1, 68);
            if (!ok) break;
            tc_fence_after();
            float sc[KEYS];
            {
                uint32_t part[PARTS][KEYS];
#pragma unroll
                for (int w = 0; w < PARTS; ++w) tmem_ld32(lane_base + (uint32_t)(S_COL + w * KEYS), part[w]);
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_empty));
#pragma unroll
                for (int c = 0; c < KEYS; c += 2) {
                    f32x2 v = pair(part[0][c], part[0][c + 1]);
#pragma unroll
                    for (int w = 1; w < PARTS; ++w) v = add2(v, pair(part[w][c], part[w][c + 1]));
                    sc[c] = low(v); sc[c + 1] = high(v);
                }
            }
            const int kbase = (tile_first + j) * KEYS;
            if (kbase + KEYS - 1 > qpos_first || kbase < lo_last || rows < BM) {        // the tile touches the causal edge or the window's
#pragma unroll
                for (int c = 0; c < KEYS; ++c) sc[c] = kbase + c <= qpos && kbase + c >= lo_r ? __fmul_rn(sc[c], p.scale) : -INFINITY;
            } else {
#pragma unroll
                for (int c = 0; c < KEYS; c += 2) {           // (a product of its own, as behind the mask: not drawn into the exponent's difference)
                    const f32x2 v = mul2(pair(__float_as_uint(sc[c]), __float_as_uint(sc[c + 1])), scale2);
                    sc[c] = low(v); sc[c + 1] = high(v);
                }
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < KEYS; c += 2) mx[(c >> 1) & 3] = fmaxf(fmaxf(mx[(c >> 1) & 3], sc[c]), sc[c + 1]);
            const float m_new = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), m_run);
            const float corr = m_run == -INFINITY ? 0.0f : expf(m_run - m_new);      // m_new >= m_run; both -inf: nothing seen yet
            m_run = m_new;
            // a masked score is -inf, whose exponential is 0; where nothing has been seen yet the maximum is too, and 0 stands in for it
            const f32x2 less2 = pair(__float_as_uint(m_new == -INFINITY ? -0.0f : -m_new), __float_as_uint(m_new == -INFINITY ? -0.0f : -m_new));
            uint32_t packed[KEYS / 2];
            float eight[4];                               // the sums of the four eighths of the keys, as latent_mma.cu's warps make them
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                float two[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int c = w * 8 + 2 * t;
                    const f32x2 x = add2(pair(__float_as_uint(sc[c]), __float_as_uint(sc[c + 1])), less2);
                    const float p0 = expf(low(x)), p1 = expf(high(x));
                    packed[c / 2] = pack_bf16(p0, p1);
                    two[t] = p0 + p1;
                }
                eight[w] = (two[0] + two[1]) + (two[2] + two[3]);
            }
            l_run = l_run * corr + ((eight[0] + eight[1]) + (eight[2] + eight[3]));
            // the accumulator moves on with the maximum (times 1 where a row's stays, which changes nothing)
            if (j > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {
                ok = wait_all(&pv_done[(j - 1) & 1], ((j - 1) >> 1) & 1, 69);      // O holds tiles 0..j-1
                if (!ok) break;
                tc_fence_after();
                const f32x2 corr2 = pair(__float_as_uint(corr), __float_as_uint(corr));
#pragma unroll 1
                for (int c = 0; c < HALF / 64; ++c) {
                    uint32_t o[2][32];
                    tmem_ld32(lane_base + (uint32_t)(c * 64), o[0]);
                    tmem_ld32(lane_base + (uint32_t)(c * 64 + 32), o[1]);
                    tmem_wait_ld();
#pragma unroll
                    for (int k = 0; k < 2; ++k)
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const f32x2 v = mul2(pair(o[k][i], o[k][i + 1]), corr2);
                            o[k][i] = __float_as_uint(low(v)); o[k][i + 1] = __float_as_uint(high(v));
                        }
                    tmem_st32(lane_base + (uint32_t)(c * 64), o[0]);
                    tmem_st32(lane_base + (uint32_t)(c * 64 + 32), o[1]);
                }
            }
            if (j > 1) {                                  // this buffer of weights is free once P V of the tile before the last is done
                ok = wait_all(&pv_done[buf], ((j - 2) >> 1) & 1, 73);
                if (!ok) break;
            }
            tmem_st16(lane_base + (uint32_t)(P_COL + buf * (KEYS / 2)), packed);
            // A key that a row does not see has P = 0 there, but 0 * V is not 0 where V is not finite: the V rows of keys that no row of the tile
            // sees (whatever an unused slot of a page holds) are cleared before the tensor core reads them, and so are rows that
            // some of the tile's rows see when they hold such values, which then reach the rows that do see them at the end.
            // (The tile's scores have been made: nobody else reads its spans.)
            const int before = max(0, min(KEYS, lo - kbase)), keep_to = min(KEYS, qpos_last + 1 - kbase);
            const int left_to = max(before, min(KEYS, lo_last - kbase)), right_from = min(keep_to, max(left_to, qpos_first + 1 - kbase));
            if (left_to > 0 || right_from < KEYS) {
                const uint32_t vb = v_s + (j % V_BUFS) * V_BYTES;
                auto piece_at = [&](int i, int& key) {            // the i-th 16 bytes of the keys in front of left_to and from right_from on
                    const int n = i / (OWN * 8), rest = i % (OWN * 8);
                    key = n < left_to ? n : right_from + (n - left_to);
                    return vb + (rest / 8) * K_SPAN_BYTES + key * ROW_BYTES + (rest % 8) * 16;
                };
                // bit of a key that only some rows see: those of the window's start, then those of the causal edge
                auto bit_of = [&](int key) { return kbase + key < lo_last ? kbase + key - lo : PARTLY + kbase + key - qpos_first; };
                const int pieces = (left_to + KEYS - right_from) * OWN * 8;
                for (int i = r; i < pieces; i += BM) {
                    int key;
                    const uint32_t addr = piece_at(i, key);
                    if (key < before || key >= keep_to) {
                        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(0u) : "memory");
                        continue;
                    }
                    uint32_t v[4];
                    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
                    bool bad = false;
#pragma unroll
                    for (int k = 0; k < 4; ++k) bad |= (v[k] & 0x7f80u) == 0x7f80u || (v[k] & 0x7f800000u) == 0x7f800000u;
                    if (bad) atomicOr(&bad_s[bit_of(key) >> 5], 1u << (bit_of(key) & 31));
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&looked));        // the four softmax warps meet
                ok = wait_all(&looked, looks++ & 1, 72);
                if (!ok) break;
                for (int i = r; i < pieces; i += BM) {
                    int key;
                    const uint32_t addr = piece_at(i, key);
                    if (key >= before && key < keep_to && (bad_s[bit_of(key) >> 5] >> (bit_of(key) & 31) & 1u))
                        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(0u) : "memory");
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // for the tensor core
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&p_full[buf]));
        }
        if (ok && n_tiles > 0) ok = wait_all(&pv_done[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1, 71);
        if (ok && n_tiles > 0) {
            tc_fence_after();
            const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
            __nv_bfloat16* const out = p.out + (row0 + r) * R + half * HALF;
            bool any_bad = false;
            for (int i = 0; i < 2 * PARTLY / 32; ++i) any_bad |= bad_s[i] != 0u;
#pragma unroll 1
            for (int c = 0; c < HALF / 32; ++c) {
                uint32_t o[32];
                tmem_ld32(lane_base + (uint32_t)(c * 32), o);
                tmem_wait_ld();
                if (any_bad && exists) {                          // values that are not finite, of keys that this row sees
                    for (int bit = 0; bit < 2 * PARTLY; ++bit) {
                        const int key = bit < PARTLY ? lo + bit : qpos_first + bit - PARTLY;
                        if (!(bad_s[bit >> 5] >> (bit & 31) & 1u) || !key_visible(key, qpos, lo_r, 0)) continue;
                        const int page = p.block_table[(size_t)seq * p.max_blocks + key / p.page_size];
                        if (page < 0 || page >= p.num_pages) continue;
                        const __nv_bfloat16* v = p.pages + ((size_t)page * p.page_size + key % p.page_size) * DK + half * HALF + c * 32;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (!isfinite(__bfloat162float(v[i]))) o[i] = 0x7fc00000u;
                    }
                }
                if (exists) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        auto two = [&](int k) { return pack_bf16(__uint_as_float(o[k]) * inv, __uint_as_float(o[k + 1]) * inv); };
                        *reinterpret_cast<uint4*>(out + c * 32 + i) = make_uint4(two(i), two(i + 2), two(i + 4), two(i + 6));
                    }
                }
            }
        }
        if (!ok) tmem_wait_st();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
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

// rows x DK bf16, row-major; box = box_rows x 64 columns, 128-byte swizzle, rows outside the matrix read as zero
int make_map(CUtensorMap* map, const void* base_ptr, long long rows, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(MLB_CUDA_ERROR, "latent_tc: cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[2] = {(cuuint64_t)DK, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)DK * 2};
    cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base_ptr), dims, strides, box, elem,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(MLB_CUDA_ERROR, "latent_tc: cuTensorMapEncodeTiled failed with %d", (int)r);
    return MLB_OK;
}

}  // namespace

MLB_EXPORT int mlb_latent_tc_rows_per_tile() { return BM; }

// q [total_rows, R + DR], pages [num_pages, page_size, R + DR], out [total_rows, R] bf16, total_rows = tokens * heads; work: num_work pairs
// (sequence, first of 128 of its query rows), two CTAs each.
MLB_EXPORT int mlb_latent_attention_tc(const void* q, const void* pages, void* out, const float* sink, const int* seq_starts, const int* seq_pos0,
                                       const int* block_table, const int* work, int num_work, int max_blocks, int num_pages, int page_size,
                                       int heads, int window, int total_rows, float scale, int* error_flag, cudaStream_t stream) {
    if (heads <= 0 || window < 0 || num_work < 0 || total_rows < 0 || max_blocks <= 0 || num_pages <= 0)
        return fail(MLB_INVALID_ARGUMENT, "latent_attention_tc: bad sizes");
    if (page_size < 8 || page_size % 8 != 0 || (KEYS % page_size != 0 && page_size % KEYS != 0))
        return fail(MLB_UNSUPPORTED_SIZE, "latent_attention_tc: page_size %d must be a multiple of 8 that divides %d or is a multiple of it", page_size, KEYS);
    if (((uintptr_t)q | (uintptr_t)pages | (uintptr_t)out) & 15) return fail(MLB_INVALID_ARGUMENT, "latent_attention_tc: operands must be 16-byte aligned");
    if ((long long)num_pages * page_size >= (1ll << 31)) return fail(MLB_UNSUPPORTED_SIZE, "latent_attention_tc: the cache has too many rows");
    if (num_work > 65535) return fail(MLB_UNSUPPORTED_SIZE, "latent_attention_tc: too many row tiles (%d)", num_work);
    if (num_work == 0 || total_rows == 0) return MLB_OK;
    const int box_rows = page_size < KEYS ? page_size : KEYS;
    static_assert(KEYS / 8 <= MAX_PAGES_PER_TILE, "a lane a page");
    CUtensorMap map_q, map_kv;
    int status = make_map(&map_q, q, total_rows, BM);
    if (status == MLB_OK) status = make_map(&map_kv, pages, (long long)num_pages * page_size, box_rows);
    if (status != MLB_OK) return status;
    LatentTcParams p{(const __nv_bfloat16*)q, (const __nv_bfloat16*)pages, (__nv_bfloat16*)out, seq_starts, seq_pos0, block_table, work, heads, max_blocks, num_pages, page_size,
                     box_rows, window, scale, sink, error_flag};
    static bool configured_on[MAX_DEVICES] = {false};         // the attribute belongs to the device
    bool& configured = configured_on[device_index()];
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(latent_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
        if (e != cudaSuccess) return fail(MLB_CUDA_ERROR, "latent_attention_tc: cannot reserve %d bytes of shared memory: %s", (int)SMEM_BYTES, cudaGetErrorString(e));
        configured = true;
    }
    launch_kernel(latent_tc_kernel, dim3(2, num_work, 1), THREADS, SMEM_BYTES, stream, map_q, map_kv, p);
    return check_launch("latent_tc");
}
