// Gated delta rule with one decay per head and key channel, fp32 throughout.  Per head, with S [DK, DV]:
//
//   S <- diag(g_t) S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t
//
//   mlb_delta_prepare   what enters the recurrence besides v: q and k as unit vectors per head (x / sqrt(sum x^2 + 1e-6),
//                       q also times DK^-1/2), beta = sigmoid(b), g = exp(-exp(A_log[h]) * softplus(W2 a + dt_bias)) with a
//                       the (narrow) output of the first of the decay's two projections; W2 is applied here.
//   mlb_delta_scan      the recurrence over the new tokens of every sequence of the step, from the state in the
//                       sequence's slot ([slots, H, DK, DV] fp32; taken as zero when the sequence starts at position 0)
//                       and back into it.  The columns of S never meet: a CTA of 128 threads owns 8 to 32 of them for one (sequence,
//                       head), eight or sixteen lanes share a column's DK rows in registers and meet by shuffles once a token, and
//                       for what is read out once a group of tokens.
//   mlb_delta_output    o / rms(o) per head * weight * sigmoid(W2g a_g), stored in the compute dtype.
//
// The scan kernel also runs the two simpler recurrences with a decay per key channel (mlb_linear_scan, `rule`):
//   rule 1, decayed sum:   S <- diag(g_t) S + k_t v_t^T;   o_t = S^T q_t
//   rule 2, bonus read:    o_t = (S + diag(u) k_t v_t^T)^T q_t;   then S <- diag(g_t) S + k_t v_t^T      (u [H, DK], fixed)
// and one with a decay per head (mlb_head_scan):
//   rule 3, head decay:    S <- g_t S + w_t k_t v_t^T;   o_t = S^T q_t, with one number g per token and head (or one per head,
//                          fixed) and an optional weight w per token and head.  Optionally a vector n [DK] beside S runs the
//                          same recurrence with 1 in the place of v: one more column, whose read-out n . q goes to `den`.
//
// The order of every addition depends on the token's place in its sequence only, never on how the sequence was cut
// into steps: a token's result is the same bits however it is scheduled.
#include "common.cuh"

#include <type_traits>

using namespace mlb;

MLB_DEFINE_LAST_ERROR()

namespace {

constexpr int WARPS = 4;
constexpr int MAX_D = 256;
constexpr int PER_LANE = MAX_D / 32;

struct Columns {
    const float* base; long long ld; int n_partials; long long partial_stride;
    __device__ __forceinline__ float at(long long row, int col) const {
        const float* p = base + row * ld + col;
        float v = p[0];
        for (int k = 1; k < n_partials; ++k) v += p[(size_t)k * partial_stride];
        return v;
    }
    // columns col + lane, col + lane + 32, ... of a row (zero from the n-th on): the partial results of all of them are asked for a step of
    // the sum at a time, four steps together, where at() would make a trip to memory of every few of them
    template <int N> __device__ __forceinline__ void at_lanes(long long row, int col, int n, float (&v)[N]) const {
        const int lane = threadIdx.x & 31;
        const float* p = base + row * ld + col + lane;
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = lane + 32 * i < n ? p[32 * i] : 0.0f;
#pragma unroll 4
        for (int k = 1; k < n_partials; ++k) {
            p += partial_stride;
#pragma unroll
            for (int i = 0; i < N; ++i) if (lane + 32 * i < n) v[i] += p[32 * i];
        }
    }
};

__device__ __forceinline__ float sigmoid(float v) {
    if (v >= 0.0f) return 1.0f / (1.0f + expf(-v));
    const float e = expf(v);
    return e / (1.0f + e);
}

__device__ __forceinline__ float softplus(float v) { return v > 20.0f ? v : log1pf(expf(v)); }

// ------------------------------------------------------------------------------ prepare
struct PrepareParams {
    const float* qkv; long long ld_qkv;      // convolved and activated [T, G*DK | G*DK | H*DV]
    Columns proj; int beta_col, a_col;       // the input projection's fp32 output: beta pre-activations [H], a [a_rank]
    const float* w2;                         // [H * DK, a_rank]; unused when `pre` is given
    Columns pre;                             // W2 a already made by a product [T, H * DK] (base null: made here)
    const float* dt_bias;                    // [H * DK]
    const float* a_log;                      // [H]
    float* qn; float* kn;                    // [T, G * DK]
    float* g;                                // [T, H * DK]
    float* beta;                             // [T, H]
    int T, H, G, DK, a_rank;
};

__global__ void __launch_bounds__(WARPS * 32) delta_prepare_kernel(PrepareParams p) {
    pdl_prologue();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int items = 2 * p.G + p.H;
    const long long item = (long long)blockIdx.x * WARPS + warp;
    if (item >= (long long)p.T * items) return;
    const int t = (int)(item / items), which = (int)(item % items);
    if (which < 2 * p.G) {                   // a head of q or of k: unit vector
        const bool is_q = which < p.G;
        const int head = is_q ? which : which - p.G;
        const float* src = p.qkv + (size_t)t * p.ld_qkv + (is_q ? 0 : p.G * p.DK) + head * p.DK;
        float x[PER_LANE];
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) {
            const int c = lane + 32 * i;
            x[i] = c < p.DK ? src[c] : 0.0f;
            ss = fmaf(x[i], x[i], ss);
        }
        float inv = 1.0f / sqrtf(warp_sum(ss) + 1e-6f);
        if (is_q) inv *= 1.0f / sqrtf((float)p.DK);
        float* dst = (is_q ? p.qn : p.kn) + ((size_t)t * p.G + head) * p.DK;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) { const int c = lane + 32 * i; if (c < p.DK) dst[c] = x[i] * inv; }
        return;
    }
    const int h = which - 2 * p.G;
    const float rate = expf(p.a_log[h]);
    // beta's partial results, one a lane, on their way beside the decay's
    const float* const beta_at = p.proj.base + (size_t)t * p.proj.ld + p.beta_col + h;
    const bool together = p.proj.n_partials <= 32;
    float part = together && lane < p.proj.n_partials ? beta_at[(size_t)lane * p.proj.partial_stride] : 0.0f;
    float pre[PER_LANE];
    if (p.pre.base) {
        p.pre.at_lanes(t, h * p.DK, p.DK, pre);
    } else {
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) pre[i] = 0.0f;
        for (int r = 0; r < p.a_rank; ++r) {
            const float a = p.proj.at(t, p.a_col + r);
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i)
                if (lane + 32 * i < p.DK) pre[i] = fmaf(p.w2[((size_t)h * p.DK + lane + 32 * i) * p.a_rank + r], a, pre[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const int c = lane + 32 * i;
        if (c < p.DK) p.g[((size_t)t * p.H + h) * p.DK + c] = expf(-rate * softplus(pre[i] + p.dt_bias[h * p.DK + c]));
    }
    float beta = __shfl_sync(0xffffffffu, part, 0);
    for (int k = 1; k < min(p.proj.n_partials, 32); ++k) beta += __shfl_sync(0xffffffffu, part, k);       // in split order
    if (!together) beta = p.proj.at(t, p.beta_col + h);
    if (lane == 0) p.beta[(size_t)t * p.H + h] = sigmoid(beta);
}

// ------------------------------------------------------------------------------ the recurrence
struct ScanParams {
    const float* qn; const float* kn;        // [T, G * DK], rows ld_qk apart
    long long ld_qk;
    const float* g;                          // [T, H * DK]
    const float* beta;                       // [T, H]: beta of the delta rule, w of rule 3 (null: 1); else unused and may be null
    const float* bonus;                      // [H, DK] (rule 2 only)
    const float* v; long long ld_v;          // [T, H * DV] (a column block of the convolved rows)
    float* o;                                // [T, H * DV]
    float* state;                            // [slots + 1, H, DK, DV]
    const int* slots; int num_slots;
    const int* seq_starts; const int* seq_pos0;
    int A, H, G, DK, DV;
    int g_pitch;                             // rule 3: numbers between two tokens' decays (H; 0: one per head, fixed)
    float* n_state;                          // rule 3: [slots + 1, H, DK], the vector beside S; null: none
    float* den;                              // rule 3: [T, H], n . q; given exactly when n_state is
    int vec;                                 // 1: every staged row starts on 16 bytes and is a multiple of four floats long
    int* error_flag;
};

__device__ __forceinline__ void copy_async_f32(float* to_shared, const float* from, bool real) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(to_shared);
    const int bytes = real ? 4 : 0;                            // 0: the four bytes are filled with zeros
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(from), "r"(bytes) : "memory");
}

__device__ __forceinline__ void copy_async_f32x4(unsigned to_shared, const float* from, bool real) {
    const int bytes = real ? 16 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(to_shared), "l"(from), "r"(bytes) : "memory");
}

// two fp32 operations an instruction, each rounded as always
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) { return ((f32x2)__float_as_uint(hi) << 32) | __float_as_uint(lo); }
__device__ __forceinline__ float low2(f32x2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float high2(f32x2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// LANES lanes share a column; ROWS: rows of the column that one lane keeps (DK <= LANES * ROWS, ROWS a multiple of 4): lane
// `part` owns rows 4 LANES j + 4 part + (0..3), so that the lanes of a column read consecutive 16-byte pieces of q, k and g.
// PER: neighbouring columns that a lane keeps.  A token's pieces of q, k and g come out of shared memory once for all of
// them, and that is what bounds a step with many columns: 16 bytes a lane take the one path out of shared memory for four cycles,
// two packed operations on them a scheduler's FMA pipe for four as well, but there are four of those.  Fewer columns a lane mean more warps, which
// is what a step with few of them wants (scan_per_lane below).  A column's bits do not depend on PER.  Against one column a lane in
// CTAs of 256 threads, scalar FMAs and a meeting of the lanes for every token's read-out: four prompts, 1,927 tokens, 16 heads of 128 x 128 506 ->
// 329 us, one of 906 tokens 303 -> 229, head decay 283 -> 195 and 141 -> 125.
// CHUNK: tokens whose q, k, g, v and beta are staged in shared memory at a time; the next chunk is copied there
// asynchronously (cp.async, zero fill for padding) while the present one is computed, so the recurrence never waits for
// global memory inside a chunk.  A thread copies the same pieces of every token: its addresses grow by fixed pitches.
constexpr int RULE_DELTA = 0, RULE_DECAYED_SUM = 1, RULE_BONUS_READ = 2, RULE_HEAD_DECAY = 3;
constexpr int SCAN_THREADS = 128;
__host__ __device__ constexpr int log2_of(int n) { return n <= 1 ? 0 : 1 + log2_of(n / 2); }

template <int LANES, int ROWS, int CHUNK, int RULE, int PER>
__global__ void __launch_bounds__(SCAN_THREADS) delta_scan_kernel(ScanParams p) {
    pdl_launch_dependents();
    constexpr int COLS = SCAN_THREADS / LANES * PER;          // columns of a CTA
    constexpr int DKP = LANES * ROWS;                         // padded key width
    constexpr int V_AT = (RULE == RULE_HEAD_DECAY ? 2 : 3) * DKP;
    constexpr int PER_TOKEN = V_AT + COLS + 4;           // q | k | g (not rule 3) | v of this CTA's columns | beta (rule 3: g, w) and unused
    constexpr int STAGED = CHUNK * PER_TOKEN;
    extern __shared__ __align__(16) float stage_s[];          // [2][STAGED]
    struct __align__(4 * PER) Own { float v[PER]; };          // a lane's columns of v, one load
    const int all_cols = RULE == RULE_HEAD_DECAY && p.n_state ? p.DV + 1 : p.DV;      // rule 3: the vector beside S is column DV
    const int col_blocks = (all_cols + COLS - 1) / COLS;
    const int cb = blockIdx.x % col_blocks, h = (blockIdx.x / col_blocks) % p.H, a = blockIdx.x / (col_blocks * p.H);
    const int part = threadIdx.x & (LANES - 1);
    const int local_col = threadIdx.x / LANES * PER;          // the first of this lane's columns
    const int col = cb * COLS + local_col;
    // rule 3 with a vector: column DV is the vector beside S
    auto col_ok = [&](int j) { return col + j < all_cols; };
    auto is_n = [&](int j) { return RULE == RULE_HEAD_DECAY && p.n_state && col + j == p.DV; };
    const int slot = p.slots[a];
    const bool slot_ok = slot >= 0 && slot < p.num_slots;
    const bool fresh = p.seq_pos0[a] == 0;
    auto row_of = [&](int i) { return (i >> 2) * (4 * LANES) + part * 4 + (i & 3); };
    // the state of column j at row 0, and the distance between its rows
    auto state_at = [&](int j) {
        return is_n(j) ? p.n_state + ((size_t)slot * p.H + h) * p.DK : p.state + (((size_t)slot * p.H + h) * p.DK) * p.DV + col + j;
    };
    auto state_pitch = [&](int j) { return is_n(j) ? (size_t)1 : (size_t)p.DV; };
    if (slot_ok && !fresh && cb * COLS < p.DV)                // on its way while the kernel in front ends (its values are read behind the wait)
        for (int r = threadIdx.x; r < p.DK; r += SCAN_THREADS)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.state + (((size_t)slot * p.H + h) * p.DK + r) * p.DV + cb * COLS));
    pdl_wait();
    const int start = p.seq_starts[a], n = p.seq_starts[a + 1] - start;
    if (!slot_ok) {
        if (threadIdx.x == 0 && p.error_flag) atomicExch(p.error_flag, 3);
        return;
    }
    const int kvh = h / (p.H / p.G);

    const float* const q_base = p.qn + (size_t)start * p.ld_qk + (size_t)kvh * p.DK;
    const float* const k_base = p.kn + (size_t)start * p.ld_qk + (size_t)kvh * p.DK;
    const float* const g_base = RULE == RULE_HEAD_DECAY ? p.g + (size_t)start * p.g_pitch + h : p.g + ((size_t)start * p.H + h) * p.DK;
    const float* const v_base = p.v + (size_t)start * p.ld_v + (size_t)h * p.DV;
    const float* const b_base = p.beta ? p.beta + (size_t)start * p.H + h : g_base;     // without beta: any readable address, the value is unused
    const size_t qk_pitch = (size_t)p.ld_qk, g_pitch = (size_t)p.H * p.DK;
    // four floats at a time (p.vec): piece u of a token is q, k, g in pieces of four, then v, then beta (rule 3: g and w)
    constexpr int UNITS = V_AT / 4 + COLS / 4 + 1, MINE = (UNITS + SCAN_THREADS - 1) / SCAN_THREADS;
    const float* from[MINE];
    size_t pitch[MINE];
    bool real[MINE];
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
        const int u = threadIdx.x + i * SCAN_THREADS;
        if (u < V_AT / 4) {
            const int which = u / (DKP / 4), c = (u % (DKP / 4)) * 4;
            real[i] = c < p.DK;
            from[i] = (which == 0 ? q_base : which == 1 ? k_base : g_base) + (real[i] ? c : 0);
            pitch[i] = which < 2 ? qk_pitch : g_pitch;
        } else if (u < UNITS - 1) {
            const int vc = cb * COLS + (u - V_AT / 4) * 4;
            real[i] = vc < p.DV;
            from[i] = v_base + (real[i] ? vc : 0);
            pitch[i] = (size_t)p.ld_v;
        } else {
            real[i] = true;
            from[i] = RULE == RULE_HEAD_DECAY ? g_base : b_base;
            pitch[i] = RULE == RULE_HEAD_DECAY ? (size_t)p.g_pitch : (size_t)p.H;
        }
    }
    // the chunk that begins at token `first` into staging buffer `buf`; padding (rows beyond DK, columns beyond DV) becomes
    // zero: a zero k and q keep such rows of S at zero whatever g is.  Tokens beyond the sequence's are not staged (nor read).
    auto stage = [&](int first, int buf) {
        const int tokens = min(CHUNK, n - first);
        float* const to = stage_s + buf * STAGED;
        if (p.vec) {                             // every row a multiple of four floats and 16-byte aligned
#pragma unroll
            for (int i = 0; i < MINE; ++i) {
                const int u = threadIdx.x + i * SCAN_THREADS;
                if (u < UNITS - 1) {
                    unsigned dst = (unsigned)__cvta_generic_to_shared(to + u * 4);
                    const float* src = from[i];
                    for (int tok = 0; tok < tokens; ++tok, dst += PER_TOKEN * 4, src += pitch[i]) copy_async_f32x4(dst, src, real[i]);
                    from[i] = src;
                } else if (u == UNITS - 1) {
                    const float* src = from[i];
                    for (int tok = 0; tok < tokens; ++tok, src += pitch[i]) {
                        copy_async_f32(to + tok * PER_TOKEN + V_AT + COLS, src, true);
                        if (RULE == RULE_HEAD_DECAY && p.beta)
                            copy_async_f32(to + tok * PER_TOKEN + V_AT + COLS + 1, b_base + (size_t)(first + tok) * p.H, true);
                    }
                    from[i] = src;
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            return;
        }
        for (int e = threadIdx.x; e < tokens * PER_TOKEN; e += SCAN_THREADS) {
            const int tok = e / PER_TOKEN, w = e % PER_TOKEN;
            const size_t t = (size_t)(first + tok);
            const int which = w / DKP, c = w % DKP;
            const int vc = cb * COLS + (w - V_AT);
            const float* at;
            bool real;
            if (which == 0) { real = c < p.DK; at = q_base + t * qk_pitch + (real ? c : 0); }
            else if (which == 1) { real = c < p.DK; at = k_base + t * qk_pitch + (real ? c : 0); }
            else if (RULE != RULE_HEAD_DECAY && which == 2) { real = c < p.DK; at = g_base + t * g_pitch + (real ? c : 0); }
            else if (w < V_AT + COLS) { real = vc < p.DV; at = v_base + t * p.ld_v + (real ? vc : 0); }
            else if (RULE == RULE_HEAD_DECAY) {
                real = w == V_AT + COLS || (w == V_AT + COLS + 1 && p.beta);
                at = w == V_AT + COLS + 1 && p.beta ? b_base + t * p.H : g_base + t * p.g_pitch;
            } else { real = w == V_AT + COLS; at = b_base + t * p.H; }
            copy_async_f32(to + e, at, real);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (n > 0) stage(0, 0);

    f32x2 S[PER][ROWS / 2];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const float* const st = state_at(j);
#pragma unroll
        for (int i = 0; i < ROWS / 2; ++i) {
            const bool there = !fresh && col_ok(j);
            const float lo = there && row_of(2 * i) < p.DK ? st[(size_t)row_of(2 * i) * state_pitch(j)] : 0.0f;
            const float hi = there && row_of(2 * i + 1) < p.DK ? st[(size_t)row_of(2 * i + 1) * state_pitch(j)] : 0.0f;
            S[j][i] = pack2(lo, hi);
        }
    }
    f32x2 U[RULE == RULE_BONUS_READ ? ROWS / 2 : 1];
    if (RULE == RULE_BONUS_READ) {
#pragma unroll
        for (int i = 0; i < ROWS / 2; ++i) {
            const float* const u = p.bonus + (size_t)h * p.DK;
            U[i] = pack2(row_of(2 * i) < p.DK ? u[row_of(2 * i)] : 0.0f, row_of(2 * i + 1) < p.DK ? u[row_of(2 * i + 1)] : 0.0f);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the distances at which the lanes of a column meet for its read-out: from the nearest on in the delta rule, from the furthest on else
    constexpr int STAGES = LANES == 16 ? 4 : 3, LOG_N = log2_of((CHUNK < LANES ? CHUNK : LANES) * PER);
    auto distance = [](int stage) { return RULE == RULE_DELTA ? 1 << stage : LANES / 2 >> stage; };
    auto store_o = [&](int t, int j, float value) {          // token t of the sequence, column j of this lane
        if (!col_ok(j)) return;
        if (is_n(j)) p.den[((size_t)start + t) * p.H + h] = value;
        else p.o[((size_t)start + t) * ((size_t)p.H * p.DV) + (size_t)h * p.DV + col + j] = value;
    };
    for (int first = 0, buf = 0; first < n; first += CHUNK, buf ^= 1) {
        if (first + CHUNK < n) stage(first + CHUNK, buf ^ 1);
        const int count = min(CHUNK, n - first);
        // one token: the state moves on, and share[j] becomes this lane's share of column j's o
        auto token = [&](int tok, float* share) {
            const float* row = stage_s + buf * STAGED + tok * PER_TOKEN;
            const ulonglong2* qs = reinterpret_cast<const ulonglong2*>(row) + part;
            const ulonglong2* ks = reinterpret_cast<const ulonglong2*>(row + DKP) + part;
            const ulonglong2* gs = reinterpret_cast<const ulonglong2*>(row + 2 * DKP) + part;          // (not rule 3)
            Own own = *reinterpret_cast<const Own*>(row + V_AT + local_col);
            float (&v)[PER] = own.v;
            const float beta = row[V_AT + COLS];                                               // (rule 3: the head's decay)
            if (RULE == RULE_HEAD_DECAY) {
                const float weight = p.beta ? row[V_AT + COLS + 1] : 1.0f;
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    if (is_n(j)) v[j] = 1.0f;
                    if (p.beta) v[j] *= weight;
                }
            }
            // four chains a column instead of one (always the same four), two to a register pair
            if constexpr (RULE != RULE_DELTA) {
                // S <- diag(g) S + k v^T with the read-out S^T q behind it (decayed sum), or in front of it with the
                // bonus u on the present token's own k v^T (bonus read); one meeting of the lanes a token
                f32x2 o01[PER], o23[PER];
#pragma unroll
                for (int j = 0; j < PER; ++j) o01[j] = o23[j] = 0ull;
#pragma unroll
                for (int i = 0; i < ROWS / 4; ++i) {
                    const ulonglong2 kk = ks[i * LANES], qq = qs[i * LANES];
                    ulonglong2 gg;
                    if (RULE == RULE_HEAD_DECAY) gg.x = gg.y = pack2(beta, beta); else gg = gs[i * LANES];
#pragma unroll
                    for (int j = 0; j < PER; ++j) {
                        const f32x2 vv = pack2(v[j], v[j]), kv01 = mul2(kk.x, vv), kv23 = mul2(kk.y, vv);
                        if (RULE == RULE_BONUS_READ) {
                            o01[j] = fma2(fma2(U[2 * i], kv01, S[j][2 * i]), qq.x, o01[j]);
                            o23[j] = fma2(fma2(U[2 * i + 1], kv23, S[j][2 * i + 1]), qq.y, o23[j]);
                        }
                        S[j][2 * i] = fma2(S[j][2 * i], gg.x, kv01);
                        S[j][2 * i + 1] = fma2(S[j][2 * i + 1], gg.y, kv23);
                        if (RULE != RULE_BONUS_READ) {
                            o01[j] = fma2(S[j][2 * i], qq.x, o01[j]);
                            o23[j] = fma2(S[j][2 * i + 1], qq.y, o23[j]);
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < PER; ++j) share[j] = (low2(o01[j]) + high2(o01[j])) + (low2(o23[j]) + high2(o23[j]));
            } else {
                ulonglong2 kk[ROWS / 4];
                f32x2 d01[PER], d23[PER];
#pragma unroll
                for (int j = 0; j < PER; ++j) d01[j] = d23[j] = 0ull;
#pragma unroll
                for (int i = 0; i < ROWS / 4; ++i) {
                    const ulonglong2 gg = gs[i * LANES];
                    kk[i] = ks[i * LANES];
#pragma unroll
                    for (int j = 0; j < PER; ++j) {
                        S[j][2 * i] = mul2(S[j][2 * i], gg.x);
                        S[j][2 * i + 1] = mul2(S[j][2 * i + 1], gg.y);
                        d01[j] = fma2(S[j][2 * i], kk[i].x, d01[j]);
                        d23[j] = fma2(S[j][2 * i + 1], kk[i].y, d23[j]);
                    }
                }
                float u[PER];
#pragma unroll
                for (int j = 0; j < PER; ++j) u[j] = (low2(d01[j]) + high2(d01[j])) + (low2(d23[j]) + high2(d23[j]));
#pragma unroll
                for (int off = 1; off < LANES; off <<= 1)
#pragma unroll
                    for (int j = 0; j < PER; ++j) u[j] += __shfl_xor_sync(0xffffffffu, u[j], off);
#pragma unroll
                for (int j = 0; j < PER; ++j) { u[j] = beta * (v[j] - u[j]); d01[j] = d23[j] = 0ull; }
#pragma unroll
                for (int i = 0; i < ROWS / 4; ++i) {
                    const ulonglong2 qq = qs[i * LANES];
#pragma unroll
                    for (int j = 0; j < PER; ++j) {
                        const f32x2 uu = pack2(u[j], u[j]);
                        S[j][2 * i] = fma2(kk[i].x, uu, S[j][2 * i]);
                        S[j][2 * i + 1] = fma2(kk[i].y, uu, S[j][2 * i + 1]);
                        d01[j] = fma2(S[j][2 * i], qq.x, d01[j]);
                        d23[j] = fma2(S[j][2 * i + 1], qq.y, d23[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < PER; ++j) share[j] = (low2(d01[j]) + high2(d01[j])) + (low2(d23[j]) + high2(d23[j]));
            }
        };
        if (count == CHUNK) {
            // A whole chunk: the lanes of a column keep their shares of o for a group of GROUP tokens and meet once for all of
            // them, since nothing waits for the read-out.  A stage at distance `off` halves what a lane carries: it keeps the
            // half of the (token, column) pairs that its own bit `off` names and adds the partner's share of those, so that
            // N shares of LANES lanes take about N shuffles instead of N log2(LANES).  Every sum is the one the lone form makes
            // (the same pairs at the same distances in the same order), so both forms give the same bits.
            constexpr int GROUP = CHUNK < LANES ? CHUNK : LANES, N = GROUP * PER;
            constexpr int LEFT = N < LANES ? 1 : N / LANES;            // values that a lane ends with
#pragma unroll 1
            for (int g0 = 0; g0 < CHUNK; g0 += GROUP) {
                float share[N];                                        // share[token * PER + column]
#pragma unroll
                for (int i = 0; i < GROUP; ++i) token(g0 + i, share + i * PER);
                int mine = 0;                                          // this lane's first value
                bool keeps = true;                                     // (of lanes that end with the same value the first one)
#pragma unroll
                for (int stage = 0; stage < STAGES; ++stage) {
                    const int off = distance(stage);
                    const bool upper = (part & off) != 0;
                    if (stage >= LOG_N) {                              // one value left, more lanes than values
                        share[0] += __shfl_xor_sync(0xffffffffu, share[0], off);
                        keeps = keeps && !upper;
                    } else {
#pragma unroll
                        for (int i = 0; i < N >> (stage + 1); ++i) {
                            const float keep = upper ? share[i + (N >> (stage + 1))] : share[i];
                            const float send = upper ? share[i] : share[i + (N >> (stage + 1))];
                            share[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                        }
                        if (upper) mine += N >> (stage + 1);
                    }
                }
                if (keeps) {
#pragma unroll
                    for (int i = 0; i < LEFT; ++i) store_o(first + g0 + (mine + i) / PER, (mine + i) % PER, share[i]);
                }
            }
        } else {
            for (int tok = 0; tok < count; ++tok) {
                float share[PER];
                token(tok, share);
#pragma unroll
                for (int stage = 0; stage < STAGES; ++stage)
#pragma unroll
                    for (int j = 0; j < PER; ++j) share[j] += __shfl_xor_sync(0xffffffffu, share[j], distance(stage));
                if (part == 0) {
#pragma unroll
                    for (int j = 0; j < PER; ++j) store_o(first + tok, j, share[j]);
                }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        float* const st = state_at(j);
#pragma unroll
        for (int i = 0; i < ROWS / 2; ++i) {
            if (col_ok(j) && row_of(2 * i) < p.DK) st[(size_t)row_of(2 * i) * state_pitch(j)] = low2(S[j][i]);
            if (col_ok(j) && row_of(2 * i + 1) < p.DK) st[(size_t)row_of(2 * i + 1) * state_pitch(j)] = high2(S[j][i]);
        }
    }
}

// ------------------------------------------------------------------------------ output norm and gate
struct OutputParams {
    const float* o;                          // [T, H * DV]
    const float* weight;                     // [DV]
    Columns proj; int g_col;                 // the narrow output of the gate's first projection [g_rank]
    const float* w2;                         // [H * DV, g_rank]; unused when `pre` is given
    Columns pre;                             // W2g a_g already made by a product [T, H * DV] (base null: made here)
    void* out;                               // [T, H * DV]
    int T, H, DV, g_rank; float eps;
};

template <typename OutT>
__global__ void __launch_bounds__(WARPS * 32) delta_output_kernel(OutputParams p) {
    pdl_prologue();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * WARPS + warp;
    if (item >= (long long)p.T * p.H) return;
    const int t = (int)(item / p.H), h = (int)(item % p.H);
    const float* src = p.o + ((size_t)t * p.H + h) * p.DV;
    float x[PER_LANE];
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const int c = lane + 32 * i;
        x[i] = c < p.DV ? src[c] : 0.0f;
        ss = fmaf(x[i], x[i], ss);
    }
    float pre[PER_LANE];
    if (p.pre.base) {
        p.pre.at_lanes(t, h * p.DV, p.DV, pre);
    } else {
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) pre[i] = 0.0f;
        for (int r = 0; r < p.g_rank; ++r) {
            const float a = p.proj.at(t, p.g_col + r);
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i)
                if (lane + 32 * i < p.DV) pre[i] = fmaf(p.w2[((size_t)h * p.DV + lane + 32 * i) * p.g_rank + r], a, pre[i]);
        }
    }
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)p.DV + p.eps);
    OutT* dst = (OutT*)p.out + ((size_t)t * p.H + h) * p.DV;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const int c = lane + 32 * i;
        if (c < p.DV) dst[c] = from_f32<OutT>(x[i] * inv * p.weight[c] * sigmoid(pre[i]));
    }
}

// out[t, c] = src[t, col0 + c] (partial results summed in split order), stored in the compute dtype: the narrow output of
// a first projection made ready for the second one (`activation` 1: its tanh).
template <typename OutT>
__global__ void take_columns_kernel(Columns src, int col0, int n, int T, OutT* out, int activation) {
    pdl_prologue();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)T * n) return;
    const float v = src.at(i / n, col0 + (int)(i % n));
    out[i] = from_f32<OutT>(activation == 1 ? tanhf(v) : v);
}

}  // namespace

MLB_EXPORT int mlb_take_columns(const float* src, long long ld, int n_partials, long long partial_stride, int col0, int n, int T,
                                void* out, int out_dtype, int activation, cudaStream_t stream) {
    if (!src || !out || n <= 0 || T < 0 || activation < 0 || activation > 1) return fail(MLB_INVALID_ARGUMENT, "take_columns: bad operands");
    if (T == 0) return MLB_OK;
    Columns c{src, ld, n_partials < 1 ? 1 : n_partials, partial_stride};
    const unsigned blocks = (unsigned)(((long long)T * n + 255) / 256);
    if (out_dtype == MLB_BF16) launch_kernel(take_columns_kernel<__nv_bfloat16>, blocks, 256, 0, stream, c, col0, n, T, (__nv_bfloat16*)out, activation);
    else launch_kernel(take_columns_kernel<float>, blocks, 256, 0, stream, c, col0, n, T, (float*)out, activation);
    return check_launch("take_columns");
}

MLB_EXPORT int mlb_delta_prepare(const float* qkv, long long ld_qkv, const float* proj, long long ld_proj, int n_partials,
                                 long long partial_stride, int beta_col, int a_col, const float* w2, const float* pre, long long ld_pre,
                                 int pre_partials, long long pre_partial_stride, const float* dt_bias,
                                 const float* a_log, float* qn, float* kn, float* g, float* beta, int T, int H, int G, int DK,
                                 int a_rank, cudaStream_t stream) {
    if (T < 0 || H <= 0 || G <= 0 || H % G || DK <= 0 || DK > MAX_D || a_rank <= 0)
        return fail(MLB_UNSUPPORTED_SIZE, "delta_prepare: heads %d/%d, key width %d (at most %d), rank %d", H, G, DK, MAX_D, a_rank);
    if (!qkv || !proj || (!w2 && !pre) || !dt_bias || !a_log || !qn || !kn || !g || !beta) return fail(MLB_INVALID_ARGUMENT, "delta_prepare: null operand");
    if (T == 0) return MLB_OK;
    PrepareParams p{qkv, ld_qkv, Columns{proj, ld_proj, n_partials < 1 ? 1 : n_partials, partial_stride}, beta_col, a_col, w2,
                    Columns{pre, ld_pre, pre_partials < 1 ? 1 : pre_partials, pre_partial_stride}, dt_bias, a_log, qn, kn, g, beta, T, H, G, DK, a_rank};
    const long long items = (long long)T * (2 * G + H);
    launch_kernel(delta_prepare_kernel, (unsigned)((items + WARPS - 1) / WARPS), WARPS * 32, 0, stream, p);
    return check_launch("delta_prepare");
}

namespace {

// Columns a lane keeps, one or two.  Measured (us, one / two; 148 SMs): 4 prompts, 1,927 tokens, 906 the longest, 16 heads of 128 x 128
// (55 columns an SM) delta rule 422 / 329, head decay 268 / 195; 8 of 512 tokens 713 / 418 and 438 / 252; one prompt of 906 (14 an SM) 229 / 240 and
// 143 / 125; 2,048 tokens of 32 heads of 128 x 64 (14) delta 504 / 531, decayed sum 444 / 297, bonus read 385 / 355, head decay 330 / 268; of 8 heads of
// 64 x 64 (3.5) 336 / 426, 158 / 166, 166 / 191, 158 / 182.  Four a lane are never the faster: 332, 207, 418, 256, 293, 176, ...
template <int RULE>
int scan_per_lane(long long columns) {
    return columns >= (RULE == RULE_DELTA ? 24ll : 8ll) * sm_count() ? 2 : 1;
}

template <int RULE>
int launch_scan(const float* qn, const float* kn, const float* g, const float* beta, const float* bonus, const float* v, long long ld_v,
                float* o, float* state, const int* slots, int num_slots, const int* seq_starts, const int* seq_pos0,
                int T, int A, int H, int G, int DK, int DV, int* error_flag, cudaStream_t stream, int g_pitch = 0, float* n_state = nullptr,
                float* den = nullptr, long long ld_qk = 0) {
    if (T < 0 || A < 0 || H <= 0 || G <= 0 || H % G || DK <= 0 || DK > MAX_D || DV <= 0)
        return fail(MLB_UNSUPPORTED_SIZE, "scan: heads %d/%d, widths %d (at most %d) / %d", H, G, DK, MAX_D, DV);
    if (!qn || !kn || !g || (RULE == RULE_DELTA && !beta) || (RULE == RULE_BONUS_READ && !bonus) || !v || !o || !state || !slots ||
        !seq_starts || !seq_pos0)
        return fail(MLB_INVALID_ARGUMENT, "scan: null operand");
    if (A == 0) return MLB_OK;
    const bool aligned = ((uintptr_t)qn | (uintptr_t)kn | (RULE == RULE_HEAD_DECAY ? 0 : (uintptr_t)g) | (uintptr_t)v) % 16 == 0;
    if (ld_qk == 0) ld_qk = (long long)G * DK;
    if (ld_qk < (long long)G * DK) return fail(MLB_INVALID_ARGUMENT, "scan: q and k rows overlap");
    const int vec = aligned && DK % 4 == 0 && DV % 4 == 0 && ld_v % 4 == 0 && ld_qk % 4 == 0;
    ScanParams p{qn, kn, ld_qk, g, beta, bonus, v, ld_v, o, state, slots, num_slots, seq_starts, seq_pos0, A, H, G, DK, DV,
                 g_pitch, n_state, den, vec, error_flag};
    // Long-running CTAs (a prompt portion: one CTA walks all its tokens) must be spread evenly over the SMs.  Started
    // early behind a predecessor that still fills the SMs, they land wherever a slot falls free, several on one SM, and
    // the slowest SM decides: such a launch waits for its predecessor the plain way.  CTAs of a few tokens (decoding) start early.
    const bool early = T <= 4 * A;
    const long long columns = (long long)A * H * (DV + (n_state ? 1 : 0));
    auto go = [&](auto kernel, int cols, int chunk, int per_token) -> int {
        const unsigned blocks = (unsigned)((long long)A * H * ((DV + (n_state ? 1 : 0) + cols - 1) / cols));
        const size_t smem = (size_t)2 * chunk * per_token * sizeof(float);
        if (early) launch_kernel(kernel, blocks, SCAN_THREADS, smem, stream, p);
        else kernel<<<blocks, SCAN_THREADS, smem, stream>>>(p);
        return check_launch("scan");
    };
    auto with = [&](auto lanes_, auto rows_, auto chunk_) -> int {
        constexpr int LANES = decltype(lanes_)::value, ROWS = decltype(rows_)::value, CHUNK = decltype(chunk_)::value;
        auto per = [&](auto per_) -> int {
            constexpr int PER = decltype(per_)::value, COLS = SCAN_THREADS / LANES * PER;
            return go(delta_scan_kernel<LANES, ROWS, CHUNK, RULE, PER>, COLS, CHUNK, (RULE == RULE_HEAD_DECAY ? 2 : 3) * LANES * ROWS + COLS + 4);
        };
        return scan_per_lane<RULE>(columns) == 2 ? per(std::integral_constant<int, 2>()) : per(std::integral_constant<int, 1>());
    };
    // (rule 3 stages a third less per token: twice the tokens at a time fit; measured for 2,048 tokens 204 against 232 us at
    // DK 64 and 342 against 412 us at DK 128)
    constexpr int MORE = RULE == RULE_HEAD_DECAY ? 2 : 1;
    using std::integral_constant;
    if (DK <= 32) return with(integral_constant<int, 8>(), integral_constant<int, 4>(), integral_constant<int, 16 * MORE>());
    if (DK <= 64) return with(integral_constant<int, 16>(), integral_constant<int, 4>(), integral_constant<int, 16 * MORE>());
    if (DK <= 128) return with(integral_constant<int, 16>(), integral_constant<int, 8>(), integral_constant<int, 8 * MORE>());
    return with(integral_constant<int, 16>(), integral_constant<int, 16>(), integral_constant<int, 4 * MORE>());
}

}  // namespace

MLB_EXPORT int mlb_delta_scan(const float* qn, const float* kn, const float* g, const float* beta, const float* v, long long ld_v,
                              float* o, float* state, const int* slots, int num_slots, const int* seq_starts, const int* seq_pos0,
                              int T, int A, int H, int G, int DK, int DV, int* error_flag, cudaStream_t stream) {
    return launch_scan<RULE_DELTA>(qn, kn, g, beta, nullptr, v, ld_v, o, state, slots, num_slots, seq_starts, seq_pos0, T, A, H, G, DK, DV,
                                   error_flag, stream);
}

// rule 1: S <- diag(g) S + k v^T, o = S^T q;   rule 2: o = (S + diag(bonus) k v^T)^T q, then S <- diag(g) S + k v^T.
// q, k [T, G * DK], g [T, H * DK], bonus [H, DK] (rule 2), v rows of pitch ld_v, o [T, H * DV], state [slots, H, DK, DV].
MLB_EXPORT int mlb_linear_scan(int rule, const float* q, const float* k, const float* g, const float* bonus, const float* v,
                               long long ld_v, float* o, float* state, const int* slots, int num_slots, const int* seq_starts,
                               const int* seq_pos0, int T, int A, int H, int G, int DK, int DV, int* error_flag, cudaStream_t stream) {
    if (rule == RULE_DECAYED_SUM)
        return launch_scan<RULE_DECAYED_SUM>(q, k, g, nullptr, nullptr, v, ld_v, o, state, slots, num_slots, seq_starts, seq_pos0, T, A, H, G,
                                             DK, DV, error_flag, stream);
    if (rule == RULE_BONUS_READ)
        return launch_scan<RULE_BONUS_READ>(q, k, g, nullptr, bonus, v, ld_v, o, state, slots, num_slots, seq_starts, seq_pos0, T, A, H, G,
                                            DK, DV, error_flag, stream);
    return fail(MLB_INVALID_ARGUMENT, "linear_scan: unknown rule %d", rule);
}

// rule 3: S <- g S + w k v^T, o = S^T q.  g [T, H] (per_token 1) or [H] (0, fixed); w [T, H] or null (1).  n_state [slots, H, DK] and
// den [T, H] together: n <- g n + w k, den = n . q.  q, k [T, G * DK] with rows ld_qk apart; head h reads q/k head h / (H / G).
MLB_EXPORT int mlb_head_scan(const float* q, const float* k, long long ld_qk, int G, const float* g, int per_token, const float* w, const float* v, long long ld_v,
                             float* o, float* state, float* n_state, float* den, const int* slots, int num_slots, const int* seq_starts,
                             const int* seq_pos0, int T, int A, int H, int DK, int DV, int* error_flag, cudaStream_t stream) {
    if ((n_state == nullptr) != (den == nullptr)) return fail(MLB_INVALID_ARGUMENT, "head_scan: the vector's state and its read-out come together");
    return launch_scan<RULE_HEAD_DECAY>(q, k, g, w, nullptr, v, ld_v, o, state, slots, num_slots, seq_starts, seq_pos0, T, A, H, G, DK, DV, error_flag,
                                        stream, per_token ? H : 0, n_state, den, ld_qk);
}

MLB_EXPORT int mlb_delta_output(const float* o, const float* weight, const float* proj, long long ld_proj, int n_partials,
                                long long partial_stride, int g_col, const float* w2, const float* pre, long long ld_pre,
                                int pre_partials, long long pre_partial_stride, void* out, int out_dtype, int T, int H,
                                int DV, int g_rank, float eps, cudaStream_t stream) {
    if (T < 0 || H <= 0 || DV <= 0 || DV > MAX_D || g_rank <= 0)
        return fail(MLB_UNSUPPORTED_SIZE, "delta_output: value width %d (at most %d), rank %d", DV, MAX_D, g_rank);
    if (!o || !weight || !proj || (!w2 && !pre) || !out) return fail(MLB_INVALID_ARGUMENT, "delta_output: null operand");
    if (T == 0) return MLB_OK;
    OutputParams p{o, weight, Columns{proj, ld_proj, n_partials < 1 ? 1 : n_partials, partial_stride}, g_col, w2,
                   Columns{pre, ld_pre, pre_partials < 1 ? 1 : pre_partials, pre_partial_stride}, out, T, H, DV, g_rank, eps};
    const long long items = (long long)T * H;
    const unsigned blocks = (unsigned)((items + WARPS - 1) / WARPS);
    if (out_dtype == MLB_BF16) launch_kernel(delta_output_kernel<__nv_bfloat16>, blocks, WARPS * 32, 0, stream, p);
    else launch_kernel(delta_output_kernel<float>, blocks, WARPS * 32, 0, stream, p);
    return check_launch("delta_output");
}
