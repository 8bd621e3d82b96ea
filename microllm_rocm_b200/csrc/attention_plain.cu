// Plain attention over the paged cache: any mix of prompt portions and decoded tokens.
//
// The query at absolute position `pos` of its sequence sees keys lo..pos, lo = max(0, pos - window + 1) for a windowed layer
// and 0 otherwise; keys beyond `pos` are never read (the reference computes no masked scores
// either: src/ops/ops.cpp:2343-2384).  Query head h uses kv head h / (NH/NKV)
// (ops.cpp:2357; consecutive query heads share one).  score = dot(q, k) * scale with the
// scale applied after the dot product (ops.cpp:2365-2369); softmax and the value sum are
// fp32 (ops.cpp:1624-1661 for the cached case).
//
// Keys are walked in tiles of 32 whose edges sit at multiples of 32 of the ABSOLUTE
// position, with a running maximum and sum.  The order of every addition therefore depends
// only on (pos, window), not on how the prompt was cut into steps, on the other requests of
// the batch, or on which physical pages hold the keys: in the fp32 path the same token gets
// bit-identical output however it is scheduled.  These kernels are the whole fp32 path's
// attention and the reference beside the tensor-core kernels.
//
//   paged_attention_rows_kernel    head sizes that are multiples of 4 (beyond 128: of 8)
//   paged_attention_plain_kernel   the others, whose rows have no such pieces: a warp per (token, head)
#include <type_traits>

#include "common.cuh"

using namespace mlb;

MLB_DEFINE_LAST_ERROR()

namespace {

constexpr int WARPS = 4;
constexpr int MAX_D = 256;

struct AttnParams {
    const void* q;           // [T, NH*D]
    const void* pages;       // [num_pages, 2, NKV, page_size, D]
    void* out;               // [T, NH*D]
    const int* positions;    // [T]
    const int* token_seq;    // [T]
    const int* block_table;  // [A, max_blocks]
    int max_blocks, num_pages, page_size;
    int tokens, num_heads, num_kv_heads, head_dim;
    int chunk;               // > 0: only keys of the query's own block of `chunk` positions (counted from 0)
    int window;              // 0: all earlier keys
    float scale;
    int* error_flag;
};

template <typename QT, typename KVT, typename OutT>
__global__ void __launch_bounds__(WARPS * 32)
paged_attention_plain_kernel(AttnParams p) {
    pdl_prologue();
    __shared__ float q_s[WARPS][MAX_D];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * WARPS + warp;
    if (item >= (long long)p.tokens * p.num_heads) return;     // whole warp leaves together
    const int t = (int)(item / p.num_heads), h = (int)(item % p.num_heads);
    const int D = p.head_dim;
    const int kvh = h / (p.num_heads / p.num_kv_heads);
    const int pos = p.positions[t];
    const int seq = p.token_seq[t];
    const int lo = first_visible_key(pos, p.window, p.chunk);

    const QT* qrow = (const QT*)p.q + ((size_t)t * p.num_heads + h) * D;
    for (int c = lane; c < D; c += 32) q_s[warp][c] = to_f32(qrow[c]);
    __syncwarp();

    constexpr int PER_LANE = MAX_D / 32;
    float acc[PER_LANE];
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) acc[i] = 0.0f;
    float m = -INFINITY, l = 0.0f;
    const size_t page_stride = (size_t)2 * p.num_kv_heads * p.page_size * D;
    const size_t v_offset = (size_t)p.num_kv_heads * p.page_size * D;
    const int* table = p.block_table + (size_t)seq * p.max_blocks;

    for (int base = (lo / 32) * 32; base <= pos; base += 32) {
        const int kp = base + lane;
        bool valid = kp >= lo && kp <= pos;
        long long k_off = -1;
        if (valid) {
            const int block = kp / p.page_size;
            const int page = block < p.max_blocks ? table[block] : -1;
            if (page < 0 || page >= p.num_pages) {
                if (p.error_flag) atomicExch(p.error_flag, 2);
                valid = false;
            } else {
                k_off = (long long)((size_t)page * page_stride + ((size_t)kvh * p.page_size + kp % p.page_size) * D);
            }
        }
        float s = -INFINITY;
        if (valid) {
            const KVT* krow = (const KVT*)p.pages + k_off;
            float dot = 0.0f;
            for (int c = 0; c < D; ++c) dot = fmaf(q_s[warp][c], to_f32(krow[c]), dot);
            s = dot * p.scale;
        }
        const float m_new = fmaxf(m, warp_max(s));
        if (m_new == -INFINITY) continue;                     // no readable key in this tile
        const float prob = valid ? expf(s - m_new) : 0.0f;
        const float corr = (m == -INFINITY) ? 0.0f : expf(m - m_new);
        l = l * corr + warp_sum(prob);
        m = m_new;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) acc[i] *= corr;
        const unsigned valid_mask = __ballot_sync(0xffffffffu, valid);
        for (int j = 0; j < 32; ++j) {
            const float pj = __shfl_sync(0xffffffffu, prob, j);
            const long long off_j = __shfl_sync(0xffffffffu, k_off, j);
            if (!((valid_mask >> j) & 1u)) continue;          // uniform over the warp
            const KVT* vrow = (const KVT*)p.pages + off_j + v_offset;
#pragma unroll
            for (int i = 0; i < PER_LANE; ++i) {
                const int c = lane + 32 * i;
                if (c < D) acc[i] = fmaf(pj, to_f32(vrow[c]), acc[i]);
            }
        }
    }
    OutT* orow = (OutT*)p.out + ((size_t)t * p.num_heads + h) * D;
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const int c = lane + 32 * i;
        if (c < D) orow[c] = from_f32<OutT>(acc[i] * inv);
    }
}

// A CTA per query token and up to R query heads of one kv head, which share every key and value read.  Tile t of 32 keys
// belongs to share t % SHARES, so that one decoded token's keys are read from many places at once; each share has its own
// running maximum, sum and accumulator per row, and they meet in the order of the shares at the end.  Scores: eight lanes a key,
// 16 bytes each, so that a warp's load takes whole 128-byte lines of four keys (a lane per key would touch 32 lines, and
// did: 390 us for two decoded tokens of 12 heads behind 300 keys, 730 us for a prompt of 333; now 14 and 67); a lane
// works on eight keys beside one another, and seven shuffles a row leave lane l with the score of key l.  Values: a lane per
// VW neighbouring columns, VW * 32 >= head size.
// What a row's bits are depends neither on R nor on how many of the CTA's WIDE warps share the work: a warp takes one share after
// the other.  Few rows (R 1, WIDE 8): a CTA a head, which waits for memory only, so all of a tile is asked for at once
// (FEW; six heads together: 35 us for the two decoded tokens).  Many rows fill the device with four warps each; eight would mostly
// idle where the keys are few (launch_rows has the measurements).
constexpr int SHARES = 8;

template <typename KVT> __device__ __forceinline__ float4 load4(const KVT* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}
template <typename KVT, int VW> __device__ __forceinline__ void load_columns(const KVT* p, float (&v)[VW]) {
    if constexpr (VW >= 4) {
#pragma unroll
        for (int i = 0; i < VW / 4; ++i) {
            const float4 x = load4(p + 4 * i);
            v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < VW; ++i) v[i] = to_f32(p[i]);
    }
}

template <typename KVT, int VW, int R, int WIDE, bool FEW>
__global__ void __launch_bounds__(WIDE * 32)
paged_attention_rows_kernel(AttnParams p, int q_bf16, int out_bf16, int chunks) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) float shared[];
    const int D = p.head_dim;
    float* q_s = shared;                                       // [R][D]
    float* acc_s = q_s + R * D;                                // [SHARES][R][D]
    float* m_s = acc_s + SHARES * R * D;                       // [SHARES][R]
    float* l_s = m_s + SHARES * R;
    float* p_s = l_s + SHARES * R + (threadIdx.x >> 5) * (R * 32);        // this warp's probabilities of a tile
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = p.num_heads / p.num_kv_heads;
    const int chunk = blockIdx.x % chunks, kvh = (blockIdx.x / chunks) % p.num_kv_heads, t = blockIdx.x / (chunks * p.num_kv_heads);
    const int h0 = kvh * group + chunk * R, rows = min(R, group - chunk * R);
    const int pos = p.positions[t], seq = p.token_seq[t];
    const int lo = first_visible_key(pos, p.window, p.chunk);
    const size_t page_stride = (size_t)2 * p.num_kv_heads * p.page_size * D;
    const size_t v_offset = (size_t)p.num_kv_heads * p.page_size * D;
    const int* table = p.block_table + (size_t)seq * p.max_blocks;
    const KVT* pages = (const KVT*)p.pages;
    const int first = lo / 32, last = pos / 32;
    auto page_of = [&](int kp) {
        const int block = kp / p.page_size;
        return block < p.max_blocks ? table[block] : -1;
    };
    auto offset_of = [&](int kp, int page) { return (long long)((size_t)page * page_stride + ((size_t)kvh * p.page_size + kp % p.page_size) * D); };
    if (FEW)                                                       // the warp's keys and values start on their way to L2 while the kernel in
        for (int tile = first + (warp - first % SHARES + SHARES) % SHARES; tile <= last; tile += SHARES) {        // front ends
            const int kp = tile * 32 + lane, page = kp >= lo && kp <= pos ? page_of(kp) : -1;
            if (page < 0 || page >= p.num_pages) continue;
            const char* row = (const char*)(pages + offset_of(kp, page));
            for (int b = 0; b < D * (int)sizeof(KVT); b += 128) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(row + b));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(row + v_offset * sizeof(KVT) + b));
            }
        }
    pdl_wait();                                                    // (positions and tables are older than the step's kernels)
    const size_t q_at = ((size_t)t * p.num_heads + h0) * D;
    for (int e = tid; e < R * D; e += WIDE * 32)
        q_s[e] = e >= rows * D ? 0.0f : q_bf16 ? to_f32(((const __nv_bfloat16*)p.q)[q_at + e]) : ((const float*)p.q)[q_at + e];
    __syncthreads();

    const int key_group = lane >> 3, c = lane & 7, pieces = D / 4;
    const bool column = lane * VW < D;

    for (int share = warp; share < SHARES; share += WIDE) {
        float acc[R][VW], m[R], l[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            m[r] = -INFINITY; l[r] = 0.0f;
#pragma unroll
            for (int i = 0; i < VW; ++i) acc[r][i] = 0.0f;
        }
        for (int tile = first + (share - first % SHARES + SHARES) % SHARES; tile <= last; tile += SHARES) {
            const int kp = tile * 32 + lane;
            bool valid = kp >= lo && kp <= pos;
            long long k_off = 0;                                   // (a key that is not visible is read from the pool's first row)
            if (valid) {
                const int page = page_of(kp);
                if (page < 0 || page >= p.num_pages) {
                    if (p.error_flag) atomicExch(p.error_flag, 2);
                    valid = false;
                } else {
                    k_off = offset_of(kp, page);
                }
            }
            float dot[R][8];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int j = 0; j < 8; ++j) dot[r][j] = 0.0f;
            long long key_at[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) key_at[j] = __shfl_sync(0xffffffffu, k_off, key_group * 8 + j);
            if (FEW && pieces <= 32) {                             // all of the lane's pieces of its eight keys at once
                float4 k[4][8];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (c + 8 * i < pieces) k[i][j] = load4(pages + key_at[j] + (c + 8 * i) * 4);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (c + 8 * i < pieces) {
                        const float4 q = *reinterpret_cast<const float4*>(q_s + (c + 8 * i) * 4);
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            dot[0][j] = fmaf(q.w, k[i][j].w, fmaf(q.z, k[i][j].z, fmaf(q.y, k[i][j].y, fmaf(q.x, k[i][j].x, dot[0][j]))));
                    }
            } else {
                for (int piece = c; piece < pieces; piece += 8) {
                    float4 k[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) k[j] = load4(pages + key_at[j] + piece * 4);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 q = *reinterpret_cast<const float4*>(q_s + r * D + piece * 4);
#pragma unroll
                        for (int j = 0; j < 8; ++j) dot[r][j] = fmaf(q.w, k[j].w, fmaf(q.z, k[j].z, fmaf(q.y, k[j].y, fmaf(q.x, k[j].x, dot[r][j]))));
                    }
                }
            }
            // The values ask for nothing that the scores make: in a row alone half of the tile's are on
            // their way while the scores meet, else a few at a time when they are needed.  (With the prefetch in front of the wait: decoding
            // two requests of 300 tokens in fp32, 12 heads of 128, 28 layers, four steps: 7,879 -> 7,342 us.)
            constexpr bool EARLY = FEW && VW <= 4;
            constexpr int BATCH = FEW ? 16 : 4;       // keys whose values are asked for together
            const unsigned seen = __ballot_sync(0xffffffffu, valid);
            float v[BATCH][VW];
            auto values = [&](int j0) {
#pragma unroll
                for (int j = 0; j < BATCH; ++j) {
                    const long long at = __shfl_sync(0xffffffffu, k_off, j0 + j);
                    if (column && ((seen >> (j0 + j)) & 1u)) {
                        load_columns<KVT, VW>(pages + at + v_offset + lane * VW, v[j]);
                    } else {
#pragma unroll
                        for (int i = 0; i < VW; ++i) v[j][i] = 0.0f;
                    }
                }
            };
            if (EARLY) values(0);
            __syncwarp();                                          // every lane is done with the last tile's probabilities
#pragma unroll
            for (int r = 0; r < R; ++r) {
                // lane c of a key group ends up with the sum over the group's lanes of dot[r][c]
                float a4[4], a2[2];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float keep = c & 4 ? dot[r][j + 4] : dot[r][j], give = c & 4 ? dot[r][j] : dot[r][j + 4];
                    a4[j] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float keep = c & 2 ? a4[j + 2] : a4[j], give = c & 2 ? a4[j] : a4[j + 2];
                    a2[j] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
                }
                const float keep = c & 1 ? a2[1] : a2[0], give = c & 1 ? a2[0] : a2[1];
                const float full = keep + __shfl_xor_sync(0xffffffffu, give, 1);
                const float s = valid ? full * p.scale : -INFINITY;
                const float m_new = fmaxf(m[r], warp_max(s));
                float prob = 0.0f;
                if (m_new != -INFINITY) {                          // else: no readable key in this tile yet
                    prob = valid ? expf(s - m_new) : 0.0f;
                    const float corr = m[r] == -INFINITY ? 0.0f : expf(m[r] - m_new);
                    l[r] = l[r] * corr + warp_sum(prob);
                    m[r] = m_new;
#pragma unroll
                    for (int i = 0; i < VW; ++i) acc[r][i] *= corr;
                }
                p_s[r * 32 + lane] = prob;
            }
            __syncwarp();
#pragma unroll (FEW ? 1 : 2)
            for (int j0 = 0; j0 < 32; j0 += BATCH) {
                if (!EARLY || j0 > 0) values(j0);
#pragma unroll
                for (int b = 0; b < BATCH; b += 4) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 w = *reinterpret_cast<const float4*>(p_s + r * 32 + j0 + b);
#pragma unroll
                        for (int i = 0; i < VW; ++i)
                            acc[r][i] = fmaf(w.w, v[b + 3][i], fmaf(w.z, v[b + 2][i], fmaf(w.y, v[b + 1][i], fmaf(w.x, v[b][i], acc[r][i]))));
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (column && m[r] != -INFINITY) {                     // (a share without keys is not read)
#pragma unroll
                for (int i = 0; i < VW; ++i) acc_s[(share * R + r) * D + lane * VW + i] = acc[r][i];
            }
            if (lane == 0) { m_s[share * R + r] = m[r]; l_s[share * R + r] = l[r]; }
        }
    }
    __syncthreads();
    for (int e = tid; e < rows * D; e += WIDE * 32) {
        const int r = e / D;
        float top = -INFINITY;
#pragma unroll
        for (int w = 0; w < SHARES; ++w) top = fmaxf(top, m_s[w * R + r]);
        float sum = 0.0f, value = 0.0f;
#pragma unroll
        for (int w = 0; w < SHARES; ++w) {
            const float mw = m_s[w * R + r];
            if (mw == -INFINITY) continue;
            const float f = expf(mw - top);
            sum = fmaf(l_s[w * R + r], f, sum);
            value = fmaf(acc_s[w * R * D + e], f, value);
        }
        const float o = value * (sum > 0.0f ? 1.0f / sum : 0.0f);
        if (out_bf16) ((__nv_bfloat16*)p.out)[q_at + e] = from_f32<__nv_bfloat16>(o);
        else ((float*)p.out)[q_at + e] = o;
    }
}

template <typename KVT, int VW, int R, int WIDE, bool FEW>
int launch_rows(const AttnParams& p, int q_bf16, int out_bf16, cudaStream_t stream) {
    static bool done[MAX_DEVICES] = {};
    auto kernel = paged_attention_rows_kernel<KVT, VW, R, WIDE, FEW>;
    const int d = device_index();
    constexpr int most = (R * VW * 32 * (SHARES + 1) + 2 * SHARES * R + WIDE * R * 32) * 4;
    if (!done[d]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) return check_launch("paged_attention_rows: shared memory");
        done[d] = true;
    }
    const int group = p.num_heads / p.num_kv_heads, chunks = (group + R - 1) / R;
    const long long blocks = (long long)p.tokens * p.num_kv_heads * chunks;
    if (blocks > 0x7fffffffll) return fail(MLB_UNSUPPORTED_SIZE, "paged_attention_plain: %d tokens are more than one launch takes", p.tokens);
    const size_t smem = (size_t)(R * p.head_dim * (SHARES + 1) + 2 * SHARES * R + WIDE * R * 32) * 4;
    launch_kernel(kernel, (unsigned)blocks, WIDE * 32, smem, stream, p, q_bf16, out_bf16, chunks);
    return check_launch("paged_attention_rows");
}

// Heads of a kv head together (at most four at head size 256, whose accumulators are long); one where there are few rows.
// Four warps a CTA instead of eight where the CTAs are many, two where besides no row has more than two tiles (the table's width).
// Measured on 148 SMs, us, fp32; heads / kv heads x head size, tokens of a prompt or (sequences x keys), eight warps -> four (-> two):
// 12/2x128: 64 11.9 -> 12.6, 333 73 -> 67, 300 x 20 49 -> 32 -> 30; 8/2x256: 333 75 -> 53; 14/2x64: 333 59 -> 53.  One head a kv head, where
// eight warps ask for all of a tile at once: 16/16x128: 30 x 300 63 -> 81, 64 34 -> 13, 333 243 -> 121, 300 x 20 203 -> 117 -> 74, 300 x 300
// 465 -> 428; 4/4x256: 333 105 -> 72, 300 x 300 226 -> 257 (eight warps spill 136 bytes at head sizes beyond 128, and still read best
// where rows are few: 17 for one token behind 300 keys).  Two to four heads of up to 64 columns: 8/4x64: 1,500 470 -> 522, 300 x 20
// 31 -> 19 -> 16 (four warps' CTAs leave less of L1 for keys that are read again): four only where the table holds few keys.
template <typename KVT, int VW>
int launch_rows(const AttnParams& p, int q_bf16, int out_bf16, cudaStream_t stream) {
    const int group = p.num_heads / p.num_kv_heads, sms = sm_count();
    const long long ctas = (long long)p.tokens * p.num_kv_heads * (VW == 8 ? (group + 3) / 4 : (group + 7) / 8);
    const long long keys = (long long)p.max_blocks * p.page_size;         // of a row at most
    if (p.tokens <= 2 * sms / p.num_heads || (group == 1 && ctas < 4 * sms)) return launch_rows<KVT, VW, 1, 8, true>(p, q_bf16, out_bf16, stream);
    const int wide = ctas < 2 * sms ? 8 : keys <= 64 ? 2 : VW > 2 || group == 1 || group > 4 || keys <= 128 ? 4 : 8;
    auto go = [&](auto r) {
        constexpr int R = decltype(r)::value;
        if (wide == 2) return launch_rows<KVT, VW, R, 2, false>(p, q_bf16, out_bf16, stream);
        if (wide == 4) return launch_rows<KVT, VW, R, 4, false>(p, q_bf16, out_bf16, stream);
        return launch_rows<KVT, VW, R, 8, false>(p, q_bf16, out_bf16, stream);
    };
    if (group == 1) return go(std::integral_constant<int, 1>());
    if constexpr (VW < 8)
        if (group > 4) return go(std::integral_constant<int, 8>());
    return go(std::integral_constant<int, 4>());
}

template <typename KVT>
int launch_rows(const AttnParams& p, int q_bf16, int out_bf16, cudaStream_t stream) {
    if (p.head_dim > 128) return launch_rows<KVT, 8>(p, q_bf16, out_bf16, stream);
    return p.head_dim > 64 ? launch_rows<KVT, 4>(p, q_bf16, out_bf16, stream) : launch_rows<KVT, 2>(p, q_bf16, out_bf16, stream);
}

}  // namespace

MLB_EXPORT int mlb_paged_attention_plain(const void* q, int q_dtype, const void* pages, int kv_dtype, void* out,
                                         int out_dtype, const int* positions, const int* token_seq,
                                         const int* block_table, int max_blocks, int num_pages, int page_size,
                                         int tokens, int num_heads, int num_kv_heads, int head_dim, int window, int chunk,
                                         float scale, int* error_flag, cudaStream_t stream) {
    if (tokens < 0 || num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads != 0)
        return fail(MLB_INVALID_ARGUMENT, "paged_attention_plain: bad head counts %d/%d", num_heads, num_kv_heads);
    if (head_dim <= 0 || head_dim > MAX_D)
        return fail(MLB_UNSUPPORTED_SIZE, "paged_attention_plain: head_dim %d not in 1..%d", head_dim, MAX_D);
    if (page_size <= 0 || num_pages <= 0 || max_blocks <= 0 || window < 0 || chunk < 0)
        return fail(MLB_INVALID_ARGUMENT, "paged_attention_plain: bad cache geometry");
    if (tokens == 0) return MLB_OK;
    AttnParams p{q, pages, out, positions, token_seq, block_table, max_blocks, num_pages, page_size,
                 tokens, num_heads, num_kv_heads, head_dim, chunk, window, scale, error_flag};
    const bool known = (q_dtype == MLB_F32 || q_dtype == MLB_BF16) && (out_dtype == MLB_F32 || (out_dtype == MLB_BF16 && q_dtype == MLB_BF16)) &&
                       (kv_dtype == MLB_BF16 || (kv_dtype == MLB_F32 && q_dtype == MLB_F32 && out_dtype == MLB_F32));
    if (known && head_dim % (head_dim > 128 ? 8 : 4) == 0 && (uintptr_t)pages % 16 == 0)
        return kv_dtype == MLB_F32 ? launch_rows<float>(p, q_dtype == MLB_BF16, out_dtype == MLB_BF16, stream)
                                   : launch_rows<__nv_bfloat16>(p, q_dtype == MLB_BF16, out_dtype == MLB_BF16, stream);
    const long long items = (long long)tokens * num_heads;
    const unsigned blocks = (unsigned)((items + WARPS - 1) / WARPS);
    if (q_dtype == MLB_F32 && kv_dtype == MLB_F32 && out_dtype == MLB_F32)
        launch_kernel(paged_attention_plain_kernel<float, float, float>, blocks, WARPS * 32, 0, stream, p);
    else if (q_dtype == MLB_BF16 && kv_dtype == MLB_BF16 && out_dtype == MLB_BF16)
        launch_kernel(paged_attention_plain_kernel<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>, blocks, WARPS * 32, 0, stream, p);
    else if (q_dtype == MLB_F32 && kv_dtype == MLB_BF16 && out_dtype == MLB_F32)
        launch_kernel(paged_attention_plain_kernel<float, __nv_bfloat16, float>, blocks, WARPS * 32, 0, stream, p);
    else if (q_dtype == MLB_BF16 && kv_dtype == MLB_BF16 && out_dtype == MLB_F32)
        launch_kernel(paged_attention_plain_kernel<__nv_bfloat16, __nv_bfloat16, float>, blocks, WARPS * 32, 0, stream, p);
    else
        return fail(MLB_INVALID_ARGUMENT, "paged_attention_plain: unsupported dtypes %d/%d/%d", q_dtype, kv_dtype, out_dtype);
    return check_launch("paged_attention_plain");
}
