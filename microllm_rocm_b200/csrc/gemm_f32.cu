// True 32-bit matrix product for the fp32 path:  C[M,N] (+)= A[M,K] * W[N,K]^T (+ bias[N]).
//
// CUDA cores only, plain fp32 FMA: no tensor cores, no TF32.  This is the role of the reference's readable matmul
// (src/ops/hip/basic_kernels.hip:319-336: one thread per output element, serial K loop).  W is kept in the checkpoint's own
// [out, in] layout (K contiguous); the reference transposes every linear weight to [in, out] at load
// (src/model/model.cpp:1928-1982).
//
// One order of additions for every M, tile and kernel, so that a row's bits do not depend on what else is in the batch: K is
// cut into sixteen ranges of range_length(K) elements; a range is summed in two chains, its even and its odd elements in
// increasing order, then even + odd; four consecutive ranges are added up in order to a quarter, the four quarters in order
// to the result, then the bias.  The ranges are what lets a product of few rows stream W from many threads at once and what a
// cluster of four CTAs shares; the two chains are the halves of a packed fma (two fp32 FMAs an instruction, each rounded as
// always).  Shorter chains also round less: the logits of 28 layers at K = 1,536 / 8,960 stood 9e-6 off 64-bit ones with one
// serial chain over K.
//
//   gemm_f32_stream_kernel   up to STREAM_MAX_M rows: bound by reading W once.  Eight (or sixteen) rows of W a CTA, one warp a quarter of K,
//                            a lane per (row, range), W and A through a ring of 32-element pieces by cp.async.
//   gemm_f32_tile_kernel     more rows: bound by the FMA pipe.  64 x 64 outputs a cluster of four CTAs, a quarter of K each, 8 x 4
//                            outputs a thread; the quarters meet through distributed shared memory.
//
// Products of a step of 28 layers (1,536 wide, 8,960 inside, 151,936-row head) on a B200: two rows 1.31 ms, 4.7 TB/s of weights (51 ms with one 64 x
// 64 tile kernel for every M, whose sixteen column threads held idle rows and whose grid left most SMs empty); 333 rows
// 29 ms, 30 TFLOP/s (77 ms).  STREAM_MAX_M, measured (us, streamed / tiled): 17 .. 32 rows (two passes over W) 1,536 -> 2,048 16 / 36,
// 8,960 -> 1,536 78 / 160, 1,536 -> 17,920 124 / 109; 33 .. 48 rows (three) 23 / 34, 79 / 160, 183 / 108; 64 rows 31 / 34, 117 / 160, 240 / 107: the
// narrow products gain with every pass less, the wide one loses from the second on, and the products of a layer together are
// even at about 48 rows (16 rows: 8 / 37, 40 / 160, 64 / 111).
#include <cooperative_groups.h>

#include "common.cuh"

using namespace mlb;
namespace cg = cooperative_groups;

MLB_DEFINE_LAST_ERROR()

namespace {

constexpr int QUARTERS = 4, RANGES = 4;              // quarters of K, ranges of a quarter
constexpr int STEP = 32;                             // elements of K that travel at a time; a range is a whole number of them

__host__ __device__ __forceinline__ int range_length(int K) {
    constexpr int n = QUARTERS * RANGES * STEP;
    return (K + n - 1) / n * STEP;
}

__device__ __forceinline__ void copy16(unsigned dst, const void* src, int bytes) {      // bytes < 16: the rest is zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copy4(unsigned dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void wait_groups() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// four elements of a row from k on, into 16 bytes of shared memory; elements at or behind K are zero.  A row whose start is not
// on 16 bytes travels in fours.
template <bool VEC>
__device__ __forceinline__ void copy_piece(unsigned dst, const float* row, int k, int K) {
    const int left = K - k;
    if (VEC) {
        copy16(dst, left > 0 ? row + k : row, left >= 4 ? 16 : left > 0 ? left * 4 : 0);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) copy4(dst + 4 * i, left > i ? row + k + i : row, left > i ? 4 : 0);
    }
}

// the even and the odd chain of one output, in the halves of a register pair
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long w) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(w));
}
__device__ __forceinline__ float chains(unsigned long long acc) {
    return __uint_as_float((unsigned)acc) + __uint_as_float((unsigned)(acc >> 32));
}

// ------------------------------------------------------------------------------------------------------- few rows of A
// Lane (r, g) of warp q: rows r (and r + 8) of the CTA's rows of W, range g of quarter q.  A stage of the warp's own ring
// holds the next STEP elements of the four ranges: of 8 * ROWS rows of W (the 16-byte pieces of a row's span turned by the row, so that
// eight lanes that read the same piece of eight rows meet no bank twice) and of MT rows of A (read by all lanes of a range
// at once).  Nothing but the end of the kernel joins the warps.
constexpr int STREAM_MAX_M = 32;

template <int MT, int ROWS> struct StreamShape {
    static constexpr int STAGE_BYTES = (8 * ROWS + MT) * RANGES * STEP * 4;
    static constexpr int STAGES = STAGE_BYTES > 12288 ? 3 : 4;
    static constexpr int SMEM = QUARTERS * STAGES * STAGE_BYTES;
};

template <int MT, int ROWS, bool VEC, bool ACCUMULATE>
__global__ void __launch_bounds__(QUARTERS * 32)
gemm_f32_stream_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                       float* __restrict__ C, int M, int N, int K, long long lda, long long ldw, long long ldc, int w_constant) {
    using Shape = StreamShape<MT, ROWS>;
    constexpr int STAGES = Shape::STAGES, SPAN = STEP * 4, W_BYTES = 8 * ROWS * RANGES * SPAN;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ float quarter[QUARTERS][MT][8 * ROWS];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * (8 * ROWS), m0 = blockIdx.y * MT;
    const int length = range_length(K), steps = length / STEP;
    const int k_base = warp * RANGES * length;
    unsigned char* ring = smem + warp * STAGES * Shape::STAGE_BYTES;
    const unsigned ring_addr = (unsigned)__cvta_generic_to_shared(ring);

    auto load_w = [&](int step) {
        const unsigned base = ring_addr + (step % STAGES) * Shape::STAGE_BYTES;
#pragma unroll
        for (int i = 0; i < 8 * ROWS; ++i) {
            const int e = i * 32 + lane, piece = e & 7, r = (e >> 3) & 7, rest = e >> 6;       // rest = range + RANGES * (row / 8)
            const int g = rest % RANGES, n = n0 + r + 8 * (rest / RANGES);
            copy_piece<VEC>(base + (e >> 3) * SPAN + ((piece ^ r) << 4), W + (size_t)min(n, N - 1) * ldw,
                            k_base + g * length + step * STEP + piece * 4, K);
        }
    };
    auto load_a = [&](int step) {
        const unsigned base = ring_addr + (step % STAGES) * Shape::STAGE_BYTES + W_BYTES;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int g = lane >> 3, piece = lane & 7, m = m0 + i;
            copy_piece<VEC>(base + (i * RANGES + g) * SPAN + piece * 16, A + (size_t)min(m, M - 1) * lda,
                            k_base + g * length + step * STEP + piece * 4, K);
        }
    };
    if (!w_constant) pdl_wait();
    for (int s = 0; s < STAGES - 1; ++s)
        if (s < steps) load_w(s);
    if (w_constant) pdl_wait();                       // only A comes from a kernel of the same step
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load_a(s);
        commit();                                     // (the first group holds W of every stage in front of it)
    }

    unsigned long long acc[ROWS][MT];
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[i][m] = 0ull;
    const int r = lane & 7, g = lane >> 3;
    for (int step = 0; step < steps; ++step) {
        wait_groups<STAGES - 2>();
        __syncwarp();
        const unsigned char* base = ring + (step % STAGES) * Shape::STAGE_BYTES;
#pragma unroll
        for (int piece = 0; piece < STEP / 4; ++piece) {
            ulonglong2 w[ROWS];
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
                w[i] = *reinterpret_cast<const ulonglong2*>(base + ((i * RANGES + g) * 8 + r) * SPAN + ((piece ^ r) << 4));
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(base + W_BYTES + (m * RANGES + g) * SPAN + piece * 16);
#pragma unroll
                for (int i = 0; i < ROWS; ++i) { fma2(acc[i][m], a.x, w[i].x); fma2(acc[i][m], a.y, w[i].y); }
            }
        }
        __syncwarp();                                 // the stage that is filled next was read by every lane
        if (step + STAGES - 1 < steps) { load_w(step + STAGES - 1); load_a(step + STAGES - 1); }
        commit();
    }
    // ranges of a quarter: lanes r, r + 8, r + 16, r + 24; quarters: the warps
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float v = chains(acc[i][m]);
            float q = __shfl_sync(0xffffffffu, v, r);
#pragma unroll
            for (int j = 1; j < RANGES; ++j) q += __shfl_sync(0xffffffffu, v, r + 8 * j);
            if (g == 0) quarter[warp][m][r + 8 * i] = q;
        }
    __syncthreads();
    for (int e = threadIdx.x; e < MT * 8 * ROWS; e += QUARTERS * 32) {
        const int m = e / (8 * ROWS), j = e % (8 * ROWS);
        if (m0 + m >= M || n0 + j >= N) continue;
        float v = quarter[0][m][j];
#pragma unroll
        for (int q = 1; q < QUARTERS; ++q) v += quarter[q][m][j];
        if (bias) v += bias[n0 + j];
        float* dst = C + (size_t)(m0 + m) * ldc + n0 + j;
        *dst = ACCUMULATE ? (*dst + v) : v;
    }
}

// ------------------------------------------------------------------------------------------------------- many rows of A
// Rows of a stage lie 36 floats apart: eight neighbouring rows' same piece fall into eight different groups of banks.  Per four
// elements of K a thread reads RI + 4 pieces of 16 bytes and issues 8 RI packed FMAs (RI = 5 to 8, an eighth of the tile's rows): full tiles reach 38
// of the FMA pipe's 74 TFLOP/s, the reads of shared memory beside it.
constexpr int BN = 64, TILE_STAGES = 3, PITCH = STEP + 4;
constexpr int stage_floats(int ri) { return (8 * ri + BN) * PITCH; }
constexpr int tile_smem(int ri) { return TILE_STAGES * stage_floats(ri) * 4; }

template <int RI, bool VEC, bool ACCUMULATE>
__global__ void __launch_bounds__(128)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ C, int M, int N, int K, long long lda, long long ldw, long long ldc, int w_constant) {
    extern __shared__ __align__(128) float tiles[];
    constexpr int BM = 8 * RI, STAGE_FLOATS = stage_floats(RI);
    pdl_prologue();
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quarter = blockIdx.x % QUARTERS;                            // = the CTA's rank in its cluster
    const int n0 = (blockIdx.x / QUARTERS) * BN, m0 = blockIdx.y * BM;
    const int length = range_length(K), per_range = length / STEP;
    const int k_base = quarter * RANGES * length;
    const int steps = max(0, min(RANGES * per_range, (K - k_base + STEP - 1) / STEP));      // those that hold any of K
    const unsigned tiles_addr = (unsigned)__cvta_generic_to_shared(tiles);

    // a stage: 64 + 64 rows of eight pieces; this thread copies piece tid % 8 of every sixteenth row
    const int piece = tid & 7, row = tid >> 3;
    auto load = [&](int step) {
        const unsigned base = tiles_addr + (step % TILE_STAGES) * (STAGE_FLOATS * 4) + piece * 16;
        const int k = k_base + step * STEP + piece * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (row + 16 * i < BM) copy_piece<VEC>(base + (row + 16 * i) * (PITCH * 4), A + (size_t)min(m0 + row + 16 * i, M - 1) * lda, k, K);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            copy_piece<VEC>(base + (BM + row + 16 * i) * (PITCH * 4), W + (size_t)min(n0 + row + 16 * i, N - 1) * ldw, k, K);
    };
    for (int s = 0; s < TILE_STAGES - 1; ++s) {
        if (s < steps) load(s);
        commit();
    }
    const int ty = lane >> 3, tx = lane & 7;                              // rows ty + 4 i, columns tx + 8 j of the warp's 4 RI x 32
    const int a_row = (warp >> 1) * (4 * RI) + ty, w_row = (warp & 1) * 32 + tx;
    unsigned long long acc[RI][4];
    float sum[RI][4];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) { acc[i][j] = 0ull; sum[i][j] = 0.0f; }
    int in_range = 0;
    for (int step = 0; step < steps; ++step) {
        wait_groups<TILE_STAGES - 2>();
        __syncthreads();                                                  // everybody's pieces are there, and the stage before was read
        if (step + TILE_STAGES - 1 < steps) load(step + TILE_STAGES - 1);
        commit();
        const float* a_base = tiles + (step % TILE_STAGES) * STAGE_FLOATS + a_row * PITCH;
        const float* w_base = tiles + (step % TILE_STAGES) * STAGE_FLOATS + (BM + w_row) * PITCH;
#pragma unroll
        for (int p = 0; p < STEP / 4; ++p) {
            ulonglong2 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(w_base + 8 * j * PITCH + 4 * p);
#pragma unroll
            for (int i = 0; i < RI; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(a_base + 4 * i * PITCH + 4 * p);
#pragma unroll
                for (int j = 0; j < 4; ++j) { fma2(acc[i][j], a.x, w[j].x); fma2(acc[i][j], a.y, w[j].y); }
            }
        }
        if (++in_range == per_range || step + 1 == steps) {
            in_range = 0;
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) { sum[i][j] += chains(acc[i][j]); acc[i][j] = 0ull; }
        }
    }
    wait_groups<0>();
    __syncthreads();
    constexpr int OUT_PITCH = BN + 4;
    float* mine = tiles;                                                  // the quarter's 8 RI x 64 sums, over the ring
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mine[(a_row + 4 * i) * OUT_PITCH + w_row + 8 * j] = sum[i][j];
    cluster.sync();
    const float* part[QUARTERS];
#pragma unroll
    for (int q = 0; q < QUARTERS; ++q) part[q] = cluster.map_shared_rank(mine, q);
    for (int e = tid; e < (BM / QUARTERS) * BN; e += 128) {
        const int i = quarter * (BM / QUARTERS) + e / BN, j = e % BN;
        if (m0 + i >= M || n0 + j >= N) continue;
        float v = part[0][i * OUT_PITCH + j];
#pragma unroll
        for (int q = 1; q < QUARTERS; ++q) v += part[q][i * OUT_PITCH + j];
        if (bias) v += bias[n0 + j];
        float* dst = C + (size_t)(m0 + i) * ldc + n0 + j;
        *dst = ACCUMULATE ? (*dst + v) : v;
    }
    cluster.sync();                                                       // nobody leaves while its sums are read
}

struct Call {
    const float *A, *W, *bias;
    float* C;
    int M, N, K;
    long long lda, ldw, ldc;
    int w_constant;
    cudaStream_t stream;
};

template <typename Kernel>
int set_smem(Kernel kernel, int bytes, bool* done) {
    const int d = device_index();
    if (!done[d]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
            return check_launch("gemm_f32: shared memory");
        done[d] = true;
    }
    return MLB_OK;
}

template <int MT, int ROWS, bool VEC, bool ACCUMULATE>
int launch_stream(const Call& c) {
    static bool done[MAX_DEVICES] = {};
    auto kernel = gemm_f32_stream_kernel<MT, ROWS, VEC, ACCUMULATE>;
    constexpr int smem = StreamShape<MT, ROWS>::SMEM;
    if (int status = set_smem(kernel, smem, done)) return status;
    const dim3 grid((c.N + 8 * ROWS - 1) / (8 * ROWS), (c.M + MT - 1) / MT);
    launch_kernel(kernel, grid, QUARTERS * 32, smem, c.stream, c.A, c.W, c.bias, c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc, c.w_constant);
    return check_launch("gemm_f32_stream");
}

// Eighths of a tile's rows: equal tiles of at most 64 rows, five to eight for more than STREAM_MAX_M.  A last tile of 64 rows that holds 13
// (333 rows) takes as long as a full one: six of 56 take 945 us where six of 64 take 1,061 (the four products of a layer of the 1.5B
// shape; 33 rows 195 / 264, 65 305 / 432, 200 625 / 704, 500 and 1,000 the same).
int tile_rows(int M) {
    const int count = (M + 63) / 64;
    return ((M + count - 1) / count + 7) / 8;
}

template <int RI, bool VEC, bool ACCUMULATE>
int launch_tile(const Call& c) {
    static bool done[MAX_DEVICES] = {};
    auto kernel = gemm_f32_tile_kernel<RI, VEC, ACCUMULATE>;
    constexpr int smem = tile_smem(RI);
    if (int status = set_smem(kernel, smem, done)) return status;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((c.N + BN - 1) / BN * QUARTERS, (c.M + 8 * RI - 1) / (8 * RI));
    config.blockDim = 128;
    config.dynamicSmemBytes = smem;
    config.stream = c.stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = QUARTERS;
    attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&config, kernel, c.A, c.W, c.bias, c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc, c.w_constant);
    return check_launch("gemm_f32_tile");
}

template <bool VEC, bool ACCUMULATE>
int launch(const Call& c) {
    if (c.M == 1) return launch_stream<1, 1, VEC, ACCUMULATE>(c);
    if (c.M == 2) return launch_stream<2, 1, VEC, ACCUMULATE>(c);
    if (c.M <= 4) return launch_stream<4, 1, VEC, ACCUMULATE>(c);
    if (c.M <= 8) return launch_stream<8, 2, VEC, ACCUMULATE>(c);
    if (c.M <= STREAM_MAX_M) return launch_stream<16, 2, VEC, ACCUMULATE>(c);
    switch (tile_rows(c.M)) {
        case 5: return launch_tile<5, VEC, ACCUMULATE>(c);
        case 6: return launch_tile<6, VEC, ACCUMULATE>(c);
        case 7: return launch_tile<7, VEC, ACCUMULATE>(c);
        default: return launch_tile<8, VEC, ACCUMULATE>(c);
    }
}

}  // namespace

// accumulate != 0:  C += A*W^T (+bias)   (the residual add of the o/down projections)
// w_constant != 0: no kernel that may still run in front of this one on the stream writes W, so W may be read before the
// dependency wait
MLB_EXPORT int mlb_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                            long long lda, long long ldw, long long ldc, int accumulate, int w_constant, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N)
        return fail(MLB_INVALID_ARGUMENT, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    if (M == 0) return MLB_OK;
    if ((M + 63) / 64 > 65535) return fail(MLB_UNSUPPORTED_SIZE, "gemm_f32: M=%d exceeds %d rows per call", M, 65535 * 64);
    const Call c{A, W, bias, C, M, N, K, lda, ldw, ldc, w_constant, stream};
    const bool vec = lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0;
    if (vec) return accumulate ? launch<true, true>(c) : launch<true, false>(c);
    return accumulate ? launch<false, true>(c) : launch<false, false>(c);
}
