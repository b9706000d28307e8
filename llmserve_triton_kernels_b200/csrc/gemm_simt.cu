// y[M, N] = x[M, K] * w[N, K]^T on the CUDA cores with 32-bit fused multiply-adds.
//
// This is the matrix product of the true 32-bit path (no tensor cores, no reduced-precision
// mode), and it takes every size.  Each output element is a sum of parts, one for every 16 k: a
// part is accumulated by one thread in ascending k, and the parts are added up in ascending order,
// so a row's result does not depend on how many other rows are in the batch, where the row lies in
// it, or which of the three kernels below ran:
//
//   gemm_simt_kernel       any type, any size, any alignment: 64 x 64 outputs a CTA.
//   gemm_f32_tile_kernel   32-bit operands whose rows start on 16 bytes, many rows: bound by the CUDA cores, 64 multiply-adds for
//                          4 shared-memory loads of 16 bytes and k.
//   gemm_f32_few_kernel    the same operands, up to 16 rows (decode steps): bound by reading w once.  The parts of an output
//                          do not depend on one another, so a warp's lanes and a CTA's warps take different parts of 16
//                          features; only the adding up is one thread's.
//
// What each measured stands at launch_f32.
#include "common.cuh"
#include "tma.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4, THREADS = 256;

template <typename TX, typename TW, typename TO>
__global__ void __launch_bounds__(THREADS)
gemm_simt_kernel(const TX* __restrict__ x, const TW* __restrict__ w, TO* __restrict__ out, int M, int N, int K,
                 int ldx, int ldw, int ldo, long long x_batch, long long w_batch, long long o_batch) {
    x += (long long)blockIdx.z * x_batch;  // one product per z: operands and result a fixed stride apart
    w += (long long)blockIdx.z * w_batch;
    out += (long long)blockIdx.z * o_batch;
    __shared__ float xs[BK][BM + 4];
    __shared__ float ws[BK][BN + 4];
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tid = threadIdx.x;
    const int tx = tid % (BN / TN), ty = tid / (BN / TN);
    const int lrow = tid / 4, lk = (tid % 4) * 4;  // each thread stages 4 consecutive k of one row

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = k0 + lk + e;
            const int m = m0 + lrow, n = n0 + lrow;
            xs[lk + e][lrow] = (m < M && k < K) ? to_float(x[(size_t)m * ldx + k]) : 0.f;
            ws[lk + e][lrow] = (n < N && k < K) ? to_float(w[(size_t)n * ldw + k]) : 0.f;
        }
        __syncthreads();
        // a partial sum per k-tile, then one addition into the total: the rounding error grows with
        // sqrt(K / BK) instead of sqrt(K), and the order is still fixed
        float part[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) part[i][j] = 0.f;
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = xs[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) part[i][j] = fmaf(a[i], b[j], part[i][j]);
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] += part[i][j];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n < N) out[(size_t)m * ldo + n] = from_float<TO>(acc[i][j]);
        }
    }
}

__device__ __forceinline__ void copy16_async(float* dst, const float* src, bool valid) {
    // a copy of no bytes fills the 16 with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(tma::smem_addr(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// RM x RN outputs a CTA, TR x TC of them a thread: rows ty + i * (RM / TR), columns tx + j * (RN / TC), so that the lanes of
// a warp read neighbouring rows of the staged tiles, which lie 20 words apart and thus in different banks.  A tile of BK = 16 k
// (one part of every output) a stage, STAGES of them on their way by cp.async.
template <int RM, int RN, int TR, int TC, int STAGES>
__global__ void __launch_bounds__((RM / TR) * (RN / TC))
gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out, int M, int N, int K,
                     int ldx, int ldw, int ldo) {
    constexpr int TX = RN / TC, TY = RM / TR, NT = TX * TY, ROW = BK + 4;
    extern __shared__ __align__(16) float tiles[];  // [STAGES][RM + RN][ROW]
    const int m0 = blockIdx.y * RM, n0 = blockIdx.x * RN;
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int kt = (K + BK - 1) / BK;
    auto fetch = [&](int t) {
        if (t < kt) {
            float* st = tiles + (size_t)(t % STAGES) * (RM + RN) * ROW;
            constexpr int PIECES = (RM + RN) * (BK / 4);
#pragma unroll
            for (int i = 0; i < (PIECES + NT - 1) / NT; ++i) {
                const int piece = tid + i * NT;
                if (PIECES % NT != 0 && piece >= PIECES) break;
                const int row = piece / (BK / 4), k = t * BK + (piece % (BK / 4)) * 4;
                // rows beyond the matrices are read as their last one and never stored
                const float* src = row < RM ? x + (size_t)min(m0 + row, M - 1) * ldx + k : w + (size_t)min(n0 + row - RM, N - 1) * ldw + k;
                copy16_async(st + row * ROW + (piece % (BK / 4)) * 4, k < K ? src : x, k < K);
            }
        }
        copies_commit();
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    float acc[TR][TC];
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
        for (int j = 0; j < TC; ++j) acc[i][j] = 0.f;
    for (int t = 0; t < kt; ++t) {
        copies_wait<STAGES - 2>();
        __syncthreads();  // tile t has arrived, and everyone is done with tile t - 1, whose place tile t + STAGES - 1 takes
        fetch(t + STAGES - 1);
        const float* xs = tiles + (size_t)(t % STAGES) * (RM + RN) * ROW + ty * ROW;
        const float* ws = tiles + (size_t)(t % STAGES) * (RM + RN) * ROW + (RM + tx) * ROW;
        float part[TR][TC];
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) part[i][j] = 0.f;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            float a[TR][4];
#pragma unroll
            for (int i = 0; i < TR; ++i) load4(xs + i * TY * ROW + kk, a[i]);
#pragma unroll
            for (int j = 0; j < TC; ++j) {
                float b[4];
                load4(ws + j * TX * ROW + kk, b);
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int i = 0; i < TR; ++i) part[i][j] = fmaf(a[i][e], b[e], part[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) acc[i][j] += part[i][j];
    }
    copies_wait<0>();
#pragma unroll
    for (int i = 0; i < TR; ++i) {
        const int m = m0 + ty + i * TY;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TC; ++j) {
            const int n = n0 + tx + j * TX;
            if (n < N) out[(size_t)m * ldo + n] = acc[i][j];
        }
    }
}

// Up to MR rows.  A CTA owns 16 features; stages of 256 k (16 parts) of them and of x arrive by cp.async.  Lanes 0-15 and 16-31
// of a warp hold the 16 features and one part each, eight warps the 16 parts of a stage; the parts meet in shared memory, where
// thread (feature, row) adds them up in order while the other warps are at the next stage.
constexpr int FEW_N = 16, FEW_K = 256, FEW_THREADS = 256, FEW_ROW = FEW_K + 4, FEW_PARTS = FEW_K / BK;

template <int MR, int STAGES>
constexpr size_t few_bytes() {
    return ((size_t)STAGES * (FEW_N + MR) * FEW_ROW + 2 * (size_t)FEW_PARTS * MR * FEW_N) * sizeof(float);
}

template <int MR, int STAGES>
__global__ void __launch_bounds__(FEW_THREADS)
gemm_f32_few_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out, int M, int N, int K,
                    int ldx, int ldw, int ldo) {
    extern __shared__ __align__(16) float tiles[];  // [STAGES][FEW_N + MR][FEW_ROW], then [2][FEW_PARTS][MR][FEW_N]
    float* parts = tiles + (size_t)STAGES * (FEW_N + MR) * FEW_ROW;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * FEW_N, stages = (K + FEW_K - 1) / FEW_K;
    auto fetch_rows = [&](int s, bool of_w) {
        float* st = tiles + (size_t)(s % STAGES) * (FEW_N + MR) * FEW_ROW + (of_w ? 0 : FEW_N * FEW_ROW);
        const int rows = of_w ? FEW_N : MR;
        for (int piece = tid; piece < rows * (FEW_K / 4); piece += FEW_THREADS) {
            const int row = piece / (FEW_K / 4), k = s * FEW_K + (piece % (FEW_K / 4)) * 4;
            const float* src = of_w ? w + (size_t)min(n0 + row, N - 1) * ldw + k : x + (size_t)min(row, M - 1) * ldx + k;
            copy16_async(st + row * FEW_ROW + (piece % (FEW_K / 4)) * 4, k < K ? src : w, k < K);
        }
    };
    // w may be the work of the kernel in front: its first stages are brought into L2, where what that kernel still writes is seen, before that
    // kernel's end, and copied from there behind it
    if (tid < FEW_N)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(w + (size_t)min(n0 + tid, N - 1) * ldw), "r"(min(K, (STAGES - 1) * FEW_K) * 4) : "memory");
    pdl_trigger();
    pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < stages) {
            fetch_rows(s, true);
            fetch_rows(s, false);
        }
        copies_commit();
    }
    float acc = 0.f;
    const int an = tid % FEW_N, am = tid / FEW_N;  // the output that this thread adds up (am < MR)
    const int pn = lane % FEW_N, pt = warp * 2 + lane / FEW_N;
    for (int s = 0; s < stages; ++s) {
        copies_wait<STAGES - 2>();
        __syncthreads();  // stage s has arrived; stage s - 1 and the parts of stage s - 2 have been read
        if (s + STAGES - 1 < stages) {
            fetch_rows(s + STAGES - 1, true);
            fetch_rows(s + STAGES - 1, false);
        }
        copies_commit();
        const float* ws = tiles + (size_t)(s % STAGES) * (FEW_N + MR) * FEW_ROW + pn * FEW_ROW + pt * BK;
        const float* xs = tiles + (size_t)(s % STAGES) * (FEW_N + MR) * FEW_ROW + FEW_N * FEW_ROW + pt * BK;
        float part[MR];
#pragma unroll
        for (int m = 0; m < MR; ++m) part[m] = 0.f;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            float b[4];
            load4(ws + kk, b);
#pragma unroll
            for (int m = 0; m < MR; ++m) {
                float a[4];
                load4(xs + m * FEW_ROW + kk, a);
#pragma unroll
                for (int e = 0; e < 4; ++e) part[m] = fmaf(a[e], b[e], part[m]);
            }
        }
        float* mine = parts + (size_t)(s & 1) * FEW_PARTS * MR * FEW_N;
#pragma unroll
        for (int m = 0; m < MR; ++m) mine[(pt * MR + m) * FEW_N + pn] = part[m];
        __syncthreads();
        if (am < MR) {
            float v[FEW_PARTS];
#pragma unroll
            for (int t = 0; t < FEW_PARTS; ++t) v[t] = mine[(t * MR + am) * FEW_N + an];
            // parts beyond K are sums of zeros, which change nothing
#pragma unroll
            for (int t = 0; t < FEW_PARTS; ++t) acc += v[t];
        }
    }
    copies_wait<0>();
    if (am < M && n0 + an < N) out[(size_t)am * ldo + n0 + an] = acc;
}

template <int RM, int RN, int TR, int TC, int STAGES>
int launch_tile(const float* x, const float* w, float* out, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    constexpr size_t smem = (size_t)STAGES * (RM + RN) * (BK + 4) * sizeof(float);
    auto kernel = gemm_f32_tile_kernel<RM, RN, TR, TC, STAGES>;
    if (smem > 48 * 1024) {  // at every launch: the limit holds for the current device, and a process may have several
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    kernel<<<dim3((N + RN - 1) / RN, (M + RM - 1) / RM), (RM / TR) * (RN / TC), smem, stream>>>(x, w, out, M, N, K, ldx, ldw, ldo);
    return launch_status();
}

template <int MR, int STAGES>
int launch_few(const float* x, const float* w, float* out, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    constexpr size_t smem = few_bytes<MR, STAGES>();
    auto kernel = gemm_f32_few_kernel<MR, STAGES>;
    if (smem > 48 * 1024) {  // at every launch: the limit holds for the current device, and a process may have several
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    return launch_pdl(kernel, dim3((N + FEW_N - 1) / FEW_N), dim3(FEW_THREADS), smem, stream, x, w, out, M, N, K, ldx, ldw, ldo);
}

// 32-bit operands whose rows start on 16 bytes and hold a multiple of 4 k.  The kernel and its tile do not show in the result.
// Up to 16 rows the weights' bytes bound the product, beyond that the CUDA cores do.  Measured on a B200, every launch behind a
// 256 MB write (microseconds): 2 rows of the gate and up product of a 1.1B model (11,264 x 2,048) 33, 2.8 TB/s, and of the output
// matrix (32,000 x 2,048) 64, 4.1 TB/s; 242 rows 320, 35 TFLOP/s, of the down product (2,048 x 5,632) 227; 1,000 rows of the
// output matrix 3,167, 41 TFLOP/s.  The 64 x 64 kernel above, which ran them all, took 279 on average over a decode step's and
// a 242-row prompt's products, these 72.
int launch_f32(const float* x, const float* w, float* out, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    if (M <= 1) return launch_few<1, 4>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    if (M <= 2) return launch_few<2, 4>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    if (M <= 4) return launch_few<4, 4>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    if (M <= 8) return launch_few<8, 3>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    if (M <= 16) return launch_few<16, 3>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    // the tile that takes the least time by how many of them the busiest SM has.  Measured (2,048 k, 17 to 300 rows of 1,024 to 11,264
    // features, microseconds; n tiles of an SM): 232 n, 145 n, 27 + 59 n and 32 + 31 n.  242 rows: 2,560 features 145 with 64 x 64, 118 with 32 x 64;
    // 2,048 features 88 and 104; 11,264 features 322 and 338.  Against the rule before (the areas of the busiest SM's tiles at assumed rates): 11,264
    // features, 200 rows 365 -> 310, 300 479 -> 377, 512 709 -> 604; 2,048 features, 700 rows 197 -> 173; most sizes as they were.
    // From 64 to 8,192 k (571 products, 17 to 2,000 rows of 256 to 32,000 features) every tile's time is in proportion to k, so the choice does
    // not depend on it: from 1,024 k on it is 0.2 % off the fastest tile on average and 16 at the most (at 5,632 k 0.1 and 3, the rule before 3.1 and
    // 29).  Below, the mean is 3 % (before: 3 as well) and single products are up to 60 % off, all with a last tile that stands beyond the matrix: its
    // threads read the last row over and over, all from one place of L2 (256 k, 200 rows of 2,048 features: 29.8 with 64 x 64, 18.5 with 32 x 64; 242 rows:
    // 16.4 and 18.5).  Zeros there, other rows, or last tiles that end with the matrix cost full tiles of 64 x 64 1 to 9 %.  64 x 128 is chosen where it ties
    // with two tiles of 64 x 64 an SM, and is 1 to 11 % faster than they are there (200 rows of 4,096 features: 153.6 and 163.9).
    struct { int rm, rn; double once, each; } const kinds[4] = {{128, 128, 0., 232.}, {64, 128, 0., 145.}, {64, 64, 27., 59.}, {32, 64, 32., 31.}};
    int best = 0;
    double best_cost = 1e30;
    const int sms = device_sms();
    for (int i = 0; i < 4; ++i) {
        const long long tiles = (long long)((M + kinds[i].rm - 1) / kinds[i].rm) * ((N + kinds[i].rn - 1) / kinds[i].rn);
        const double cost = kinds[i].once + kinds[i].each * (double)((tiles + sms - 1) / sms);
        if (cost < best_cost) {
            best_cost = cost;
            best = i;
        }
    }
    if (best == 0) return launch_tile<128, 128, 8, 8, 4>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    if (best == 1) return launch_tile<64, 128, 8, 8, 4>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    if (best == 2) return launch_tile<64, 64, 4, 8, 4>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    return launch_tile<32, 64, 4, 4, 4>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
}

template <typename TX, typename TW, typename TO>
int launch(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int ldw, int ldo,
           cudaStream_t stream, int batches = 1, long long x_batch = 0, long long w_batch = 0, long long o_batch = 0) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batches);
    gemm_simt_kernel<TX, TW, TO><<<grid, THREADS, 0, stream>>>((const TX*)x, (const TW*)w, (TO*)out, M, N, K, ldx,
                                                               ldw, ldo, x_batch, w_batch, o_batch);
    return launch_status();
}

}  // namespace

LLM_EXPORT int llm_gemm_simt(const void* x, int x_dtype, const void* w, int w_dtype, void* out, int out_dtype, int M,
                             int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K < 0 || ldx < K || ldw < K || ldo < N) return LLM_ERR_BAD_ARGUMENT;
    if ((M + BM - 1) / BM > 65535) return LLM_ERR_UNSUPPORTED;
    using bf = __nv_bfloat16;
    if (x_dtype == LLM_F32 && w_dtype == LLM_F32 && out_dtype == LLM_F32) {
        if (K > 0 && !((K | ldx | ldw) & 3) && !(((uintptr_t)x | (uintptr_t)w) & 15))
            return launch_f32((const float*)x, (const float*)w, (float*)out, M, N, K, ldx, ldw, ldo, stream);
        return launch<float, float, float>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    }
    if (x_dtype == LLM_BF16 && w_dtype == LLM_BF16 && out_dtype == LLM_BF16)
        return launch<bf, bf, bf>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    if (x_dtype == LLM_BF16 && w_dtype == LLM_BF16 && out_dtype == LLM_F32)
        return launch<bf, bf, float>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    if (x_dtype == LLM_F32 && w_dtype == LLM_BF16 && out_dtype == LLM_F32)  // an input that stays 32-bit against stored weights
        return launch<float, bf, float>(x, w, out, M, N, K, ldx, ldw, ldo, stream);
    return LLM_ERR_BAD_ARGUMENT;
}

// `batches` products of one shape: product b reads x + b * x_batch and w + b * w_batch (in elements) and writes
// out + b * o_batch.  Heads that lie side by side in a row are batches with a stride of one head.
LLM_EXPORT int llm_gemm_simt_batched(const void* x, const void* w, void* out, int dtype, int out_dtype, int M, int N, int K,
                                     int ldx, int ldw, int ldo, int batches, long long x_batch, long long w_batch,
                                     long long o_batch, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batches <= 0) return 0;
    if (K < 0 || ldx < K || ldw < K || ldo < N) return LLM_ERR_BAD_ARGUMENT;
    if ((M + BM - 1) / BM > 65535 || batches > 65535) return LLM_ERR_UNSUPPORTED;
    using bf = __nv_bfloat16;
    if (dtype == LLM_F32 && out_dtype == LLM_F32)
        return launch<float, float, float>(x, w, out, M, N, K, ldx, ldw, ldo, stream, batches, x_batch, w_batch, o_batch);
    if (dtype == LLM_BF16 && out_dtype == LLM_BF16)
        return launch<bf, bf, bf>(x, w, out, M, N, K, ldx, ldw, ldo, stream, batches, x_batch, w_batch, o_batch);
    if (dtype == LLM_BF16 && out_dtype == LLM_F32)
        return launch<bf, bf, float>(x, w, out, M, N, K, ldx, ldw, ldo, stream, batches, x_batch, w_batch, o_batch);
    return LLM_ERR_BAD_ARGUMENT;
}
