// Sigmoid attention with mixed heads (see sigmoid_attention.cu for the mechanism) for steps in which every request brings one token
// (bfloat16, keys and values of 64 lanes, up to 8 key/value heads of up to 8 query heads, up to 64 heads).
//
// What bounds it: latency.  Four requests of 600 keys are 5 MB of keys and values a layer.  The tensor-core kernel's tile of 16 tokens is one token
// and fifteen rows of nothing here, its keys pass shared memory between five meetings a tile, and its shares leave partial sums to a kernel of
// their own.
//
// A cluster of up to 8 CTAs has a request.  A CTA is two sets of eight warps, a chunk of 32 keys each at a time: chunk s of the keys (counted from
// the first that the token sees) is set s % (2 CTAs)'s.  A warp has a key/value head: a lane scores one key with its row in registers, the next
// chunk's rows on their way meanwhile; the set's weights meet in shared memory, are mixed there in 32 bits, a lane a key again, and meet the values
// with a lane for two of their lanes.  The sums of all sets meet once, through distributed shared memory.  All of it is 32-bit.
#include "common.cuh"

namespace {

using bf16 = __nv_bfloat16;
constexpr int THREADS = 512, SETS = 2, SET_WARPS = 8, CHUNK = 32, LANES = 64, MAX_H = 64, MAX_GROUP = 8;

struct StepParams {
    const bf16* q;
    int ldq;
    const bf16* pool;
    const int *page_table, *positions, *token_request;
    int table_width;
    const float *bias, *mix;
    bf16* out;
    int H, KV, Dp, page_size, window;
    float scale, cap;
};

__device__ __forceinline__ float exp2_fast(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ void meet_set(int set) { asm volatile("barrier.cta.sync %0, %1;\n" ::"r"(1 + set), "n"(SET_WARPS * 32) : "memory"); }
__device__ __forceinline__ void meet_cluster() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// the value at the same place in the shared memory of the cluster's CTA `rank`
__device__ __forceinline__ float value_of(const float* here, unsigned rank) {
    unsigned there;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(there) : "r"((unsigned)__cvta_generic_to_shared(here)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(there) : "memory");
    return v;
}

template <int GROUP>  // query heads a key/value head, at most
__global__ void __launch_bounds__(THREADS)
sigmoid_attention_step_kernel(const StepParams p, const int shares) {
    extern __shared__ __align__(16) float smem[];
    const int H = p.H, KV = p.KV, group = H / KV, WP = H + 4;
    float* sq = smem;                            // [H][64] the token's queries
    float* st = sq + H * LANES;                  // [H][H]: st[g][h] = mix[h][g]
    float* sp = st + H * H;                      // [SETS][H][32] weights of a chunk
    float* sw = sp + SETS * H * CHUNK;           // [SETS][32][WP] mixed
    float* so = sw + SETS * CHUNK * WP;          // [SETS][H][64] sums
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, set = warp / SET_WARPS, c = warp % SET_WARPS;
    const int t = blockIdx.x / shares, rank = blockIdx.x - t * shares;
    pdl_trigger();
    const int pos = p.positions[t];
    const int* table = p.page_table + (size_t)p.token_request[t] * p.table_width;
    const int first = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    for (int i = tid; i < H * H; i += THREADS) {
        const int g = i / H, h = i - g * H;
        st[i] = p.mix ? p.mix[(size_t)h * H + g] : (g == h ? 1.f : 0.f);
    }
    const int chunks = (pos - first) / CHUNK + 1, mine = rank * SETS + set, stride = shares * SETS;
    const float LOG2E = 1.4426950408889634f, inv_cap = p.cap > 0.f ? 1.f / p.cap : 0.f;
    const float c1 = p.scale * 2.f * inv_cap * LOG2E, c2 = -p.scale * LOG2E, ncap = -p.cap * LOG2E;
    float nb[GROUP];
#pragma unroll
    for (int e = 0; e < GROUP; ++e) nb[e] = e < group && c < KV && p.bias ? -p.bias[c * group + e] * LOG2E : 0.f;
    // the row (of key/value head 0's keys) of this lane's key in chunk s
    auto row_of = [&](int s) {
        const int j = min(first + s * CHUNK + lane, pos);
        return table[j / p.page_size] * 2 * KV * p.page_size + j % p.page_size;
    };
    int row = mine < chunks ? row_of(mine) : 0;
    pdl_wait();
    for (int i = tid; i < H * (LANES / 4); i += THREADS) {
        float v[4];
        load4(p.q + (size_t)t * p.ldq + i * 4, v);
        store4(sq + i * 4, v);
    }
    uint4 key[8];
    auto fetch_keys = [&]() {
        if (c >= KV) return;
        const uint4* src = reinterpret_cast<const uint4*>(p.pool + (size_t)(row + c * p.page_size) * p.Dp);
#pragma unroll
        for (int i = 0; i < 8; ++i) key[i] = src[i];
    };
    if (mine < chunks) fetch_keys();
    __syncthreads();
    float acc[GROUP][2];
#pragma unroll
    for (int e = 0; e < GROUP; ++e) acc[e][0] = acc[e][1] = 0.f;
    float *my_p = sp + set * H * CHUNK, *my_w = sw + set * CHUNK * WP;
    for (int s = mine; s < chunks; s += stride) {
        const int live = min(CHUNK, pos - first - s * CHUNK + 1);  // keys of this chunk
        const int rows = row;                                       // this lane's key's row, for the values
        __nv_bfloat162 val[CHUNK];
        if (c < KV) {
            // the chunk's values, two lanes a thread, on their way while the keys are scored; a key that is not there reads nothing
#pragma unroll
            for (int j = 0; j < CHUNK; ++j) {
                const int r = __shfl_sync(0xffffffffu, rows, j);
                val[j] = __floats2bfloat162_rn(0.f, 0.f);
                if (j < live) val[j] = reinterpret_cast<const __nv_bfloat162*>(p.pool + (size_t)(r + (KV + c) * p.page_size) * p.Dp)[lane];
            }
            float dot[GROUP];
#pragma unroll
            for (int e = 0; e < GROUP; ++e) dot[e] = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const __nv_bfloat162* k2 = reinterpret_cast<const __nv_bfloat162*>(&key[i]);
                float kf[8];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    kf[2 * x] = __low2float(k2[x]);
                    kf[2 * x + 1] = __high2float(k2[x]);
                }
#pragma unroll
                for (int e = 0; e < GROUP; ++e) {
                    if (e >= group) break;
                    float qa[4], qb[4];
                    load4(sq + (c * group + e) * LANES + i * 8, qa);
                    load4(sq + (c * group + e) * LANES + i * 8 + 4, qb);
#pragma unroll
                    for (int x = 0; x < 4; ++x) dot[e] = fmaf(kf[x], qa[x], dot[e]);
#pragma unroll
                    for (int x = 0; x < 4; ++x) dot[e] = fmaf(kf[4 + x], qb[x], dot[e]);
                }
            }
#pragma unroll
            for (int e = 0; e < GROUP; ++e) {
                if (e >= group) break;
                // cap * tanh(x / cap) = cap * (1 - 2 / (1 + 2^(x c1))), the sigmoid 1 / (1 + 2^(-y log2 e)), as in the tensor-core kernel
                float y = fmaf(dot[e], c2, nb[e]);
                if (p.cap > 0.f) y = fmaf(ncap, 1.f - __fdividef(2.f, 1.f + exp2_fast(fminf(dot[e] * c1, 100.f))), nb[e]);
                const float w = __fdividef(1.f, 1.f + exp2_fast(fminf(y, 100.f)));
                my_p[(c * group + e) * CHUNK + lane] = lane < live ? w : 0.f;
            }
        }
        if (s + stride < chunks) {
            row = row_of(s + stride);
            fetch_keys();
        }
        meet_set(set);
        for (int h0 = c * 4; h0 < H; h0 += SET_WARPS * 4) {
            float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
            for (int g = 0; g < H; ++g) {
                const float pv = my_p[g * CHUNK + lane];
                float w[4];
                load4(st + g * H + h0, w);
#pragma unroll
                for (int e = 0; e < 4; ++e) m[e] = fmaf(w[e], pv, m[e]);
            }
            store4(my_w + lane * WP + h0, m);
        }
        meet_set(set);  // (the weights of the next chunk are written by warps that have left the mixing: behind this meeting)
        if (c < KV) {
#pragma unroll
            for (int j = 0; j < CHUNK; ++j) {
                const float a = __low2float(val[j]), b = __high2float(val[j]);
                const float* w = my_w + j * WP + c * group;
#pragma unroll
                for (int e = 0; e < GROUP; ++e) {
                    if (e >= group) break;
                    acc[e][0] = fmaf(w[e], a, acc[e][0]);
                    acc[e][1] = fmaf(w[e], b, acc[e][1]);
                }
            }
        }
        // the mixed weights are written again behind the next chunk's first meeting, by when everybody has read these
    }
    if (c < KV)
#pragma unroll
        for (int e = 0; e < GROUP; ++e)
            if (e < group) *reinterpret_cast<float2*>(so + ((size_t)set * H + c * group + e) * LANES + lane * 2) = make_float2(acc[e][0], acc[e][1]);
    if (shares > 1) meet_cluster();
    else __syncthreads();
    const int total = H * LANES;
    for (int i = rank * THREADS + tid; i < total; i += shares * THREADS) {
        float sum = 0.f;
        for (int r = 0; r < shares; ++r)
#pragma unroll
            for (int b = 0; b < SETS; ++b) sum += shares > 1 ? value_of(so + (size_t)b * total + i, r) : so[(size_t)b * total + i];
        p.out[(size_t)t * total + i] = __float2bfloat16_rn(sum);
    }
    if (shares > 1) meet_cluster();  // nobody leaves while its sums are being read
}

template <int GROUP>
int launch(const StepParams& p, int tokens, int shares, size_t smem, cudaStream_t stream) {
    auto kernel = sigmoid_attention_step_kernel<GROUP>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tokens * shares);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = shares;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = shares > 1 ? 2 : 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, p, shares);
}

}  // namespace

// One token a request: arguments as llm_sigmoid_attention, `shares` (1, 2, 4 or 8) CTAs a token.  Keys and values of 64 lanes, H at most 64 in
// multiples of 4, at most 8 key/value heads and 8 query heads to one, rows on 16 bytes; LLM_ERR_UNSUPPORTED otherwise.
LLM_EXPORT int llm_sigmoid_attention_step(const void* q, int ldq, const void* pool, long long pool_pages, const int* page_table, int table_width,
                                          const int* positions, const int* token_request, const float* bias, const float* mix, void* out, int N, int H,
                                          int KV, int D, int V, int Dp, int page_size, float scale, float cap, int window, int shares,
                                          cudaStream_t stream) {
    if (N <= 0) return 0;
    if (H <= 0 || KV <= 0 || H % KV || Dp < D || Dp < V || page_size < 1 || (shares != 1 && shares != 2 && shares != 4 && shares != 8)) return LLM_ERR_BAD_ARGUMENT;
    if (D != LANES || V != LANES || H > MAX_H || (H & 3) || KV > SET_WARPS || H / KV > MAX_GROUP || (Dp & 7) || (ldq & 3) || ((uintptr_t)q & 7) ||
        ((uintptr_t)pool & 15) || pool_pages * 2 * KV * page_size > 0x7fffffffLL)
        return LLM_ERR_UNSUPPORTED;
    const StepParams p = {(const bf16*)q, ldq, (const bf16*)pool, page_table, positions, token_request, table_width, bias, mix, (bf16*)out, H, KV, Dp,
                          page_size, window, scale, cap};
    const size_t smem = (size_t)(H * LANES + H * H + SETS * (H * CHUNK + CHUNK * (H + 4) + H * LANES)) * sizeof(float);
    return H / KV <= 4 ? launch<4>(p, N, shares, smem, stream) : launch<8>(p, N, shares, smem, stream);
}
