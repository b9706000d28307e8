// What a token's projections go through between the stacked product and attention, together with the write of what
// the cache keeps: for latent attention the rotation of the query's rotated parts, the RMS norm of the latent and the
// rotation of the shared key part; for attention with unit-RMS queries and keys the two norms.
//
// Angles are 32-bit (float(position) * frequency, then sincosf), statistics are 32-bit, results are rounded once.
#include "common.cuh"

namespace {

// The rotated lanes of `heads` heads, `src_head` and `dst_head` elements apart: pair i of a head turns by turn[i] (worked out once per
// token), lanes (2i, 2i + 1), or with `halves` (i, i + rot_dims / 2); the lanes behind the first `rot_dims` pass unchanged.  The pairs
// of all heads are dealt over the threads, so that a token's loads are in flight together.
template <typename T>
__device__ __forceinline__ void rotate_heads(const T* __restrict__ src, int src_head, T* __restrict__ dst, int dst_head, int heads, int lanes,
                                             int rot_dims, int halves, const float2* __restrict__ turn, int first, int step) {
    const int pairs = rot_dims >> 1, rest = lanes - rot_dims;
#pragma unroll 4
    for (int at = first; at < heads * pairs; at += step) {
        const int h = at / pairs, i = at - h * pairs;
        const int a = halves ? i : 2 * i, b = halves ? i + pairs : 2 * i + 1;
        const float c = turn[i].x, s = turn[i].y;
        const float u = to_float(src[(size_t)h * src_head + a]), v = to_float(src[(size_t)h * src_head + b]);
        dst[(size_t)h * dst_head + a] = from_float<T>(u * c - v * s);
        dst[(size_t)h * dst_head + b] = from_float<T>(v * c + u * s);
    }
    for (int at = first; at < heads * rest; at += step) {
        const int h = at / rest, i = rot_dims + at - h * rest;
        dst[(size_t)h * dst_head + i] = src[(size_t)h * src_head + i];
    }
}

constexpr int MAX_TURNS = 320;  // pairs of a rotated part of at most 640 lanes
// For steps of few tokens: the product of every head's plain query lanes with the key up matrix, in the same launch.
constexpr int UP_ROWS = 64, UP_MAX_DIM = 128, UP_MAX_TOKENS = 16;

// One CTA: out[t, h, m0 .. m0 + 63] = sum_d w[h, m, d] * q[t, h, d] for all tokens; two threads a row, each with half of its lanes, which
// are on their way before the kernel in front has ended.  dim a multiple of 16, at most UP_MAX_DIM.
__device__ __forceinline__ void head_up_product(const __nv_bfloat16* __restrict__ queries, int ldq, int head_step, const __nv_bfloat16* __restrict__ w,
                                                __nv_bfloat16* __restrict__ out, int n, int H, int dim, int rank, int block) {
    __shared__ __align__(16) float x_s[UP_MAX_TOKENS * UP_MAX_DIM];
    const int slices = (rank + UP_ROWS - 1) / UP_ROWS, h = block / slices, m = (block - h * slices) * UP_ROWS + (threadIdx.x >> 1);
    const int half = dim >> 1, d0 = (threadIdx.x & 1) * half;
    const __nv_bfloat16* row = w + ((size_t)h * rank + min(m, rank - 1)) * dim + d0;
    uint4 wv[UP_MAX_DIM / 16];
#pragma unroll
    for (int i = 0; i < UP_MAX_DIM / 16; ++i)
        if (i * 8 < half) wv[i] = *reinterpret_cast<const uint4*>(row + i * 8);
    pdl_wait();
    for (int i = threadIdx.x; i < n * dim; i += blockDim.x) {
        const int t = i / dim, d = i - t * dim;
        x_s[i] = to_float(queries[(size_t)t * ldq + (size_t)h * head_step + d]);
    }
    __syncthreads();
    for (int t = 0; t < n; ++t) {
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < UP_MAX_DIM / 16; ++i)
            if (i * 8 < half) {
                const unsigned words[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
                const float* xv = x_s + t * dim + d0 + i * 8;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc = fmaf(__uint_as_float(words[e] << 16), xv[2 * e], acc);
                    acc = fmaf(__uint_as_float(words[e] & 0xffff0000u), xv[2 * e + 1], acc);
                }
            }
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        if (!(threadIdx.x & 1) && m < rank) out[((size_t)t * H + h) * rank + m] = __float2bfloat16_rn(acc);
    }
}

// Latent attention.  proj row: [H x (dim | rot) queries][rank latent | rot shared key part][...]; or the queries in rows
// of their own (`queries`, row pitch ldq) and the latent part at column `kv_col` of proj.  `halves`: the rotated lanes
// pair as (i, i + rot_dims / 2) instead of (2i, 2i + 1).
//   q_rot[t, h, :]   = rotate(proj query h's last rot lanes)
//   cache[slot, :]   = [ latent / sqrt(mean(latent^2) + eps) * weight | rotate(shared key part) ]
//   fresh[t, :]      = the same row (optional)
//   q_up[t, h, :]    = w_up[h] (rank x dim) times query h's first dim lanes (optional, bfloat16, few tokens)
// One block per token, and behind them, for q_up, one per head and UP_ROWS of its rows.
template <typename T>
__global__ void __launch_bounds__(128)
latent_prepare_kernel(const T* __restrict__ proj, int ldp, T* __restrict__ q_rot, T* __restrict__ fresh,
                      const int* __restrict__ positions, const int* __restrict__ slot_map, T* __restrict__ cache,
                      const float* __restrict__ weight,
                      const float* __restrict__ freq, float eps, int H, int dim, int rot, int rank, int rot_dims,
                      const T* __restrict__ queries, int ldq, int kv_col, int halves, int n, const T* __restrict__ w_up, T* __restrict__ q_up) {
    __shared__ float scratch[33];
    __shared__ float2 turn[MAX_TURNS];
    pdl_trigger();
    if constexpr (sizeof(T) == 2) {
        if ((int)blockIdx.x >= n) {
            head_up_product(queries ? queries : proj, queries ? ldq : ldp, dim + rot, w_up, q_up, n, H, dim, rank, (int)blockIdx.x - n);
            return;
        }
    }
    const int t = blockIdx.x;
    const float position = (float)positions[t];
    const size_t slot = (size_t)slot_map[t];
    // the angles depend on the token alone: every head and the shared key part turn by the same ones
    for (int i = threadIdx.x; i < (rot_dims >> 1); i += blockDim.x) {
        float s, c;
        sincosf(position * freq[i], &s, &c);
        turn[i] = make_float2(c, s);
    }
    __syncthreads();
    pdl_wait();
    const T* row = proj + (size_t)t * ldp;
    const T* qrow = queries ? queries + (size_t)t * ldq : row;
    const T* latent = row + (queries ? (size_t)kv_col : (size_t)H * (dim + rot));
    T* kept = cache + slot * (size_t)(rank + rot);
    float ss = 0.f;
    for (int i = threadIdx.x; i < rank; i += blockDim.x) {
        const float v = to_float(latent[i]);
        ss = fmaf(v, v, ss);
    }
    rotate_heads(qrow + dim, dim + rot, q_rot + (size_t)t * H * rot, rot, H, rot, rot_dims, halves, turn, (int)threadIdx.x, (int)blockDim.x);
    ss = block_sum(ss, scratch);
    const float scale = 1.f / sqrtf(ss / (float)rank + eps);
    for (int i = threadIdx.x; i < rank; i += blockDim.x) kept[i] = from_float<T>(to_float(latent[i]) * scale * weight[i]);
    rotate_heads(latent + rank, 0, kept + rank, 0, 1, rot, rot_dims, halves, turn, (int)threadIdx.x, (int)blockDim.x);
    if (fresh) {  // the same row once more, token by token, for whoever wants the step's own rows side by side
        __syncthreads();
        T* copy = fresh + (size_t)t * (rank + rot);
        for (int i = threadIdx.x; i < rank + rot; i += blockDim.x) copy[i] = kept[i];
    }
}

// Attention with unit-RMS queries and keys.  qkv row: [H x dk queries | KV x dk keys | KV x dv values].
//   queries: divided by sqrt(mean(q^2) + eps) per head, in place
//   keys:    the same, written to the key plane of the token's slot;  values: copied to the value plane
// pool plane: [pages, 2, KV, page_size, D] with D >= max(dk, dv).  One warp per head; a block per token, or, for few tokens, several
// that share its heads (a warp that takes ten heads one after the other shows ten loads' latency: 12.7 us of a step of 1.0 ms, now 3.3).
template <typename T>
__global__ void __launch_bounds__(128)
unit_norm_kv_write_kernel(T* __restrict__ qkv, int ld, const int* __restrict__ slot_map, T* __restrict__ pool, float eps,
                          int normed, int H, int KV, int dk, int dv, int D, int page_size) {
    pdl_trigger();
    const int t = blockIdx.x;
    const int slot = slot_map[t];
    const int page = slot / page_size, off = slot - page * page_size;
    pdl_wait();
    T* row = qkv + (size_t)t * ld;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const size_t head_stride = (size_t)page_size * D;
    for (int item = blockIdx.y * warps + warp; item < H + 2 * KV; item += warps * gridDim.y) {
        if (item < H + KV) {
            const T* src = row + (size_t)item * dk;
            T* dst = item < H ? row + (size_t)item * dk
                              : pool + ((size_t)(page * 2 + 0) * KV + (item - H)) * head_stride + (size_t)off * D;
            float scale = 1.f;
            if (normed) {
                float ss = 0.f;
                for (int i = lane; i < dk; i += 32) {
                    const float v = to_float(src[i]);
                    ss = fmaf(v, v, ss);
                }
                ss = warp_sum(ss);
                scale = 1.f / sqrtf(ss / (float)dk + eps);
            }
            for (int i = lane; i < dk; i += 32) dst[i] = from_float<T>(to_float(src[i]) * scale);
        } else {
            const int h = item - H - KV;
            const T* src = row + (size_t)(H + KV) * dk + (size_t)h * dv;
            T* dst = pool + ((size_t)(page * 2 + 1) * KV + h) * head_stride + (size_t)off * D;
            for (int i = lane; i < dv; i += 32) dst[i] = src[i];
        }
    }
}

}  // namespace

LLM_EXPORT int llm_latent_prepare(const void* proj, int dtype, int ldp, void* q_rot, void* fresh, const int* positions,
                                  const int* slot_map, void* cache, const float* weight, const float* freq, float eps, int n,
                                  int H, int dim, int rot, int rank, int rot_dims, const void* queries, int ldq, int kv_col,
                                  int halves, const void* w_up, void* q_up, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (H <= 0 || dim < 0 || rot < 0 || rank <= 0 || rot_dims < 0 || rot_dims > rot || (rot_dims & 1) || rot_dims > 2 * MAX_TURNS ||
        (queries ? (ldq < H * (dim + rot) || kv_col < 0 || ldp < kv_col + rank + rot) : ldp < H * (dim + rot) + rank + rot))
        return LLM_ERR_BAD_ARGUMENT;
    if (w_up && (dtype != LLM_BF16 || !q_up || n > UP_MAX_TOKENS || dim > UP_MAX_DIM || dim < 16 || (dim & 15) || ((uintptr_t)w_up & 15)))
        return LLM_ERR_BAD_ARGUMENT;
    const int up_blocks = w_up ? H * ((rank + UP_ROWS - 1) / UP_ROWS) : 0;
    if (dtype == LLM_F32)
        return launch_pdl(latent_prepare_kernel<float>, dim3(n), dim3(128), 0, stream, (const float*)proj, ldp, (float*)q_rot,
                          (float*)fresh, positions, slot_map, (float*)cache, weight, freq, eps, H, dim, rot, rank, rot_dims,
                          (const float*)queries, ldq, kv_col, halves, n, (const float*)nullptr, (float*)nullptr);
    if (dtype == LLM_BF16)
        return launch_pdl(latent_prepare_kernel<__nv_bfloat16>, dim3(n + up_blocks), dim3(128), 0, stream, (const __nv_bfloat16*)proj, ldp,
                          (__nv_bfloat16*)q_rot, (__nv_bfloat16*)fresh, positions, slot_map, (__nv_bfloat16*)cache, weight, freq, eps, H, dim, rot,
                          rank, rot_dims, (const __nv_bfloat16*)queries, ldq, kv_col, halves, n, (const __nv_bfloat16*)w_up, (__nv_bfloat16*)q_up);
    return LLM_ERR_BAD_ARGUMENT;
}

LLM_EXPORT int llm_unit_norm_kv_write(void* qkv, int dtype, int ld, const int* slot_map, void* pool, float eps, int normed,
                                      int n, int H, int KV, int dk, int dv, int D, int page_size, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (H <= 0 || KV <= 0 || dk <= 0 || dv <= 0 || D < dk || D < dv || page_size <= 0 || ld < (H + KV) * dk + KV * dv)
        return LLM_ERR_BAD_ARGUMENT;
    // an item a warp up to 1,024 tokens (32 + 2 x 8 heads of 64, one CTA a token / several: 200 tokens 12.4 / 4.3 us, 600 12.8 / 8.2, 2,000 22.3 / 25.6)
    const dim3 grid(n, n <= 1024 ? (H + 2 * KV + 3) / 4 : 1);
    if (dtype == LLM_F32)
        return launch_pdl(unit_norm_kv_write_kernel<float>, grid, dim3(128), 0, stream, (float*)qkv, ld, slot_map,
                          (float*)pool, eps, normed, H, KV, dk, dv, D, page_size);
    if (dtype == LLM_BF16)
        return launch_pdl(unit_norm_kv_write_kernel<__nv_bfloat16>, grid, dim3(128), 0, stream, (__nv_bfloat16*)qkv, ld,
                          slot_map, (__nv_bfloat16*)pool, eps, normed, H, KV, dk, dv, D, page_size);
    return LLM_ERR_BAD_ARGUMENT;
}
