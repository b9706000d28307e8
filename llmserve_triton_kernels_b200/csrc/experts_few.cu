// A mixture of small feed-forward layers for steps of few tokens (bfloat16, at most 8): only the experts that a token of the step
// uses are read.
//
// In a decode step (1,408 + 704 x 4 of 32 experts, 2,048 wide) they take 11.0 + 8.3 us a layer for one token and 17.1 + 12.5 for three,
// where the products over all experts and the activation between them took 30.4 + 2.6 + 15.7.
//
// What bounds it: the bytes of the weights.  One token that uses 4 of 32 experts needs 52 of the 294 MB that the products over all
// experts read; eight tokens need about two thirds.  Two kernels, the activation in the first one's end:
//   up    act[t, j] = act(x W_up^T) * weight[t, expert of j]           (gated: gate and up rows of the same feature in one tile)
//   down  y[t, n] = sum over the used experts' j of act[t, j] W_down[n, j], plain or added to the residual stream
// Which experts are used is known on the device alone (the router's weights, or the table's row of each token id): every CTA makes the
// list and walks the tiles of the listed blocks.  The products are mma.sync m16n8k16, the weights its sixteen rows and the tokens its
// eight columns; a thread's 16 bytes of a row hold its operands of two k-steps if the tokens' lanes are permuted alike.
//   up    a CTA an SM, a tile of 16 rows at a time, whole rows by bulk copies into a ring of three tiles (192 KB in flight), asked for by a
//         warp of its own; each of sixteen warps takes every sixteenth piece of 32 k, its part of x in registers.
//   down  a CTA 16 features, each of its sixteen warps pieces of 32 k of the listed blocks, straight into registers, two rounds of weights
//         and activations on their way.  Which warp has a piece depends on the piece's place in w_down alone: a token's bits are the
//         same whatever experts the other tokens use.
// Behind its own tiles the up kernel has the down kernel's weights brought into L2, so that memory does not stand still between the two.
// The shared expert's tiles (and, with a table, everybody's) are on their way before the kernel in front has ended.  The up kernel
// lets its dependent start only behind its own wait, by when the router has ended: the down kernel makes its list without waiting.  Its CTAs
// (128 registers x 512 threads, an SM's whole register file) start where an up CTA has ended, and ask for their first weights while
// others still run.
#include "common.cuh"
#include "tma.cuh"

namespace {

using bf16 = __nv_bfloat16;
constexpr int MAX_M = 8, MAX_E = 256, WARPS = 16, UP_THREADS = WARPS * 32 + 32, UP_KB = 4, DOWN_THREADS = WARPS * 32, DOWN_AHEAD = 4, MAX_SLOTS = 8;
constexpr size_t AHEAD_BYTES = 32 << 20;  // the most of w_down that the up kernel brings into L2
constexpr int UP_RING = 196 * 1024;  // three tiles of 2,048 k

struct Experts {
    const bf16 *x, *w_up, *w_down;
    bf16* act;  // [M, E * ff + fs]: only used blocks are written and read
    int ldx, M, K, N, E, ff, fs, kind;  // kind: -1 gated, else the activation
    float limit, limit_s, slope, up_shift;
    const float* weights;  // [M, ldw], or null:
    int ldw;
    const int *ids, *table;
    int top, vocab;
    float *out, *resid;  // out [M, N], or resid [M, N] += alpha * y
    const float* norm_w;  // with resid: xw_out = resid * norm_w, ss_out [N / 16, M] = sums of resid^2
    bf16* xw_out;
    float* ss_out;
    float alpha;
    int up_slots;
    int* error_flag;
};

__device__ __forceinline__ void mma_bf16(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// both k-steps of a piece of 32 k: a0, a1: rows g and g + 8 of the weights, b: column g of the tokens
__device__ __forceinline__ void mma_piece(float (&c)[4], float (&d)[4], const uint4& a0, const uint4& a1, const uint4& b) {
    mma_bf16(c, a0.x, a1.x, a0.y, a1.y, b.x, b.y);
    mma_bf16(d, a0.z, a1.z, a0.w, a1.w, b.z, b.w);
}
// weights are read once: no place in L1
__device__ __forceinline__ uint4 load_weight(const bf16* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// `bytes` (a multiple of 16) into shared memory, counted on `bar`
__device__ __forceinline__ void copy_bulk(void* to, const void* from, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(tma::smem_addr(to)), "l"(from), "r"(bytes), "r"(tma::smem_addr(bar)) : "memory");
}

__device__ __forceinline__ float weight_of(const Experts& p, int m, int e) {
    if (p.weights) return __ldcg(p.weights + (size_t)m * p.ldw + e);
    if (e == p.E) return 1.f;
    int id = p.ids[m];
    if (id < 0 || id >= p.vocab) id = 0;
    float w = 0.f;
    for (int c = 0; c < p.top; ++c) w = p.table[(size_t)id * p.top + c] == e ? 1.f / (float)p.top : w;
    return w;
}

// The used experts in ascending order, and (wt_s not null) every token's weight of every expert and of the shared one, by warp 0; the
// caller meets before it reads them.
__device__ __forceinline__ void list_experts(const Experts& p, short* list, int* count, float (*wt_s)[MAX_E + 1]) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    int n = 0;
    if (wt_s && lane < p.M && p.fs > 0) wt_s[lane][p.E] = weight_of(p, lane, p.E);
    for (int e0 = 0; e0 < p.E; e0 += 32) {
        const int e = e0 + lane;
        float wt[MAX_M];
        bool used = false;
#pragma unroll
        for (int m = 0; m < MAX_M; ++m) wt[m] = m < p.M && e < p.E ? weight_of(p, m, e) : 0.f;
#pragma unroll
        for (int m = 0; m < MAX_M; ++m) {
            used |= wt[m] != 0.f;
            if (wt_s && e < p.E) wt_s[m][e] = wt[m];
        }
        const unsigned mask = __ballot_sync(0xffffffffu, used);
        if (used) list[n + __popc(mask & ((1u << lane) - 1))] = (short)e;
        n += __popc(mask);
    }
    if (lane == 0) *count = n;
}

__device__ __forceinline__ float activate(float v, int kind) {
    if (kind == 0) { const float r = fmaxf(v, 0.f); return r * r; }                                    // relu^2
    if (kind == 1) return 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));  // gelu (tanh)
    if (kind == 3) return v / (1.f + expf(-v));                                                        // silu
    return v;
}

// The sixteen warps' sums of a lane's four values, in order.
__device__ __forceinline__ void add_up(const float (*red)[32][4], int lane, float (&s)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
        float part[4];
        load4(red[w][lane], part);
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] += part[i];
    }
}

__global__ void __launch_bounds__(UP_THREADS, 1) experts_up_kernel(const Experts p) {
    extern __shared__ __align__(128) unsigned char ring[];  // [slots][16][2 K + 64]
    __shared__ short list[MAX_E];
    __shared__ int count, gave_up;
    __shared__ __align__(16) float red[2][WARPS][32][4];
    __shared__ float wt_s[MAX_M][MAX_E + 1];
    __shared__ __align__(8) unsigned long long full[MAX_SLOTS], empty[MAX_SLOTS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const bool gated = p.kind < 0, known = p.weights == nullptr;  // the table's experts do not depend on the kernel in front
    const int step = gated ? 8 : 16, tiles_e = p.ff / step, tiles_s = p.fs / step, per = gated ? 2 : 1;
    const int pitch = p.K * 2 + 64, slot_bytes = 16 * pitch;
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.up_slots; ++s) {
            tma::mbar_init(&full[s], 1);
            tma::mbar_init(&empty[s], WARPS);
        }
        tma::mbar_fence_init();
        gave_up = 0;
    }
    if (known) list_experts(p, list, &count, wt_s);
    __syncthreads();
    // tile v: the shared expert's first, then the listed experts'
    auto place = [&](int v, int& e, int& f0) {
        e = v < tiles_s ? p.E : list[(v - tiles_s) / tiles_e];
        f0 = (v < tiles_s ? v : (v - tiles_s) % tiles_e) * step;
    };
    auto fail = [&]() {
        gave_up = 1;
        if (p.error_flag) atomicExch(p.error_flag, 1);
    };
    // the asking warp asks for the CTA's n-th tile, sixteen lanes a row each
    auto ask = [&](int n) {
        int e, f0;
        place(blockIdx.x + n * gridDim.x, e, f0);
        const int s = n % p.up_slots;
        if (lane == 0) tma::mbar_expect_tx(&full[s], 16 * p.K * 2);
        __syncwarp();
        if (lane < 16) {
            const size_t row = (size_t)e * per * p.ff + f0 + (gated && lane >= 8 ? (e == p.E ? p.fs : p.ff) + lane - 8 : lane);
            copy_bulk(ring + (size_t)s * slot_bytes + lane * pitch, p.w_up + row * p.K, p.K * 2, &full[s]);
        }
    };
    int asked = 0, total = known ? tiles_s + count * tiles_e : tiles_s;
    auto mine = [&]() { return (int)blockIdx.x < total ? (total - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0; };
    if (warp == WARPS)
        for (const int n = min(mine(), p.up_slots); asked < n; ++asked) ask(asked);
    pdl_wait();
    pdl_trigger();  // behind the wait: see above
    uint4 xb[UP_KB];
    if (warp < WARPS) {
#pragma unroll
        for (int i = 0; i < UP_KB; ++i) {
            const int k = (warp + i * WARPS) * 32;
            xb[i] = k < p.K && g < p.M ? *reinterpret_cast<const uint4*>(p.x + (size_t)g * p.ldx + k + q * 8) : make_uint4(0, 0, 0, 0);
        }
    }
    if (!known) {
        list_experts(p, list, &count, wt_s);
        __syncthreads();
        total = tiles_s + count * tiles_e;
    }
    const int tiles = mine(), lda = p.E * p.ff + p.fs;
    if (warp == WARPS) {
        for (; asked < tiles; ++asked) {
            if (asked >= p.up_slots && !__all_sync(0xffffffffu, tma::mbar_wait(&empty[asked % p.up_slots], (asked / p.up_slots - 1) & 1))) {
                fail();
                break;
            }
            ask(asked);
        }
        // the down kernel's weights on their way into L2 behind this kernel's: memory does not stand still while this one ends and that one
        // starts (row by row of a block, dealt over the CTAs)
        const int blocks = (p.fs > 0 ? 1 : 0) + count, ldk = p.E * p.ff + p.fs;
        const int items = (int)min((long long)blocks * p.N, (long long)(AHEAD_BYTES / (2 * (size_t)max(p.ff, p.fs))));
        for (int i = blockIdx.x * 32 + lane; i < items; i += gridDim.x * 32) {
            const int b = i / p.N, n = i - b * p.N;
            const bool shared = p.fs > 0 && b == 0;
            const bf16* at = p.w_down + (size_t)n * ldk + (size_t)(shared ? p.E : list[b - (p.fs > 0 ? 1 : 0)]) * p.ff;
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(at), "r"((shared ? p.fs : p.ff) * 2) : "memory");
        }
        // the other warps wait for every tile that was asked for, but not once a wait has given up: no copy is left on its way to a CTA that
        // has ended
        for (int n = max(0, asked - p.up_slots); n < asked; ++n) tma::mbar_wait(&full[n % p.up_slots], (n / p.up_slots) & 1);
        return;
    }
    for (int n = 0; n < tiles; ++n) {
        const int s = n % p.up_slots;
        if (!*(volatile int*)&gave_up && !tma::mbar_wait(&full[s], (n / p.up_slots) & 1)) fail();
        const unsigned char* row = ring + (size_t)s * slot_bytes + g * pitch + q * 16;
        float c[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < UP_KB; ++i) {
            const int k = (warp + i * WARPS) * 32;
            if (k < p.K) mma_piece(c, d, *reinterpret_cast<const uint4*>(row + k * 2), *reinterpret_cast<const uint4*>(row + 8 * pitch + k * 2), xb[i]);
        }
        __syncwarp();
        if (lane == 0) tma::mbar_arrive(&empty[s]);
        *reinterpret_cast<float4*>(red[n & 1][warp][lane]) = make_float4(c[0] + d[0], c[1] + d[1], c[2] + d[2], c[3] + d[3]);
        // the sixteen warps meet; the other buffer of sums is written next, and this one read until the meeting after that
        asm volatile("bar.sync 1, %0;\n" ::"n"(WARPS * 32) : "memory");
        if (warp != n % WARPS) continue;
        int e, f0;
        place(blockIdx.x + n * gridDim.x, e, f0);
        float sum[4];
        add_up(red[n & 1], lane, sum);
#pragma unroll
        for (int i = 0; i < 2; ++i) {  // token 2 q + i; sum[i]: row g, sum[i + 2]: row g + 8
            const int m = 2 * q + i;
            if (m >= p.M) continue;
            const float wt = wt_s[m][e];
            bf16* y = p.act + (size_t)m * lda + (size_t)e * p.ff + f0 + g;
            if (gated) {
                const float lim = e == p.E ? p.limit_s : p.limit, gc = fminf(sum[i], lim), uc = fminf(fmaxf(sum[i + 2], -lim), lim);
                y[0] = __float2bfloat16_rn(wt == 0.f ? 0.f : gc / (1.f + expf(-p.slope * gc)) * (uc + p.up_shift) * wt);
            } else {
                y[0] = __float2bfloat16_rn(wt == 0.f ? 0.f : activate(sum[i], p.kind) * wt);
                y[8] = __float2bfloat16_rn(wt == 0.f ? 0.f : activate(sum[i + 2], p.kind) * wt);
            }
        }
    }
}

__global__ void __launch_bounds__(DOWN_THREADS, 1) experts_down_kernel(const Experts p) {
    __shared__ short list[MAX_E];
    __shared__ int count;
    __shared__ __align__(16) float red[WARPS][32][4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int n0 = blockIdx.x * 16, ldk = p.E * p.ff + p.fs, pieces_e = p.ff >> 5, pieces_s = p.fs >> 5;
    pdl_trigger();
    list_experts(p, list, &count, nullptr);  // the router ended before the up kernel let this one start
    __syncthreads();
    // The warp's pieces: the neighbouring pairs (whole lines of 128 bytes) whose number among all of w_down's columns is the warp's own modulo
    // WARPS, of the shared expert, then of the listed ones.  So the order of a token's sums does not depend on the experts of others,
    // whose pieces in between add zeros.
    int block = pieces_s > 0 ? -1 : 0, at = -1, end = -1;  // `at`: the next piece, one of the block that ends at `end`
    auto enter = [&]() {  // the block's first piece of this warp, or a later block's; at = -1: none is left
        for (; block < count; ++block) {
            const int a0 = (block < 0 ? p.E : list[block]) * pieces_e, pair = a0 >> 1, skip = (warp - pair) & (WARPS - 1);
            at = skip == 0 ? a0 : (pair + skip) * 2;
            end = a0 + (block < 0 ? pieces_s : pieces_e);
            if (at < end) return;
        }
        at = -1;
    };
    enter();
    auto take = [&]() {
        if (at < 0) return -1;
        const int k = at * 32;
        at += (at & 1) ? 2 * WARPS - 1 : 1;
        if (at >= end) {
            ++block;
            enter();
        }
        return k;
    };
    const bf16 *row0 = p.w_down + (size_t)(n0 + g) * ldk + q * 8, *row1 = row0 + (size_t)8 * ldk, *tokens = p.act + (size_t)g * ldk + q * 8;
    struct Round { uint4 a[DOWN_AHEAD][2], b[DOWN_AHEAD]; int k[DOWN_AHEAD]; };  // first k of each piece, or -1
    auto ask = [&](Round& r) {
#pragma unroll
        for (int u = 0; u < DOWN_AHEAD; ++u) {
            r.k[u] = take();
            r.a[u][0] = r.k[u] >= 0 ? load_weight(row0 + r.k[u]) : make_uint4(0, 0, 0, 0);
            r.a[u][1] = r.k[u] >= 0 ? load_weight(row1 + r.k[u]) : make_uint4(0, 0, 0, 0);
        }
    };
    auto ask_tokens = [&](Round& r) {
#pragma unroll
        for (int u = 0; u < DOWN_AHEAD; ++u)
            r.b[u] = r.k[u] >= 0 && g < p.M ? __ldcg(reinterpret_cast<const uint4*>(tokens + r.k[u])) : make_uint4(0, 0, 0, 0);
    };
    float c4[4] = {0.f, 0.f, 0.f, 0.f}, d4[4] = {0.f, 0.f, 0.f, 0.f};
    auto multiply = [&](const Round& r) {
#pragma unroll
        for (int u = 0; u < DOWN_AHEAD; ++u) mma_piece(c4, d4, r.a[u][0], r.a[u][1], r.b[u]);
    };
    Round r0, r1;
    ask(r0);
    ask(r1);
    pdl_wait();
    ask_tokens(r0);
    ask_tokens(r1);
    while (r0.k[0] >= 0) {  // (pieces behind the last are zeros)
        multiply(r0);
        ask(r0);
        ask_tokens(r0);
        multiply(r1);
        ask(r1);
        ask_tokens(r1);
    }
    *reinterpret_cast<float4*>(red[warp][lane]) = make_float4(c4[0] + d4[0], c4[1] + d4[1], c4[2] + d4[2], c4[3] + d4[3]);
    __syncthreads();
    if (warp != 0) return;
    float s[4], ss[2] = {0.f, 0.f};
    add_up(red, lane, s);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = 2 * q + (i & 1), n = n0 + g + (i >> 1) * 8;
        if (m >= p.M) continue;
        const size_t at = (size_t)m * p.N + n;
        if (!p.resid) {
            p.out[at] = s[i];
            continue;
        }
        const float r = fmaf(p.alpha, s[i], p.resid[at]);
        p.resid[at] = r;
        if (p.norm_w) {
            p.xw_out[at] = __float2bfloat16_rn(r * p.norm_w[n]);
            ss[i & 1] = fmaf(r, r, ss[i & 1]);
        }
    }
    if (p.norm_w) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], o);
            if (g == 0 && 2 * q + i < p.M) p.ss_out[(size_t)blockIdx.x * p.M + 2 * q + i] = ss[i];
        }
    }
}

}  // namespace

// x [M, K] (row stride ldx) through a mixture of E experts of inner size ff and a shared one of fs (0: none).
//   kind -1: w_up holds, expert by expert, the gate's ff rows and the up's ff rows, then the shared expert's fs and fs; the activation is
//            g * sigmoid(slope * g) * (u + up_shift), g = min(gate, limit), u = clamp(up, -limit, limit) (limit_s for the shared one)
//   kind 0, 1, 3: w_up holds ff rows an expert, then fs; the activation is relu^2, gelu (tanh), silu
//   weights [M, E (+ 1)] (row stride ldw), or null: 1 / top for the entries of table[ids[m]], 1 for the shared expert
//   w_down [N, E * ff + fs];  act: scratch [M, E * ff + fs], of which only the used experts' columns are written
//   out [M, N] float32, or resid [M, N] += alpha * result and, with norm_w, xw_out [M, N] and ss_out [N / 16, M] (see llm_linear_decode)
// Needs M <= 8, K <= 2048, K, ff and fs multiples of 32, N of 16, E <= 256, 16-byte aligned rows; otherwise LLM_ERR_UNSUPPORTED.
LLM_EXPORT int llm_experts_few(const void* x, int ldx, const void* w_up, const void* w_down, void* act, int M, int K, int N, int E, int ff,
                               int fs, int kind, float limit, float limit_s, float slope, float up_shift, const float* weights, int ldw,
                               const int* ids, const int* table, int top, int vocab, float* out, float* resid, const float* norm_w,
                               void* xw_out, float* ss_out, float alpha, int* error_flag, cudaStream_t stream) {
    if (M <= 0) return 0;
    if ((!weights && (!ids || !table || top < 1 || vocab < 1)) || (!out && !resid) || (norm_w && (!resid || !xw_out || !ss_out)) || kind < -1 ||
        kind == 2 || kind > 3 || fs < 0)
        return LLM_ERR_BAD_ARGUMENT;
    auto aligned = [](const void* a) { return ((uintptr_t)a & 15) == 0; };
    if (M > MAX_M || K < 32 || K > WARPS * UP_KB * 32 || (K & 31) || ff < 32 || (ff & 31) || (fs & 31) || N < 16 || (N & 15) || E < 1 || E > MAX_E ||
        (ldx & 7) || !aligned(x) || !aligned(w_up) || !aligned(w_down) || !aligned(act))
        return LLM_ERR_UNSUPPORTED;
    Experts p = {};
    p.x = (const bf16*)x; p.w_up = (const bf16*)w_up; p.w_down = (const bf16*)w_down; p.act = (bf16*)act;
    p.ldx = ldx; p.M = M; p.K = K; p.N = N; p.E = E; p.ff = ff; p.fs = fs; p.kind = kind;
    p.limit = limit; p.limit_s = limit_s; p.slope = slope; p.up_shift = up_shift;
    p.weights = weights; p.ldw = ldw; p.ids = ids; p.table = table; p.top = top; p.vocab = vocab;
    p.out = out; p.resid = resid; p.norm_w = norm_w; p.xw_out = (bf16*)xw_out; p.ss_out = ss_out; p.alpha = alpha; p.error_flag = error_flag;
    const int up_slot = 16 * (K * 2 + 64);
    p.up_slots = UP_RING / up_slot < MAX_SLOTS ? UP_RING / up_slot : MAX_SLOTS;
    const int sms = device_sms();
    const cudaError_t set = cudaFuncSetAttribute(experts_up_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, UP_RING);
    if (set != cudaSuccess) return (int)set;
    const int most = (E * ff + fs) / (kind < 0 ? 8 : 16);
    const int code = launch_pdl(experts_up_kernel, dim3(most < sms ? most : sms), dim3(UP_THREADS), (size_t)p.up_slots * up_slot, stream, p);
    return code != 0 ? code : launch_pdl(experts_down_kernel, dim3(N / 16), dim3(DOWN_THREADS), 0, stream, p);
}
