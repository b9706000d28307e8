// A mixture of small feed-forward layers for steps of few tokens (bfloat16, at most 8): only the experts that a token of the step
// uses are read.
//
// What bounds it: the bytes of the weights.  One token that uses 4 of 32 experts needs 52 of the 294 MB that the products over all
// experts read; eight tokens need about two thirds.  Two kernels, the activation in the first one's end:
//   up    act[t, j] = act(x W_up^T) * weight[t, expert of j]           (gated: gate and up rows of the same feature in one tile)
//   down  y[t, n] = sum over the used experts' j of act[t, j] W_down[n, j], plain or added to the residual stream
// Which experts are used is known on the device alone (the router's weights, or the table's row of each token id): every warp makes the
// list and walks the listed blocks.  The products are mma.sync m16n8k16, the weights its sixteen rows and the tokens its
// eight columns; a thread's 16 bytes of a row hold its operands of two k-steps if the tokens' lanes are permuted alike.
//
// Both kernels are CTAs of eight warps, every warp with a ring of TMA boxes of its own (as in linear_stream.cuh), so that neither a meeting
// of the CTA nor another warp's pace stands between a box's arrival and the next one's request:
//   up    a CTA an SM, a tile of 16 rows at a time; a warp has one or two boxes of 128 k of every tile and its part of x in registers.
//         The warps' sums wait in shared memory and meet once every four tiles.
//   down  a CTA 16 features; boxes of 64 k, the tokens' lanes of the same k behind the weights in the slot.  Which warp has a box depends on
//         the box's place in w_down alone: a token's bits are the same whatever experts the other tokens use.
// An up CTA and a down CTA share an SM (at most 120 registers x 256 threads and 227 KB together): the up kernel lets its dependent start
// behind its own wait, by when the router has ended, so that the down kernel makes its list and asks for its first boxes (the weights' 48 KB
// a CTA: 6.3 MB at 2,048 wide) while the up kernel runs.  The shared expert's boxes (and, with a table, everybody's) are on their way before
// the kernel in front has ended.
// Measured (us for both behind a router, weights in memory; before: sixteen warps that met at every tile, a down kernel whose registers kept it
// off every SM until the up kernel had left, its weights brought into L2 by the up kernel): 32 experts of 704, 4 used, a shared one of
// 1,408, 2,048 wide: one token 20.4 -> 17.6, 3 34.0 -> 31.9, 8 55.5 -> 51.6; 8 experts of 5,632, 2 used: 45.9 -> 40.5, 8 tokens 131 -> 109; 128 of
// 192, 8 used: 20.0 -> 14.5, 8 tokens 66.4 -> 51.0.  The up kernel bringing the down kernel's weights into L2 costs 2 to 11 us of that;
// rings of 4 to 6 boxes in the up kernel (and fewer in the other, or one CTA an SM) 1 to 7 us.
#include "common.cuh"
#include "experts.cuh"
#include "linear_stream.cuh"
#include "tma.cuh"

namespace {

using bf16 = __nv_bfloat16;
constexpr int MAX_M = 8, MAX_E = 256, WARPS = 8, THREADS = WARPS * 32, MEET = 4;  // MEET: tiles between two meetings of the up kernel
constexpr int UP_BOXK = 128, UP_KB = 2, UP_SLOTS = 3, UP_SLOT = 16 * UP_BOXK;  // elements of a slot; UP_KB: most boxes a warp has of a tile
constexpr int DOWN_BOXK = 64, DOWN_SLOTS = 3, DOWN_SLOT = (16 + MAX_M) * DOWN_BOXK;
constexpr size_t UP_SMEM = 1024 + (size_t)WARPS * UP_SLOTS * UP_SLOT * 2 + 2 * (size_t)MEET * WARPS * 32 * 16;
constexpr size_t DOWN_SMEM = 1024 + (size_t)WARPS * DOWN_SLOTS * DOWN_SLOT * 2 + (size_t)WARPS * 32 * 16;

struct Experts {
    const bf16 *x, *w_up, *w_down;
    bf16* act;  // [M, E * ff + fs]: only used blocks are written and read
    int ldx, M, K, N, E, ff, fs, kind;  // kind: -1 gated, else the activation
    float limit, limit_s, slope, up_shift;
    experts::Weights weights;
    float *out, *resid;  // out [M, N], or resid [M, N] += alpha * y
    const float* norm_w;  // with resid: xw_out = resid * norm_w, ss_out [N / 16, M] = sums of resid^2
    bf16* xw_out;
    float* ss_out;
    float alpha;
    int* error_flag;
};

using lin::feature_row;  // which row of eight in a box holds the weights of MMA row g

// both k-steps of a piece of 32 k: a0, a1: rows g and g + 8 of the weights, b: column g of the tokens
__device__ __forceinline__ void mma_piece(float (&c)[4], float (&d)[4], const uint4& a0, const uint4& a1, const uint4& b) {
    lin::mma_bf16(c, a0.x, a1.x, a0.y, a1.y, b.x, b.y);
    lin::mma_bf16(d, a0.z, a1.z, a0.w, a1.w, b.z, b.w);
}

// The used experts in ascending order, by the calling warp for itself (list: its own place), and where wt_s is given every token's weight of
// every expert and of the shared one.  Returns their number.
__device__ __forceinline__ int list_experts(const Experts& p, unsigned char* list, float (*wt_s)[MAX_E + 1]) {
    const int lane = threadIdx.x & 31;
    int n = 0;
    if (wt_s && lane < p.M && p.fs > 0) wt_s[lane][p.E] = p.weights.of(lane, p.E);
    for (int e0 = 0; e0 < p.E; e0 += 32) {
        const int e = e0 + lane;
        float wt[MAX_M];
        bool used = false;
#pragma unroll
        for (int m = 0; m < MAX_M; ++m) wt[m] = m < p.M && e < p.E ? p.weights.of(m, e) : 0.f;
#pragma unroll
        for (int m = 0; m < MAX_M; ++m) {
            used |= wt[m] != 0.f;
            if (wt_s && e < p.E) wt_s[m][e] = wt[m];
        }
        const unsigned mask = __ballot_sync(0xffffffffu, used);
        if (used) list[n + __popc(mask & ((1u << lane) - 1))] = (unsigned char)e;
        n += __popc(mask);
    }
    __syncwarp();
    return n;
}

// The warps' sums of a lane's four values, in order.
__device__ __forceinline__ void add_up(const float4* red, int lane, float (&s)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
        const float4 part = red[w * 32 + lane];
        s[0] += part.x; s[1] += part.y; s[2] += part.z; s[3] += part.w;
    }
}

// map: w_up in boxes of 8 (gated) or 16 rows and two neighbouring pieces of 64 k where `whole` (rows are whole pieces), else one piece.
__global__ void __maxnreg__(120) experts_up_kernel(const Experts p, const __grid_constant__ CUtensorMap map, const int whole) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ unsigned char lists[WARPS][MAX_E];
    __shared__ float wt_s[MAX_M][MAX_E + 1];
    __shared__ __align__(8) unsigned long long full[WARPS][UP_SLOTS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, fr = feature_row(g);
    bf16* rings = reinterpret_cast<bf16*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    bf16* ring = rings + (size_t)warp * UP_SLOTS * UP_SLOT;
    float4* red = reinterpret_cast<float4*>(rings + (size_t)WARPS * UP_SLOTS * UP_SLOT);  // [2][MEET][WARPS][32]
    const bool gated = p.kind < 0, known = p.weights.w == nullptr;  // the table's experts do not depend on the kernel in front
    const int step = gated ? 8 : 16, tiles_e = p.ff / step, tiles_s = p.fs / step, per = gated ? 2 : 1;
    const int kblocks = (p.K + UP_BOXK - 1) / UP_BOXK, my_kb = kblocks > warp ? (kblocks - 1 - warp) / WARPS + 1 : 0;
    unsigned long long* my_full = full[warp];
    unsigned char* list = lists[warp];
    if (lane == 0) {
        for (int s = 0; s < UP_SLOTS; ++s) tma::mbar_init(&my_full[s], 1);
        tma::mbar_fence_init();
        if (warp == 0) tma::prefetch_map(&map);
    }
    __syncwarp();
    int count = known ? list_experts(p, list, warp == 0 ? wt_s : nullptr) : 0;
    // tile v: the shared expert's first, then the listed experts'
    auto place = [&](int v, int& e, int& f0) {
        e = v < tiles_s ? p.E : list[(v - tiles_s) / tiles_e];
        f0 = (v < tiles_s ? v : (v - tiles_s) % tiles_e) * step;
    };
    auto tiles_of = [&](int total) { return (int)blockIdx.x < total ? (total - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0; };
    int tiles = tiles_of(tiles_s + count * tiles_e), armed = 0, a_tile = 0, a_kb = warp;
    // asks for the warp's next box (lane 0)
    auto arm = [&]() {
        int e, f0;
        place(blockIdx.x + a_tile * gridDim.x, e, f0);
        const int s = armed % UP_SLOTS, rows = gated ? 8 : 16;
        const int row = e * per * p.ff + f0;  // (of the gate, whose up rows lie ff or fs further)
        bf16* dst = ring + (size_t)s * UP_SLOT;
        tma::mbar_expect_tx(&my_full[s], UP_SLOT * 2);
        for (int half = 0; half < per; ++half, dst += 8 * UP_BOXK) {
            const int r = row + half * (e == p.E ? p.fs : p.ff);
            if (whole) tma::load_3d(dst, &map, 0, r, a_kb * 2, &my_full[s]);
            else {
                tma::load_2d(dst, &map, a_kb * UP_BOXK, r, &my_full[s]);
                tma::load_2d(dst + rows * 64, &map, a_kb * UP_BOXK + 64, r, &my_full[s]);
            }
        }
        ++armed;
        a_kb += WARPS;
        if (a_kb >= kblocks) {
            a_kb = warp;
            ++a_tile;
        }
    };
    auto fill = [&](int consumed) {
        if (lane == 0)
            while (armed < tiles * my_kb && armed < consumed + UP_SLOTS) arm();
    };
    fill(0);
    pdl_wait();
    pdl_trigger();  // behind the wait: see above
    uint4 xb[UP_KB][4];
#pragma unroll
    for (int j = 0; j < UP_KB; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = (warp + j * WARPS) * UP_BOXK + i * 32;
            xb[j][i] = k < p.K && g < p.M ? __ldcg(reinterpret_cast<const uint4*>(p.x + (size_t)g * p.ldx + k + q * 8)) : make_uint4(0, 0, 0, 0);
        }
    if (!known) {
        count = list_experts(p, list, warp == 0 ? wt_s : nullptr);
        tiles = tiles_of(tiles_s + count * tiles_e);
        fill(0);
    }
    const int lda = p.E * p.ff + p.fs;
    int unit = 0;
    bool gave_up = false;
    for (int t0 = 0, round = 0; t0 < tiles; t0 += MEET, ++round) {
        const int t1 = min(tiles, t0 + MEET);
        float4* mine = red + (size_t)(round & 1) * MEET * WARPS * 32;
        for (int t = t0; t < t1; ++t) {
            float c[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < UP_KB; ++j) {
                if (j >= my_kb) break;
                const int s = unit % UP_SLOTS;
                if (!gave_up && !tma::mbar_wait(&my_full[s], (unit / UP_SLOTS) & 1)) {
                    gave_up = true;
                    if (p.error_flag) atomicExch(p.error_flag, 1);
                }
                // [2 pieces of 64 k][rows][64], the 16 bytes c of row r at c ^ (r & 7); gated: eight rows of the gate, then of the up
                const bf16* slot = ring + (size_t)s * UP_SLOT + fr * 64;
                uint4 a[4][2];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bf16* at = slot + (i >> 1) * (gated ? 8 * 64 : 16 * 64) + ((((i & 1) << 2) | q) ^ fr) * 8;
                    a[i][0] = *reinterpret_cast<const uint4*>(at);
                    a[i][1] = *reinterpret_cast<const uint4*>(at + (gated ? 8 * UP_BOXK : 8 * 64));
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) mma_piece(c, d, a[i][0], a[i][1], xb[j][i]);
                __syncwarp();  // the products have been issued: every lane's pieces are in registers, and the slot may take the next box
                ++unit;
                fill(unit);
            }
            mine[((t - t0) * WARPS + warp) * 32 + lane] = make_float4(c[0] + d[0], c[1] + d[1], c[2] + d[2], c[3] + d[3]);
        }
        __syncthreads();  // this buffer of sums is written again two meetings on
        for (int t = t0 + warp; t < t1; t += WARPS) {
            int e, f0;
            place(blockIdx.x + t * gridDim.x, e, f0);
            float sum[4];
            add_up(mine + (size_t)(t - t0) * WARPS * 32, lane, sum);
#pragma unroll
            for (int i = 0; i < 2; ++i) {  // token 2 q + i; sum[i]: row g, sum[i + 2]: row g + 8
                const int m = 2 * q + i;
                if (m >= p.M) continue;
                const float wt = wt_s[m][e];
                bf16* y = p.act + (size_t)m * lda + (size_t)e * p.ff + f0 + fr;
                if (gated) {
                    const float lim = e == p.E ? p.limit_s : p.limit, gc = fminf(sum[i], lim), uc = fminf(fmaxf(sum[i + 2], -lim), lim);
                    y[0] = __float2bfloat16_rn(wt == 0.f ? 0.f : gc / (1.f + expf(-p.slope * gc)) * (uc + p.up_shift) * wt);
                } else {
                    y[0] = __float2bfloat16_rn(wt == 0.f ? 0.f : experts::activate(sum[i], p.kind) * wt);
                    y[8] = __float2bfloat16_rn(wt == 0.f ? 0.f : experts::activate(sum[i + 2], p.kind) * wt);
                }
            }
        }
    }
    // every box that was asked for has been waited for; where a wait gave up, once more, so that no copy lands after the CTA has left
    if (gave_up && lane == 0)
        for (int n = max(0, armed - UP_SLOTS); n < armed; ++n) tma::mbar_wait(&my_full[n % UP_SLOTS], (n / UP_SLOTS) & 1);
}

// map: w_down in boxes of 16 rows and 64 columns; act_map: act in boxes of 8 rows (what is not there reads as zeros) and 64 columns.
__global__ void __maxnreg__(120) experts_down_kernel(const Experts p, const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap act_map) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ unsigned char lists[WARPS][MAX_E];
    __shared__ __align__(8) unsigned long long full[WARPS][DOWN_SLOTS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, fr = feature_row(g);
    bf16* rings = reinterpret_cast<bf16*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    bf16* ring = rings + (size_t)warp * DOWN_SLOTS * DOWN_SLOT;
    float4* red = reinterpret_cast<float4*>(rings + (size_t)WARPS * DOWN_SLOTS * DOWN_SLOT);  // [WARPS][32]
    const int n0 = blockIdx.x * 16, boxes_e = (p.ff + DOWN_BOXK - 1) / DOWN_BOXK, boxes_s = (p.fs + DOWN_BOXK - 1) / DOWN_BOXK;
    unsigned long long* my_full = full[warp];
    unsigned char* list = lists[warp];
    if (lane == 0) {
        for (int s = 0; s < DOWN_SLOTS; ++s) tma::mbar_init(&my_full[s], 1);
        tma::mbar_fence_init();
        if (warp == 0) {
            tma::prefetch_map(&map);
            tma::prefetch_map(&act_map);
        }
    }
    __syncwarp();
    pdl_trigger();
    const int count = list_experts(p, list, nullptr);  // the router ended before the up kernel let this one start
    // The warp's boxes: those whose number among all of w_down's (boxes_e an expert, the shared one's last) is the warp's own modulo WARPS,
    // of the shared expert, then of the listed ones.  So the order of a token's sums does not depend on the experts of others, whose
    // boxes in between add zeros.
    struct Walk {
        int block, box;  // block -1: the shared expert's
    };
    auto expert = [&](const Walk& w) { return w.block < 0 ? p.E : (int)list[w.block]; };
    auto enter = [&](Walk& w) { w.box = w.block < count ? (warp - expert(w) * boxes_e) & (WARPS - 1) : 0; };
    // moves on to a box that exists; false: none is left
    auto settle = [&](Walk& w) {
        while (w.block < count && w.box >= (w.block < 0 ? boxes_s : boxes_e)) {
            ++w.block;
            enter(w);
        }
        return w.block < count;
    };
    Walk ask = {-1, 0};
    enter(ask);
    Walk use = ask;
    int armed = 0;
    bool may_read = false;  // the tokens' lanes are there
    auto column = [&](const Walk& w) { return expert(w) * p.ff + w.box * DOWN_BOXK; };
    auto fill = [&](int consumed) {  // lane 0
        while (armed < consumed + DOWN_SLOTS && settle(ask)) {
            const int s = armed % DOWN_SLOTS, k = column(ask);
            bf16* dst = ring + (size_t)s * DOWN_SLOT;
            tma::mbar_expect_tx(&my_full[s], DOWN_SLOT * 2);
            tma::load_2d(dst, &map, k, n0, &my_full[s]);
            if (may_read) tma::load_2d(dst + 16 * DOWN_BOXK, &act_map, k, 0, &my_full[s]);
            ++armed;
            ask.box += WARPS;
        }
    };
    if (lane == 0) fill(0);
    pdl_wait();
    if (lane == 0) {
        may_read = true;
        Walk w = use;
        for (int n = 0; n < armed; ++n, w.box += WARPS)
            if (settle(w)) tma::load_2d(ring + (size_t)n * DOWN_SLOT + 16 * DOWN_BOXK, &act_map, column(w), 0, &my_full[n]);
    }
    // what the end needs besides the sums
    float before[4] = {0.f, 0.f, 0.f, 0.f}, norm_w[2] = {0.f, 0.f};
    if (warp == 0 && p.resid) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int m = 2 * q + (i & 1), n = n0 + fr + (i >> 1) * 8;
            if (m < p.M) before[i] = __ldcg(p.resid + (size_t)m * p.N + n);
            if (p.norm_w) norm_w[i >> 1] = p.norm_w[n];
        }
    }
    float c[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
    int unit = 0;
    bool gave_up = false;
    for (; settle(use); use.box += WARPS) {
        const int s = unit % DOWN_SLOTS;
        if (!gave_up && !tma::mbar_wait(&my_full[s], (unit / DOWN_SLOTS) & 1)) {
            gave_up = true;
            if (p.error_flag) atomicExch(p.error_flag, 1);
        }
        const bf16 *w = ring + (size_t)s * DOWN_SLOT + fr * 64, *x = ring + (size_t)s * DOWN_SLOT + 16 * DOWN_BOXK + g * 64;
        uint4 a[2][2], b[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            a[i][0] = *reinterpret_cast<const uint4*>(w + (((i << 2) | q) ^ fr) * 8);
            a[i][1] = *reinterpret_cast<const uint4*>(w + 8 * 64 + (((i << 2) | q) ^ fr) * 8);
            b[i] = *reinterpret_cast<const uint4*>(x + (((i << 2) | q) ^ g) * 8);
        }
        mma_piece(c, d, a[0][0], a[0][1], b[0]);
        // an expert's last box may hold 32 columns of its neighbour
        if (use.box * DOWN_BOXK + 32 < (use.block < 0 ? p.fs : p.ff)) mma_piece(c, d, a[1][0], a[1][1], b[1]);
        __syncwarp();  // the products have been issued: every lane's pieces are in registers, and the slot may take the next box
        ++unit;
        if (lane == 0) fill(unit);
    }
    red[warp * 32 + lane] = make_float4(c[0] + d[0], c[1] + d[1], c[2] + d[2], c[3] + d[3]);
    if (gave_up && lane == 0)
        for (int n = max(0, armed - DOWN_SLOTS); n < armed; ++n) tma::mbar_wait(&my_full[n % DOWN_SLOTS], (n / DOWN_SLOTS) & 1);
    __syncthreads();
    if (warp != 0) return;
    float s[4], ss[2] = {0.f, 0.f};
    add_up(red, lane, s);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = 2 * q + (i & 1), n = n0 + fr + (i >> 1) * 8;
        if (m >= p.M) continue;
        const size_t at = (size_t)m * p.N + n;
        if (!p.resid) {
            p.out[at] = s[i];
            continue;
        }
        const float r = fmaf(p.alpha, s[i], before[i]);
        p.resid[at] = r;
        if (p.norm_w) {
            p.xw_out[at] = __float2bfloat16_rn(r * norm_w[i >> 1]);
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
    if (M > MAX_M || K < 32 || K > WARPS * UP_KB * UP_BOXK || (K & 31) || ff < 32 || (ff & 31) || (fs & 31) || N < 16 || (N & 15) || E < 1 || E > MAX_E ||
        (ldx & 7) || !aligned(x) || !aligned(w_up) || !aligned(w_down) || !aligned(act))
        return LLM_ERR_UNSUPPORTED;
    Experts p = {};
    p.x = (const bf16*)x; p.w_up = (const bf16*)w_up; p.w_down = (const bf16*)w_down; p.act = (bf16*)act;
    p.ldx = ldx; p.M = M; p.K = K; p.N = N; p.E = E; p.ff = ff; p.fs = fs; p.kind = kind;
    p.limit = limit; p.limit_s = limit_s; p.slope = slope; p.up_shift = up_shift;
    p.weights = {weights, ldw, ids, table, top, vocab, E};
    p.out = out; p.resid = resid; p.norm_w = norm_w; p.xw_out = (bf16*)xw_out; p.ss_out = ss_out; p.alpha = alpha; p.error_flag = error_flag;
    const int sms = device_sms(), per = kind < 0 ? 2 : 1, C = E * ff + fs;
    const bool whole = K % 64 == 0;  // rows are whole pieces of 64 k: two of them in one box
    CUtensorMap up_map, down_map, act_map;
    if (!(whole ? tma::make_map_row_pieces_bf16(&up_map, w_up, (uint64_t)per * C, K, kind < 0 ? 8 : 16)
                : tma::make_map_2d_bf16(&up_map, w_up, (uint64_t)per * C, K, K, kind < 0 ? 8 : 16, 64, CU_TENSOR_MAP_SWIZZLE_128B)))
        return LLM_ERR_UNSUPPORTED;
    if (!tma::cached_map_2d_bf16(&down_map, w_down, N, C, C, 16, DOWN_BOXK, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !tma::make_map_2d_bf16(&act_map, act, M, C, C, MAX_M, DOWN_BOXK, CU_TENSOR_MAP_SWIZZLE_128B))
        return LLM_ERR_UNSUPPORTED;
    // at every launch: the limits hold for the current device, and a process may have several; all of the SM's memory as shared memory, so
    // that CTAs of both kernels share it
    for (int k = 0; k < 2; ++k) {
        const void* kernel = k == 0 ? (const void*)experts_up_kernel : (const void*)experts_down_kernel;
        cudaError_t set = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(k == 0 ? UP_SMEM : DOWN_SMEM));
        if (set == cudaSuccess) set = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (set != cudaSuccess) return (int)set;
    }
    const int most = (E * ff + fs) / (kind < 0 ? 8 : 16);
    const int code = launch_pdl(experts_up_kernel, dim3(most < sms ? most : sms), dim3(THREADS), UP_SMEM, stream, p, up_map, (int)whole);
    return code != 0 ? code : launch_pdl(experts_down_kernel, dim3(N / 16), dim3(THREADS), DOWN_SMEM, stream, p, down_map, act_map);
}
