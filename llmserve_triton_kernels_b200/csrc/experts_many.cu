// A mixture of small feed-forward layers for prompts (bfloat16): every token's rows go through the experts that it uses and no others.
//
//   sort     per expert, the tokens that use it, in order (a CTA an expert)
//   gather   the experts' rows of x one after the other (in the place that y takes later)
//   up       act[row, j] = act(x[token of row] W_up^T) * weight          (gated: gate and up rows of the same feature in one tile)
//   down     y[row, n] = act[row] W_down[:, the expert's columns]^T      (32 bits)
//   combine  out[t] = sum of the token's rows in the order of the experts + the shared expert's row, plain or into the residual stream
//
// What bounds it: the weights' bytes up to about 1,500 tokens (32 experts of 704 in 2,048: 294 MB a layer), beyond that the tensor cores; the
// products over all experts with the token's weight as a factor, which ran before, did eight times the operations for 4 of 32 experts.
// Measured (us a layer, launches back to back, weights from memory; products over all experts -> these launches): 32 experts of 704, 4 used, a
// shared one of 1,408, 2,048 wide: 256 tokens 88 -> 78, 512 127 -> 89, 1,024 222 -> 121, 1,801 383 -> 183 (up 89 at 0.42 of the tensor peak, down
// 67, combine 19, gather 8, sort 6).  Rows gathered by the product itself (TMA, four rows a box) were no faster than all experts.
//
// The products are tcgen05 with the WEIGHTS as the 128 rows of the tile and an expert's tokens as its columns: an expert has as many
// tokens as it has, and N goes up to 64, 128 or 256 (the fewer, the deeper the ring) in steps of 16 where M is 128 whatever there is to do.  One persistent CTA an SM walks (group,
// tile of features, tile of tokens), the shared expert's tiles first (the largest), token tiles innermost so that neighbours in time share
// weights in L2.  Warp 0 brings operands by TMA through a ring of slots (where the experts are gated a box of eight rows of gate, of up, of
// gate ..., so that a feature's two sums lie eight lanes apart in tensor memory), warp 1 issues the products into one of two accumulators,
// warps 2-5 end the tile before meanwhile.
// Every wait is bounded; one that gives up sets the error flag, and the roles run to their end.
#include "common.cuh"
#include "experts.cuh"
#include "tma.cuh"
#include "umma.cuh"

#include <type_traits>

namespace {

using bf16 = __nv_bfloat16;
constexpr int MAX_E = 256, BM = 128, BK = 64, THREADS = 192;
constexpr int A_BYTES = BM * BK * 2, X_BOX = 32;
constexpr int CHUNK = 32;  // tokens that the epilogue turns round in shared memory at a time

struct Many {
    int T, K, N, E, ff, fs, cap;  // cap: rows of act and y (tokens x experts of a token)
    int kind;                     // -1 gated, else the activation
    float limit, limit_s, slope, up_shift;
    experts::Weights weights;
    int *counts, *list, *place;  // [E], [E, T] tokens of an expert, [T, E] a token's row among its expert's
    bf16 *act, *act_s;           // [cap, ff], [T, fs]
    float *y, *y_s;              // [cap, N], [T, N]
    float *out, *resid;          // out [T, N], or resid [T, N] += alpha * sum
    float alpha;
    int* error_flag;
};

__global__ void __launch_bounds__(1024) experts_sort_kernel(const Many p) {
    __shared__ int of_warp[32];
    const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    pdl_trigger();
    pdl_wait();
    int base = 0;
    for (int t0 = 0; t0 < p.T; t0 += blockDim.x) {
        const int t = t0 + threadIdx.x;
        const bool uses = t < p.T && p.weights.of(t, e) != 0.f;
        const unsigned mask = __ballot_sync(0xffffffffu, uses);
        if (lane == 0) of_warp[warp] = __popc(mask);
        __syncthreads();
        const int c = lane < warps ? of_warp[lane] : 0;
        const int before = __reduce_add_sync(0xffffffffu, lane < warp ? c : 0), all = __reduce_add_sync(0xffffffffu, c);
        if (uses) {
            const int at = base + before + __popc(mask & ((1u << lane) - 1));
            p.list[(size_t)e * p.T + at] = t;
            p.place[(size_t)t * p.E + e] = at;
        }
        base += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) p.counts[e] = base;
}

// Where the experts' rows and tiles start.  Group 0 is the shared expert, group e + 1 expert e.
struct Groups {
    int row0[MAX_E + 1], rows[MAX_E + 1], tile0[MAX_E + 2];
};

template <int NT>
__device__ __forceinline__ int token_tiles(int rows) { return (rows + NT - 1) / NT; }

__device__ __forceinline__ int sum_up_to(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += up;
    }
    return v;
}

// By one warp; the caller meets before it reads.  NT: most tokens of a tile.
template <int NT>
__device__ __forceinline__ void find_groups(const Many& p, Groups* g, int tiles_s, int tiles_e) {
    const int lane = threadIdx.x & 31;
    int rows = 0, tiles = p.fs > 0 ? tiles_s * token_tiles<NT>(p.T) : 0;
    if (lane == 0) {
        g->row0[0] = 0;
        g->rows[0] = p.fs > 0 ? p.T : 0;
        g->tile0[0] = 0;
        g->tile0[1] = tiles;
    }
    for (int e0 = 0; e0 < p.E; e0 += 32) {
        const int e = e0 + lane;
        const int mine = e < p.E ? __ldcg(p.counts + e) : 0, sum = sum_up_to(mine, lane);
        // a token has no more experts than the caller made room for; whatever the counts say, nobody leaves the buffers
        const int from = min(rows + sum - mine, p.cap), n = min(mine, p.cap - from);
        const int t_sum = sum_up_to(tiles_e * token_tiles<NT>(n), lane);
        if (e < p.E) {
            g->row0[e + 1] = from;
            g->rows[e + 1] = n;
            g->tile0[e + 2] = tiles + t_sum;
        }
        rows += __shfl_sync(0xffffffffu, sum, 31);
        tiles += __shfl_sync(0xffffffffu, t_sum, 31);
    }
}

// A tile: the group's features from f0 on, its rows [row, row + valid), n = valid rounded up to 16.
struct Tile {
    int group, f0, row, valid, n;
};

// `cursor`: the last group looked at (tiles are walked in order).
template <int NT>
__device__ __forceinline__ Tile tile_at(const Groups& g, int tile, int& cursor, int step) {
    while (tile >= g.tile0[cursor + 1]) ++cursor;
    const int rows = g.rows[cursor], over = token_tiles<NT>(rows), each = ((rows + over - 1) / over + 15) & ~15;
    const int local = tile - g.tile0[cursor];
    Tile t;
    t.group = cursor;
    t.f0 = (local / over) * step;
    t.row = (local % over) * each;
    t.valid = min(each, rows - t.row);
    t.n = (max(t.valid, 1) + 15) & ~15;
    return t;
}

__device__ __forceinline__ void load_5d(void* smem, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4, unsigned long long* bar) {
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];\n"
                 ::"r"(tma::smem_addr(smem)), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(tma::smem_addr(bar)) : "memory");
}

// Whether one of the 128 threads that end tiles says so.
__device__ __forceinline__ bool any_of_128(bool mine) {
    unsigned any;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.or.pred q, 1, 128, p;\nselp.u32 %0, 1, 0, q;\n}\n" : "=r"(any) : "r"((unsigned)mine) : "memory");
    return any != 0;
}
__device__ __forceinline__ void meet_128() { asm volatile("barrier.cta.sync 1, 128;\n" ::: "memory"); }

enum { UP, UP_GATED, DOWN, DOWN_RAGGED };  // ragged: experts whose columns do not fill their last box

// rows: the experts' rows of x (up) or of act (down); rows_s: x, or the shared expert's act, all in boxes of X_BOX rows;
// w, w_s: the experts' and the shared expert's matrix (the same map but where they are gated or ragged).
template <int WHAT, int NT, int STAGES>
__global__ void __launch_bounds__(THREADS)
experts_product_kernel(const Many p, const __grid_constant__ CUtensorMap rows_map, const __grid_constant__ CUtensorMap rows_s_map,
                       const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap w_s_map) {
    constexpr bool IS_UP = WHAT == UP || WHAT == UP_GATED;
    constexpr int STEP = WHAT == UP_GATED ? 64 : 128;  // features a tile
    constexpr int SLOT_BYTES = A_BYTES + NT * BK * 2;
    constexpr int PITCH = STEP * 2 + 32;               // bytes from token to token in the epilogue's pieces
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* turn = ring + (size_t)STAGES * SLOT_BYTES;  // [2][CHUNK][PITCH]
    __shared__ __align__(8) unsigned long long full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], drained;
    __shared__ Groups groups;
    __shared__ float factor[NT];
    __shared__ unsigned tmem_base;
    __shared__ volatile int gave_up;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) {
            tma::mbar_init(&full[s], 1);
            tma::mbar_init(&empty[s], 1);
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            tma::mbar_init(&acc_full[b], 1);
            tma::mbar_init(&acc_empty[b], 4);
        }
        tma::mbar_init(&drained, 1);
        gave_up = 0;
        tma::mbar_fence_init();
        tma::prefetch_map(&rows_map);
        tma::prefetch_map(&rows_s_map);
        tma::prefetch_map(&w_map);
        tma::prefetch_map(&w_s_map);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tma::smem_addr(&tmem_base)), "n"(2 * NT) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    pdl_trigger();
    pdl_wait();
    const int width_e = IS_UP ? p.ff : p.N, width_s = IS_UP ? p.fs : p.N;
    if (warp == 0) find_groups<NT>(p, &groups, (width_s + STEP - 1) / STEP, (width_e + STEP - 1) / STEP);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const int tiles = groups.tile0[p.E + 1];

    auto fail = [&]() {
        gave_up = 1;
        if (p.error_flag) atomicExch(p.error_flag, 1);
    };
    auto inner = [&](int group) { return IS_UP ? p.K : group == 0 ? p.fs : p.ff; };

    int cursor = 0;
    if (warp == 0) {
        // ---- producer: a lane a box ----
        int it = 0;
        bool ok = true;  // the same in all lanes
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            const Tile t = tile_at<NT>(groups, tile, cursor, STEP);
            const bool shared = t.group == 0;
            const int e = t.group - 1, kblocks = (inner(t.group) + BK - 1) / BK;
            const int n_boxes = (t.n + X_BOX - 1) / X_BOX, row = groups.row0[t.group] + t.row + lane * X_BOX;
            const unsigned bytes = A_BYTES + n_boxes * X_BOX * BK * 2;
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const int s = it % STAGES;
                ok = (it < STAGES || tma::mbar_wait(&empty[s], ((it / STAGES) - 1) & 1)) && !gave_up;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                unsigned char *a = ring + (size_t)s * SLOT_BYTES, *b = a + A_BYTES;
                if (lane == 0) {
                    tma::mbar_expect_tx(&full[s], bytes);
                    if constexpr (WHAT == UP_GATED) load_5d(a, shared ? &w_s_map : &w_map, kb * BK, 0, 0, t.f0 / 8, shared ? 0 : e, &full[s]);
                    else if constexpr (WHAT == UP) tma::load_2d(a, &w_map, kb * BK, (shared ? p.E : e) * p.ff + t.f0, &full[s]);
                    else if constexpr (WHAT == DOWN_RAGGED) tma::load_3d(a, shared ? &w_s_map : &w_map, kb * BK, shared ? 0 : e, t.f0, &full[s]);
                    else tma::load_2d(a, &w_map, (shared ? p.E : e) * p.ff + kb * BK, t.f0, &full[s]);
                }
                __syncwarp();
                if (lane < n_boxes) tma::load_2d(b + (size_t)lane * X_BOX * BK * 2, shared ? &rows_s_map : &rows_map, kb * BK, row, &full[s]);
            }
        }
        if (!ok) {
            if (lane == 0) fail();
            // nothing lands in this memory after the CTA has left it
            for (int k = max(0, it - STAGES); k < it; ++k) tma::mbar_wait(&full[k % STAGES], (k / STAGES) & 1);
        }
    } else if (warp == 1) {
        // ---- tensor-core issuer: one elected lane; the others keep it company so that the descriptors stay uniform ----
        unsigned elected;
        asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(elected));
        int it = 0, i = 0;
        bool ok = true;  // the same in all lanes
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++i) {
            const Tile t = tile_at<NT>(groups, tile, cursor, STEP);
            const int kblocks = (inner(t.group) + BK - 1) / BK;
            const unsigned idesc = umma::idesc_bf16(BM, t.n, false);
            const int buf = i & 1;
            const unsigned d_tmem = tmem_base + buf * NT;
            ok = __all_sync(0xffffffffu, i < 2 || tma::mbar_wait(&acc_empty[buf], ((i >> 1) - 1) & 1));
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            for (int kb = 0; kb < kblocks && ok; ++kb, ++it) {
                const int s = it % STAGES;
                ok = __all_sync(0xffffffffu, !gave_up && tma::mbar_wait(&full[s], (it / STAGES) & 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const unsigned char* slot = ring + (size_t)s * SLOT_BYTES;
                const unsigned long long a = umma::desc_sw128(slot), b = umma::desc_sw128(slot + A_BYTES);
                if (elected) {
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma::mma_bf16(d_tmem, a + 2 * k, b + 2 * k, idesc, (kb | k) != 0);
                    umma::commit(&empty[s]);
                }
            }
            if (ok && elected) umma::commit(&acc_full[buf]);
        }
        if (!ok) {
            if (elected) {
                fail();
                umma::commit(&drained);
            }
            __syncwarp();
            tma::mbar_wait(&drained, 0);
        }
    } else {
        // ---- the tiles' ends: a warp has the 32 features of its lanes of tensor memory, a token a column ----
        const int quarter = warp & 3, mine = threadIdx.x - 64;  // mine: 0 .. 127
        int i = 0, piece = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++i) {
            const Tile t = tile_at<NT>(groups, tile, cursor, STEP);
            const bool shared = t.group == 0;
            const int e = t.group - 1, buf = i & 1;
            const size_t row0 = (size_t)groups.row0[t.group] + t.row;
            if constexpr (IS_UP) {  // the tokens' weights of this expert, once everybody has read those of the tile before
                meet_128();
                for (int c = mine; c < NT; c += 128) {
                    const int token = c < t.valid ? (shared ? t.row + c : __ldcg(p.list + (size_t)e * p.T + t.row + c)) : -1;
                    factor[c] = token >= 0 ? p.weights.of(token, shared ? p.E : e) : 0.f;
                }
            }
            const bool ok = !gave_up && tma::mbar_wait(&acc_full[buf], (i >> 1) & 1);
            if (!ok) fail();
            if (any_of_128(!ok)) break;  // the four warps meet in a tile's pieces: they leave together
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const unsigned lane_base = tmem_base + buf * NT + ((unsigned)(quarter * 32) << 16);
            if constexpr (!IS_UP) {
                const int n = t.f0 + quarter * 32 + lane;
                float* y = (shared ? p.y_s : p.y) + row0 * p.N + n;
#pragma unroll 1
                for (int c = 0; c < t.n; c += 32) {
                    float v[32];
                    umma::tmem_ld32(lane_base + c, v);
                    if (n < p.N) {
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (c + j < t.valid) y[(size_t)(c + j) * p.N] = v[j];
                    }
                }
            } else {
                const float limit = shared ? p.limit_s : p.limit;
                const int width = shared ? p.fs : p.ff;
                bf16* act = (shared ? p.act_s : p.act) + row0 * width + t.f0;
#pragma unroll 1
                for (int c = 0; c < t.n; c += CHUNK, ++piece) {
                    float v[32];
                    umma::tmem_ld32(lane_base + c, v);
                    unsigned char* dst = turn + (size_t)(piece & 1) * CHUNK * PITCH;
                    if constexpr (WHAT == UP_GATED) {
                        // lanes 0-7 (16-23) have the gate's sums of eight features, lanes 8-15 (24-31) the up's: each takes every
                        // other token and gets what it lacks
                        const bool has_up = lane & 8;
                        unsigned char* at = dst + (quarter * 16 + (lane >> 4) * 8 + (lane & 7)) * 2 + (has_up ? PITCH : 0);
                        const float* f = factor + c + (has_up ? 1 : 0);  // (c is a multiple of 32 below NT)
#pragma unroll
                        for (int j = 0; j < 32; j += 2) {
                            const float other = __shfl_xor_sync(0xffffffffu, has_up ? v[j] : v[j + 1], 8);
                            const float g = fminf(has_up ? other : v[j], limit), u = fminf(fmaxf(has_up ? v[j + 1] : other, -limit), limit);
                            *reinterpret_cast<bf16*>(at + j * PITCH) = __float2bfloat16_rn(g / (1.f + expf(-p.slope * g)) * (u + p.up_shift) * f[j]);
                        }
                    } else {
                        unsigned char* at = dst + (quarter * 32 + lane) * 2;
#pragma unroll
                        for (int j = 0; j < 32; ++j) *reinterpret_cast<bf16*>(at + j * PITCH) = __float2bfloat16_rn(experts::activate(v[j], p.kind) * factor[c + j]);
                    }
                    meet_128();
                    for (int q = mine; q < CHUNK * (STEP / 8); q += 128) {
                        const int token = q / (STEP / 8), f = (q % (STEP / 8)) * 8;
                        if (c + token < t.valid && t.f0 + f < width)
                            *reinterpret_cast<uint4*>(act + (size_t)(c + token) * width + f) = *reinterpret_cast<const uint4*>(dst + token * PITCH + f * 2);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) tma::mbar_arrive(&acc_empty[buf]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "n"(2 * NT) : "memory");
    }
}

// The rows of token t among the experts', in the order of the experts, by one warp; returns their number.
__device__ __forceinline__ int rows_of_token(const Many& p, int t, int* rows) {
    const int lane = threadIdx.x & 31;
    int before = 0, n = 0;
    for (int e0 = 0; e0 < p.E; e0 += 32) {
        const int e = e0 + lane;
        const int mine = e < p.E ? __ldcg(p.counts + e) : 0, sum = sum_up_to(mine, lane);
        const bool uses = e < p.E && p.weights.of(t, e) != 0.f;
        const int at = uses ? __ldcg(p.place + (size_t)t * p.E + e) : 0;
        const unsigned mask = __ballot_sync(0xffffffffu, uses);
        if (uses) rows[n + __popc(mask & ((1u << lane) - 1))] = min(before + sum - mine + at, p.cap - 1);
        n += __popc(mask);
        before += __shfl_sync(0xffffffffu, sum, 31);
    }
    return n;
}

// One CTA a token: its row of x to each of its experts.
__global__ void __launch_bounds__(128) experts_gather_kernel(const Many p, const bf16* __restrict__ x, int ldx, bf16* __restrict__ xs) {
    __shared__ int rows[MAX_E];
    __shared__ int count;
    const int t = blockIdx.x;
    pdl_trigger();
    pdl_wait();
    if (threadIdx.x < 32) {
        const int n = rows_of_token(p, t, rows);
        if (threadIdx.x == 0) count = n;
    }
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)t * ldx);
    uint4 v[2];  // the first two pieces are on their way before the rows are known
#pragma unroll
    for (int i = 0; i < 2; ++i) v[i] = (int)threadIdx.x + 128 * i < p.K / 8 ? src[threadIdx.x + 128 * i] : make_uint4(0, 0, 0, 0);
    __syncthreads();
    const int n = count;
    for (int i = threadIdx.x, j = 0; i < p.K / 8; i += 128, ++j) {
        const uint4 u = j < 2 ? v[j & 1] : src[i];
        for (int k = 0; k < n; ++k) reinterpret_cast<uint4*>(xs + (size_t)rows[k] * p.K)[i] = u;
    }
}

// One CTA a token.  Bound by memory: top + 1 rows of y read (32 bits), one written.
__global__ void __launch_bounds__(256) experts_combine_kernel(const Many p) {
    __shared__ int rows[MAX_E];
    __shared__ int count;
    const int t = blockIdx.x;
    pdl_trigger();
    pdl_wait();
    if (threadIdx.x < 32) {
        const int n = rows_of_token(p, t, rows);
        if (threadIdx.x == 0) count = n;
    }
    __syncthreads();
    const int n = count;
    for (int c = threadIdx.x * 4; c < p.N; c += blockDim.x * 4) {
        float shared[4] = {0.f, 0.f, 0.f, 0.f}, before[4] = {0.f, 0.f, 0.f, 0.f}, sum[4] = {0.f, 0.f, 0.f, 0.f};
        if (p.fs > 0) load4(p.y_s + (size_t)t * p.N + c, shared);
        if (p.resid) load4(p.resid + (size_t)t * p.N + c, before);
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
            float v[4];
            load4(p.y + (size_t)rows[k] * p.N + c, v);
#pragma unroll
            for (int j = 0; j < 4; ++j) sum[j] += v[j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            sum[j] += shared[j];
            if (p.resid) sum[j] = fmaf(p.alpha, sum[j], before[j]);
        }
        store4((p.resid ? p.resid : p.out) + (size_t)t * p.N + c, sum);
    }
}

// The gate and up rows of `experts` equal experts, [experts][2][ff][K], as (k, row of eight, gate or up, run of eight, expert).
bool make_gated_map(CUtensorMap* map, const bf16* w, int experts, int ff, int K) {
    tma::EncodeTiledFn fn = tma::encode_fn();
    if (!fn) return false;
    const cuuint64_t row = (cuuint64_t)K * 2;
    const cuuint64_t dims[5] = {(cuuint64_t)K, 8, 2, (cuuint64_t)(ff / 8), (cuuint64_t)experts};
    const cuuint64_t strides[4] = {row, row * ff, row * 8, row * ff * 2};
    const cuuint32_t box[5] = {BK, 8, 2, 8, 1}, elem[5] = {1, 1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(w), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The columns of `experts` experts' down matrix, rows [N] of C columns, as (column of an expert, expert, row): what a box holds behind an
// expert's last column is zeros, not the next expert's (whose weights may hold no number).  Experts that are whole boxes have a map of two
// dimensions and a kernel of their own: with three dimensions, or a choice at every box, the layer takes 1 to 5 % longer (32 experts of 704, 256
// tokens: 77.0 us, 80.3).
bool make_down_map(CUtensorMap* map, const bf16* w, int experts, int ff, int N, uint64_t C) {
    tma::EncodeTiledFn fn = tma::encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)ff, (cuuint64_t)experts, (cuuint64_t)N};
    const cuuint64_t strides[2] = {(cuuint64_t)ff * 2, C * 2};
    const cuuint32_t box[3] = {BK, 1, BM}, elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(w), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int WHAT, int NT, int STAGES>
int launch_product(const Many& p, const CUtensorMap& rows, const CUtensorMap& rows_s, const CUtensorMap& w, const CUtensorMap& w_s, cudaStream_t stream) {
    constexpr int STEP = WHAT == UP_GATED ? 64 : 128;
    constexpr size_t smem = (size_t)STAGES * (A_BYTES + NT * BK * 2) + 1024 + (WHAT == UP || WHAT == UP_GATED ? 2 * CHUNK * (STEP * 2 + 32) : 0);
    auto kernel = experts_product_kernel<WHAT, NT, STAGES>;
    // at every launch: the limit holds for the current device, and a process may have several
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    return launch_pdl(kernel, dim3(device_sms()), dim3(THREADS), smem, stream, p, rows, rows_s, w, w_s);
}

}  // namespace

// x [T, K] (row stride ldx) through the used experts: arguments as llm_experts_few, any number of tokens.  cap: rows that act [cap, ff] and
// y [cap, N] have room for (tokens x experts of a token); act_s [T, fs] and y_s [T, N] for the shared expert; ints: E + 2 E T words.  width: most tokens of a tile,
// 64, 128 or 256.
// Needs K, ff and fs multiples of 8, N a multiple of 4, K <= 2 N, E <= 256; LLM_ERR_UNSUPPORTED otherwise, and then nothing has been launched.
LLM_EXPORT int llm_experts_many(const void* x, int ldx, const void* w_up, const void* w_down, int T, int K, int N, int E, int ff, int fs, int kind,
                                float limit, float limit_s, float slope, float up_shift, const float* weights, int ldw, const int* ids,
                                const int* table, int listed, int vocab, int* ints, int cap, void* act, void* act_s, float* y, float* y_s, float* out,
                                float* resid, float alpha, int width, int* error_flag, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (K < 8 || ff < 8 || ((K | ff | fs | ldx) & 7) || (N & 3) || N <= 0 || K > 2 * N || E < 1 || E > MAX_E || cap < 1 || fs < 0 || T > (1 << 20)) return LLM_ERR_UNSUPPORTED;
    if (((uintptr_t)x | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)act | (uintptr_t)act_s | (uintptr_t)y | (uintptr_t)y_s | (uintptr_t)out | (uintptr_t)resid) & 15)
        return LLM_ERR_UNSUPPORTED;
    const uint64_t C = (uint64_t)E * ff + fs;
    if (C > 0x7fffffffull) return LLM_ERR_UNSUPPORTED;
    if (!(weights || (ids && table)) || !(out || resid) || !act || !y || (fs > 0 && !(act_s && y_s))) return LLM_ERR_BAD_ARGUMENT;
    Many p = {};
    p.T = T; p.K = K; p.N = N; p.E = E; p.ff = ff; p.fs = fs; p.cap = cap; p.kind = kind;
    p.limit = limit; p.limit_s = limit_s; p.slope = slope; p.up_shift = up_shift;
    p.weights = {weights, ldw, ids, table, listed, vocab, E};
    p.counts = ints; p.list = ints + E; p.place = ints + E + (size_t)E * T;
    p.act = (bf16*)act; p.act_s = (bf16*)act_s; p.y = y; p.y_s = y_s; p.out = out; p.resid = resid; p.alpha = alpha; p.error_flag = error_flag;

    CUtensorMap x_rows, x_boxes, up, up_s, act_rows, act_s_rows, down, down_s;
    const CUtensorMapSwizzle sw = CU_TENSOR_MAP_SWIZZLE_128B;
    bf16* xs = reinterpret_cast<bf16*>(y);  // [cap, K]: read before the first y is written
    const bool ragged = ff % BK != 0;
    bool ok = tma::make_map_2d_bf16(&x_rows, xs, cap, K, K, X_BOX, BK, sw) && tma::make_map_2d_bf16(&x_boxes, x, T, K, ldx, X_BOX, BK, sw) &&
              tma::make_map_2d_bf16(&act_rows, act, cap, ff, ff, X_BOX, BK, sw) &&
              (ragged ? make_down_map(&down, (const bf16*)w_down, E, ff, N, C) : tma::make_map_2d_bf16(&down, w_down, N, C, C, BM, BK, sw));
    if (kind < 0) ok = ok && make_gated_map(&up, (const bf16*)w_up, E, ff, K);
    else ok = ok && tma::make_map_2d_bf16(&up, w_up, C, K, K, BM, BK, sw);
    act_s_rows = act_rows;
    up_s = up;
    down_s = down;
    if (ok && fs > 0) {
        ok = tma::make_map_2d_bf16(&act_s_rows, act_s, T, fs, fs, X_BOX, BK, sw);
        if (kind < 0) ok = ok && make_gated_map(&up_s, (const bf16*)w_up + (size_t)E * 2 * ff * K, 1, fs, K);
        if (ragged) ok = ok && make_down_map(&down_s, (const bf16*)w_down + (size_t)E * ff, 1, fs, N, C);
    }
    if (!ok) return LLM_ERR_UNSUPPORTED;
    const int threads = T >= 1024 ? 1024 : (T + 31) & ~31;
    int code = launch_pdl(experts_sort_kernel, dim3(E), dim3(threads), 0, stream, p);
    if (code) return code;
    code = launch_pdl(experts_gather_kernel, dim3(T), dim3(128), 0, stream, p, (const bf16*)x, ldx, xs);
    if (code) return code;
    auto products = [&](auto width, auto stages) {
        constexpr int NT = decltype(width)::value, STAGES = decltype(stages)::value;
        const int up_code = kind < 0 ? launch_product<UP_GATED, NT, STAGES>(p, x_rows, x_boxes, up, up_s, stream) : launch_product<UP, NT, STAGES>(p, x_rows, x_boxes, up, up_s, stream);
        if (up_code) return up_code;
        return ragged ? launch_product<DOWN_RAGGED, NT, STAGES>(p, act_rows, act_s_rows, down, down_s, stream)
                      : launch_product<DOWN, NT, STAGES>(p, act_rows, act_s_rows, down, down_s, stream);
    };
    code = width <= 64 ? products(std::integral_constant<int, 64>{}, std::integral_constant<int, 8>{})
         : width <= 128 ? products(std::integral_constant<int, 128>{}, std::integral_constant<int, 6>{})
                        : products(std::integral_constant<int, 256>{}, std::integral_constant<int, 4>{});
    if (code) return code;
    return launch_pdl(experts_combine_kernel, dim3(T), dim3(256), 0, stream, p);
}
