// Attention in its general form for steps that bring few rows per request and key/value head (decoded tokens): the keys are cut
// over warps instead of the rows, and the parts meet inside the kernel.
//
// What bounds it: latency.  A decoded token's keys are some hundred KB over the chip; the time is the chain page table -> key ->
// score -> softmax -> value -> merge.  So
//   * a CTA owns sixteen rows (one mma.sync tile) of one (request, key/value head) and each of its eight warps takes tiles of 16 keys
//     of its own; `splits` CTAs share the keys.  Most contexts are then one tile a warp.
//   * keys and values go from memory straight into the fragments of the products: a thread's 16 bytes of a key hold its operands of
//     two k-steps if the query's lanes are permuted alike, and the 16 bytes of two neighbouring keys' values, interleaved, are
//     its operands of eight n-blocks if the output's columns are numbered alike.  No shared memory, no barrier before the merge.
//   * where the caller says that keys cached before this step were written behind a full dependency (`cached_early`), a warp's first
//     tile is on its way while the kernel in front still runs.  Keys and values bypass L1, where a line could be kept that the kernel
//     in front is still writing its newest row to.
//   * the CTAs that share a row tile are a thread-block cluster and merge through distributed shared memory: no partial results in
//     memory and no second kernel.  (Latent attention leaves its partial results instead: the product behind it merges them.)
// Measured on a B200 against the kernel for many rows and its merge, back to back in a graph, the keys in L2 (microseconds; inside a decode
// step, behind its weights, 7 to 9.5 where this says 5.6 to 8): 32 heads on 8 of 64 lanes,
// window 512 of 2,000 keys: 13.4 -> 5.6 for one request, 18.2 -> 7.5 for 8; all of 2,000 keys, 8 requests: 38.3 -> 14.4; two maps of 64 on
// values of 128: 17.9 -> 7.9; latents of 256 + 32 with 32 heads and the product behind them, 2,000 keys: 20.8 -> 12.1.
#include <type_traits>

#include "attention_rows.cuh"

namespace {

using bf16 = __nv_bfloat16;
constexpr float LOG2E = 1.4426950408889634f;
constexpr int WARPS = 8, THREADS = WARPS * 32, BN = 16, ROWS = 16;

__device__ __forceinline__ void mma_bf16(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ unsigned word_of(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
// the value at the same place in the shared memory of the cluster's CTA `rank`
__device__ __forceinline__ float load_of(const float* mine, unsigned rank) {
    unsigned addr = (unsigned)__cvta_generic_to_shared(mine), there;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(there) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(there) : "memory");
    return v;
}

template <int DVW>
constexpr int PITCH = DVW + 4;  // floats from row to row of a warp's output in shared memory

// KB: blocks of 32 key lanes (dk <= 32 KB); DVW: value lanes a warp keeps; DSPLIT: warps that share a key tile, DVW of its value lanes
// each.  QSMEM: the queries wait in shared memory (long keys), else in registers.
template <int KB, int DVW, int DSPLIT, int MAPS, bool QSMEM, bool LEAVE>
__global__ void __launch_bounds__(THREADS, (KB <= 2 ? 2 : 1))
attention_rows_few_kernel(const RowsArgs<bf16> a, int splits, float* __restrict__ part_o, float* __restrict__ part_ml) {
    constexpr int KG = WARPS / DSPLIT, VG = DVW / 64, PAIRS = ROWS / MAPS, QP = KB * 32 + 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* o_s = reinterpret_cast<float*>(smem_raw);       // [WARPS][ROWS][PITCH]
    float* ml_s = o_s + WARPS * ROWS * PITCH<DVW>;         // [WARPS][ROWS][2]
    float* cta_ml = ml_s + WARPS * ROWS * 2;               // [ROWS][2]
    float* cta_o = cta_ml + ROWS * 2;                      // [ROWS][DVW * DSPLIT] (LEAVE: absent)
    bf16* q_s = reinterpret_cast<bf16*>(cta_o + (LEAVE ? 0 : ROWS * DVW * DSPLIT));  // QSMEM: [ROWS][QP]
    __shared__ float rows_s[WARPS][256];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int kg = warp / DSPLIT, d_lane0 = (warp % DSPLIT) * DVW;
    const int r = blockIdx.z, kvh = blockIdx.y, tile = blockIdx.x / splits, split = blockIdx.x - tile * splits;
    const int group = a.H / a.KV, dk = MAPS * a.d0 + a.d1, dv = a.dv;
    const int q_begin = a.cu_tokens[r], q_len = a.cu_tokens[r + 1] - q_begin, ctx_len = a.ctx_lens[r];
    const int rows_total = q_len * group, row0 = tile * PAIRS;
    // (the same for every CTA of a cluster)
    if ((a.skip_from > 0 && q_len >= a.skip_from) || row0 >= rows_total) return;
    const int rows_here = min(PAIRS, rows_total - row0);
    const int first_pos = ctx_len - q_len;

    // the keys that the tile's rows see, in tiles of 16: those below keep_first that stay visible, then the window's
    const int pos_min = first_pos + row0 / group, pos_max = first_pos + (row0 + rows_here - 1) / group;
    int key_lo = a.window > 0 ? max(0, pos_min - a.window + 1) : 0;
    if (a.chunk > 0) key_lo = max(key_lo, pos_min - pos_min % a.chunk);
    const int kf = a.window > 0 ? a.keep_first : 0;
    int j_first = (key_lo / BN) * BN, kept_tiles = (min(kf, key_lo) + BN - 1) / BN;
    if (kept_tiles * BN >= j_first) { j_first = 0; kept_tiles = 0; }
    const int n_tiles = (pos_max - j_first) / BN + 1 + kept_tiles;
    auto tile_start = [&](int t) { return t < kept_tiles ? t * BN : j_first + (t - kept_tiles) * BN; };
    const int* table = a.page_table + (size_t)r * a.table_width;

    uint4 kr[KB][2], vr[VG][4];
    auto load_keys = [&](int t) {
        const int j0 = tile_start(t);
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
            const int j = j0 + nb * 8 + g;
            const bool valid = j < ctx_len;
            long long off = 0;
            if (valid) off = (long long)table[j / a.page_size] * a.k_page + (long long)kvh * a.k_head + (long long)(j % a.page_size) * a.k_token;
            const bf16* row = a.keys + off + q * 8;
#pragma unroll
            for (int kb = 0; kb < KB; ++kb)
                kr[kb][nb] = valid && kb * 32 + q * 8 < dk ? __ldcg(reinterpret_cast<const uint4*>(row + kb * 32)) : make_uint4(0, 0, 0, 0);
        }
    };
    auto load_values = [&](int t) {
        const int j0 = tile_start(t);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = j0 + (i >> 1) * 8 + 2 * q + (i & 1);
            const bool valid = j < ctx_len;
            long long off = 0;
            if (valid) off = (long long)table[j / a.page_size] * a.v_page + (long long)kvh * a.v_head + (long long)(j % a.page_size) * a.v_token;
            const bf16* row = a.values + off + d_lane0 + g * 8;
#pragma unroll
            for (int vg = 0; vg < VG; ++vg)
                vr[vg][i] = valid && d_lane0 + vg * 64 + g * 8 < dv ? __ldcg(reinterpret_cast<const uint4*>(row + vg * 64)) : make_uint4(0, 0, 0, 0);
        }
    };
    const int t_step = splits * KG;
    int t = kg * splits + split;  // neighbouring tiles on different CTAs
    const bool early = a.cached_early && t < n_tiles && tile_start(t) + BN <= first_pos;  // all of the first tile was cached before this step
    if (early) {
        load_keys(t);
        load_values(t);
    }
    pdl_trigger();
    pdl_wait();  // the queries and the newest cached rows are the work of the kernels in front
    if (!early && t < n_tiles) {
        load_keys(t);
        load_values(t);
    }

    // the query lanes [8 c, 8 c + 8) of a row of the tile
    auto query_chunk = [&](int row, int c) {
        const int lane0 = c * 8, R = row0 + (MAPS == 2 ? (row & 7) : row);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (lane0 >= dk || R >= rows_total) return v;
        const int tok = q_begin + R / group, h = kvh * group + R % group;
        const bf16* src;
        if constexpr (MAPS == 2) {  // rows 0-7 are the pairs' first maps, 8-15 their second: a map's lanes are zeros in the other's rows
            if ((row >= 8) != (lane0 >= a.d0)) return v;
            src = a.q0 + (long long)tok * a.q0_token + (long long)h * a.q0_head + (lane0 < a.d0 ? lane0 : a.q_map + (lane0 - a.d0));
        } else {
            src = lane0 < a.d0 ? a.q0 + (long long)tok * a.q0_token + (long long)h * a.q0_head + lane0
                               : a.q1 + (long long)tok * a.q1_token + (long long)h * a.q1_head + (lane0 - a.d0);
        }
        return *reinterpret_cast<const uint4*>(src);
    };
    uint4 qr[QSMEM ? 1 : KB][2];
    if constexpr (QSMEM) {
        for (int i = tid; i < ROWS * KB * 4; i += THREADS)
            *reinterpret_cast<uint4*>(q_s + (i / (KB * 4)) * QP + (i % (KB * 4)) * 8) = query_chunk(i / (KB * 4), i % (KB * 4));
        __syncthreads();
    } else {
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
#pragma unroll
            for (int e = 0; e < 2; ++e) qr[kb][e] = query_chunk(g + 8 * e, kb * 4 + q);
    }

    int pos[2], lo[2];
    float slope[2], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int R = min(row0 + g + (MAPS == 1 ? 8 * e : 0), rows_total - 1);
        pos[e] = first_pos + R / group;
        lo[e] = a.window > 0 ? max(0, pos[e] - a.window + 1) : 0;
        if (a.chunk > 0) lo[e] = max(lo[e], pos[e] - pos[e] % a.chunk);
        slope[e] = a.slopes ? a.slopes[kvh * group + R % group] * LOG2E : 0.f;
        if (a.sinks && split == 0 && kg == 0) {  // a key of score sinks[h] without a value, counted once a row
            m[e] = a.sinks[kvh * group + R % group] * LOG2E;
            l[e] = q == 0 ? 1.f : 0.f;
        }
    }
    const float scale2 = a.scale * LOG2E, cap2 = a.softcap * LOG2E, cap_in2 = a.softcap > 0.f ? 2.f * LOG2E * a.scale / a.softcap : 0.f;
    const bool biased = a.slopes != nullptr, capped = a.softcap > 0.f;
    float o[VG][8][4];
#pragma unroll
    for (int vg = 0; vg < VG; ++vg)
#pragma unroll
        for (int i = 0; i < 8; ++i) o[vg][i][0] = o[vg][i][1] = o[vg][i][2] = o[vg][i][3] = 0.f;

    for (; t < n_tiles; t += t_step) {
        const int j0 = tile_start(t);
        float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) {
            if (kb > 1 && kb * 32 >= dk) break;
            uint4 q0v, q1v;
            if constexpr (QSMEM) {
                q0v = *reinterpret_cast<const uint4*>(q_s + g * QP + kb * 32 + q * 8);
                q1v = *reinterpret_cast<const uint4*>(q_s + (g + 8) * QP + kb * 32 + q * 8);
            } else {
                q0v = qr[kb][0];
                q1v = qr[kb][1];
            }
#pragma unroll
            for (int nb = 0; nb < 2; ++nb) {
                mma_bf16(s[nb], q0v.x, q1v.x, q0v.y, q1v.y, kr[kb][nb].x, kr[kb][nb].y);
                mma_bf16(s[nb], q0v.z, q1v.z, q0v.w, q1v.w, kr[kb][nb].z, kr[kb][nb].w);
            }
        }
        if (t + t_step < n_tiles) load_keys(t + t_step);
        // scale, cap, bias, mask (scores in units of log 2 from here on)
        float tile_max[2] = {-INFINITY, -INFINITY}, rescale[2], m_use[2];
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int e = c >> 1, j = j0 + nb * 8 + 2 * q + (c & 1);
                // tanh(x) = 1 - 2 / (e^(2x) + 1), as in the kernel for many rows
                float v = capped ? cap2 * (1.f - __fdividef(2.f, exp2f(s[nb][c] * cap_in2) + 1.f)) : s[nb][c] * scale2;
                if (biased) v -= slope[e] * (float)(pos[e] - j);
                v = ((j >= lo[e] || j < kf) && j <= pos[e]) ? v : -INFINITY;
                s[nb][c] = v;
                tile_max[e] = fmaxf(tile_max[e], v);
            }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            tile_max[e] = fmaxf(tile_max[e], __shfl_xor_sync(0xffffffffu, tile_max[e], 1));
            tile_max[e] = fmaxf(tile_max[e], __shfl_xor_sync(0xffffffffu, tile_max[e], 2));
            const float m_new = fmaxf(m[e], tile_max[e]);
            m_use[e] = m_new == -INFINITY ? 0.f : m_new;  // a row that has seen no key yet
            rescale[e] = exp2f(m[e] - m_use[e]);
            m[e] = m_new;
            l[e] *= rescale[e];
        }
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s[nb][c] = exp2f(s[nb][c] - m_use[c >> 1]);
                l[c >> 1] += s[nb][c];
            }
        const unsigned p0 = pack2(s[0][0], s[0][1]), p1 = pack2(s[0][2], s[0][3]), p2 = pack2(s[1][0], s[1][1]), p3 = pack2(s[1][2], s[1][3]);
#pragma unroll
        for (int vg = 0; vg < VG; ++vg)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                o[vg][i][0] *= rescale[0]; o[vg][i][1] *= rescale[0];
                o[vg][i][2] *= rescale[1]; o[vg][i][3] *= rescale[1];
                // lane 8 g + i of keys 2q, 2q + 1 and of keys 2q + 8, 2q + 9
                const unsigned half = i & 1 ? 0x7632 : 0x5410;
                const unsigned b0 = __byte_perm(word_of(vr[vg][0], i >> 1), word_of(vr[vg][1], i >> 1), half);
                const unsigned b1 = __byte_perm(word_of(vr[vg][2], i >> 1), word_of(vr[vg][3], i >> 1), half);
                mma_bf16(o[vg][i], p0, p1, p2, p3, b0, b1);
            }
        if (t + t_step < n_tiles) load_values(t + t_step);
    }

    // the warps' parts meet: n-block i, column n is value lane 8 n + i, so a thread holds lanes 16 q .. 16 q + 15 of its rows
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 1);
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 2);
        const int row = g + 8 * e;
        if (q == 0) {
            ml_s[(warp * ROWS + row) * 2] = m[e];
            ml_s[(warp * ROWS + row) * 2 + 1] = l[e];
        }
        if (l[e] != 0.f) {  // (NaN is not 0: a row whose scores are NaN is a part like any other)
            float* to = o_s + (warp * ROWS + row) * PITCH<DVW>;
#pragma unroll
            for (int vg = 0; vg < VG; ++vg)
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 8; i += 4)
                        *reinterpret_cast<float4*>(to + vg * 64 + q * 16 + c * 8 + i) =
                            make_float4(o[vg][i][2 * e + c], o[vg][i + 1][2 * e + c], o[vg][i + 2][2 * e + c], o[vg][i + 3][2 * e + c]);
        }
    }
    __syncthreads();
    const int quads = dv >> 2;
    for (int i = tid; i < ROWS * quads; i += THREADS) {
        const int row = i / quads, d = (i - row * quads) * 4, pair = MAPS == 2 ? row & 7 : row;
        if (pair >= rows_here) continue;
        const int first = DSPLIT == 1 ? 0 : d / DVW;  // the first of the warps that hold this lane
        float M = -INFINITY, L = 0.f, ws[KG], ls[KG];
#pragma unroll
        for (int k = 0; k < KG; ++k) {
            ws[k] = ml_s[((k * DSPLIT + first) * ROWS + row) * 2];
            ls[k] = ml_s[((k * DSPLIT + first) * ROWS + row) * 2 + 1];
            M = fmaxf(M, ws[k]);
        }
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < KG; ++k) {
            if (ls[k] == 0.f) continue;  // no key for this row: nothing was written
            const float w = ws[k] == -INFINITY ? 0.f : exp2f(ws[k] - M);  // (0: a sink of -inf, or NaN, which stays NaN)
            L = fmaf(w, ls[k], L);
            const float4 v = *reinterpret_cast<const float4*>(o_s + ((k * DSPLIT + first) * ROWS + row) * PITCH<DVW> + (d - first * DVW));
            sum.x = fmaf(w, v.x, sum.x);
            sum.y = fmaf(w, v.y, sum.y);
            sum.z = fmaf(w, v.z, sum.z);
            sum.w = fmaf(w, v.w, sum.w);
        }
        if constexpr (LEAVE) {
            const int R = row0 + row;
            const size_t at = ((size_t)(q_begin + R / group) * a.H + kvh * group + R % group) * splits + split;
            if (L != 0.f) *reinterpret_cast<float4*>(part_o + at * dv + d) = sum;  // no key in this share: the merge does not use it
            if (d == 0) {
                part_ml[at * 2] = M;
                part_ml[at * 2 + 1] = L;
            }
        } else {
            *reinterpret_cast<float4*>(cta_o + row * (DVW * DSPLIT) + d) = sum;
            if (d == 0) {
                cta_ml[row * 2] = M;
                cta_ml[row * 2 + 1] = L;
            }
        }
    }
    if constexpr (!LEAVE) {
        cluster_sync();
        const unsigned rank = cluster_rank();
        for (int pair = warp * splits + (int)rank; pair < rows_here; pair += WARPS * splits) {
            float y[8];
#pragma unroll
            for (int map = 0; map < MAPS; ++map) {
                const int row = pair + 8 * map;
                const float ms = lane < splits ? load_of(cta_ml + row * 2, lane) : -INFINITY;
                const float ls = lane < splits ? load_of(cta_ml + row * 2 + 1, lane) : 0.f;
                const float M = warp_max(ms), w = ms == -INFINITY ? 0.f : exp2f(ms - M), total = warp_sum(w * ls);
                const float inv = total == 0.f ? 0.f : 1.f / total;
                float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
                for (int s = 0; s < splits; ++s) {
                    const float ws = __shfl_sync(0xffffffffu, w, s);
#pragma unroll
                    for (int i = 0; i < 2 * VG * DSPLIT; ++i) {
                        const int d = lane + 32 * i;
                        if (d < dv) acc[i] = fmaf(ws, load_of(cta_o + row * (DVW * DSPLIT) + d, s), acc[i]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] = map == 0 ? acc[i] * inv : y[i] - a.diff_weight * (acc[i] * inv);
            }
            if constexpr (MAPS == 2) {
                float ss = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) ss = fmaf(y[i], y[i], ss);  // lanes beyond dv hold zeros
                const float norm = a.diff_scale / sqrtf(warp_sum(ss) / (float)dv + a.diff_eps);
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] *= norm;
            }
#pragma unroll
            for (int i = 0; i < 2 * VG * DSPLIT; ++i) rows_s[warp][lane + 32 * i] = y[i];
            __syncwarp();
            const int R = row0 + pair, tok = q_begin + R / group, h = kvh * group + R % group;
            const float* gp = a.gate ? a.gate + (long long)tok * a.gate_token + (a.gate_per_head ? (long long)h : (long long)h * dv) : nullptr;
            write_head<bf16>(rows_s[warp], dv, lane, a.turn ? a.turn + (size_t)tok * (dv >> 1) : nullptr, a.turn_neighbours, gp,
                             a.gate_per_head ? 0 : 1, a.out + (long long)tok * a.out_token + (long long)h * a.out_head);
            __syncwarp();
        }
        cluster_sync();  // nobody leaves while its share is being read
    }
}

// a == null: nothing is launched, and `resident` becomes the number of CTAs that the device runs at once in clusters of `splits`
template <int KB, int DVW, int DSPLIT, int MAPS, bool LEAVE>
int launch_few(const RowsArgs<bf16>* a, int requests, int max_query_len, int splits, float* part_o, float* part_ml, cudaStream_t stream, int* resident) {
    constexpr bool QSMEM = KB > 4;
    constexpr size_t smem = ((size_t)WARPS * ROWS * (PITCH<DVW> + 2) + ROWS * 2 + (LEAVE ? 0 : ROWS * DVW * DSPLIT)) * sizeof(float) +
                            (QSMEM ? (size_t)ROWS * (KB * 32 + 32) * 2 : 0);
    auto kernel = attention_rows_few_kernel<KB, DVW, DSPLIT, MAPS, QSMEM, LEAVE>;
    if (smem > 40 * 1024) {  // (with the fixed 8 KB)
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    const long long tiles = a ? ((long long)max_query_len * (a->H / a->KV) + ROWS / MAPS - 1) / (ROWS / MAPS) : 1;
    if (tiles * splits > 0x7fffffffLL || requests > 65535 || (a && a->KV > 65535)) return LLM_ERR_UNSUPPORTED;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * splits), a ? a->KV : 1, requests);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = LEAVE ? 1 : 2;
    if (a) return (int)cudaLaunchKernelEx(&cfg, kernel, *a, splits, part_o, part_ml);
    if (LEAVE) {
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(resident, kernel, THREADS, smem);
        *resident *= device_sms();
        return (int)e;
    }
    const cudaError_t e = cudaOccupancyMaxActiveClusters(resident, kernel, &cfg);
    *resident *= splits;
    return (int)e;
}

int pick_few(int dk, int dv, int maps, bool leave, const RowsArgs<bf16>* a, int requests, int max_query_len, int splits, float* part_o, float* part_ml,
             cudaStream_t stream, int* resident) {
    const bool small = dk <= 64 && dv <= 64, medium = dk <= 128 && dv <= 128;
    if ((dk & 31) || (dv & 63) || !(medium || (maps == 1 && dk <= 320 && dv <= 256))) return LLM_ERR_UNSUPPORTED;
    auto go = [&](auto of) { return of(a, requests, max_query_len, splits, part_o, part_ml, stream, resident); };
    if (leave) {
        if (maps != 1 || splits < 1 || splits > 32) return LLM_ERR_BAD_ARGUMENT;
        if (small) return go(launch_few<2, 64, 1, 1, true>);
        if (medium) return go(launch_few<4, 128, 1, 1, true>);
        return dv <= 128 ? go(launch_few<10, 64, 2, 1, true>) : go(launch_few<10, 128, 2, 1, true>);
    }
    if (splits != 1 && splits != 2 && splits != 4 && splits != 8) return LLM_ERR_BAD_ARGUMENT;  // clusters of any device
    if (maps == 2) return small ? go(launch_few<2, 64, 1, 2, false>) : go(launch_few<4, 128, 1, 2, false>);
    if (small) return go(launch_few<2, 64, 1, 1, false>);
    if (medium) return go(launch_few<4, 128, 1, 1, false>);
    return dv <= 128 ? go(launch_few<10, 64, 2, 1, false>) : go(launch_few<10, 128, 2, 1, false>);
}

}  // namespace

// The shapes that the kernel takes: dk and dv <= 128, or (one map) dk <= 320 with dv <= 256; whole pieces of 32 key lanes and 64 value
// lanes (shorter ones would leave threads without work: they stay with the kernel for many rows).  `splits` CTAs share a tile's keys: a
// cluster (1, 2, 4 or 8) that writes the result, or, with out null, up to 32 that leave part_o [n_tokens * H * splits * dv] and part_ml
// [n_tokens * H * splits * 2]; of a share without keys for a row only part_ml (-inf, 0) is written.  A NaN score makes its row NaN: a share
// is left out by its sum, which is then NaN, and not by its maximum, which passes NaN by.
int launch_rows_few(const RowsArgs<__nv_bfloat16>& a, int requests, int max_query_len, int splits, float* part_o, float* part_ml, cudaStream_t stream) {
    if (a.key_part != 0 || a.stats) return LLM_ERR_UNSUPPORTED;
    if (a.out == nullptr && (!part_o || !part_ml)) return LLM_ERR_BAD_ARGUMENT;
    return pick_few(a.maps * a.d0 + a.d1, a.dv, a.maps, a.out == nullptr, &a, requests, max_query_len, splits, part_o, part_ml, stream, nullptr);
}

// The CTAs of that kernel that the current device runs at once, `splits` of them a cluster (leave: none; partial results are left).  Clusters
// do not fill the device: eight large CTAs need one group of SMs with eight free ones.  Negative: an error.
LLM_EXPORT int llm_rows_few_resident(int dk, int dv, int maps, int leave, int splits) {
    int resident = 0;
    const int code = pick_few(dk, dv, maps, leave != 0, nullptr, 1, 1, splits, nullptr, nullptr, nullptr, &resident);
    return code == 0 ? resident : -code;
}
