// Attention in the CPU path's own order (src/ops/naive.rs:420-466): per (query row, kv head) the scores are left-fold dot
// products over the head dimension, the softmax subtracts the maximum, sums its exponentials in position order and divides,
// and every output element is a left fold over the positions. None of that is reassociated here, so the result equals the
// CPU's bit for bit (the exponential is the C library's, itb_internal.cuh); the parallelism is across positions for the
// scores, across (head, dimension) for the outputs, with the inherently serial chains (head_dim adds per score, n_pos adds
// per softmax sum, n_pos multiply-adds per output) one thread each. Selected by exact=1; exact=0 keeps the split-K kernels,
// which reassociate the sums (tolerance class) and are faster at long contexts.
#pragma once
#include <type_traits>
#include "itb_kernels.cuh"
#include "itb_tile.cuh"

namespace {

constexpr int AX_TP = 64;          // positions per block of the scores kernel
constexpr int AX_QSTRIDE_PAD = 4;  // q rows in shared memory are head_dim + 4 floats apart: the heads of a group hit different banks

__device__ __forceinline__ float kv_elem(uint32_t word, int hi, int bf16) {
    const uint16_t h = (uint16_t)(word >> (hi * 16));
    return bf16 ? bf16_bits_to_f32(h) : f16_bits_to_f32(h);
}

// scores[row][head][s] = (sum_i q[i] * k_s[i], i ascending) * scale for s < n_pos(row).
// grid (ceil(n_pos_max / AX_TP), n_head_kv, rows); block AX_TP * group threads: thread = (position in tile, head of the group).
struct AxScores {
    const float* q; const uint16_t* kslab; size_t slab_stride; int rows_per_seq;   // q [rows][n_head][hd]; row r reads the slab of sequence r / rows_per_seq
    const int* n_pos_dev; int n_pos_last, n_q;                                      // per-row positions, or n_pos_last - n_q + 1 + row
    int kv_dim, hd, n_head, n_head_kv; float scale; int bf16;
    float* scores; int s_stride;                                                    // [rows][n_head][s_stride]
};
__global__ void k_attn_scores_exact(AxScores p) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* qs = (float*)smem;                                    // [group][hd + pad]
    const int hk = blockIdx.y, r = blockIdx.z, hd = p.hd, group = p.n_head / p.n_head_kv, qst = hd + AX_QSTRIDE_PAD;
    pdl_trigger(); pdl_wait();
    const int n_pos = p.n_pos_dev ? p.n_pos_dev[r] : p.n_pos_last - p.n_q + 1 + r;
    const int p0 = blockIdx.x * AX_TP;
    if (p0 >= n_pos) return;
    for (int i = threadIdx.x; i < group * hd; i += blockDim.x)
        qs[(i / hd) * qst + i % hd] = p.q[((size_t)r * p.n_head + hk * group) * hd + i];
    __syncthreads();
    const int g = threadIdx.x % group, s = p0 + threadIdx.x / group;
    if (s >= n_pos) return;
    const uint16_t* key = p.kslab + (size_t)(r / max(1, p.rows_per_seq)) * p.slab_stride + (size_t)s * p.kv_dim + hk * hd;
    const float* qg = qs + g * qst;
    float dot = 0.0f;
#pragma unroll 2
    for (int i = 0; i < hd; i += 8) {
        const uint4 kw = *(const uint4*)(key + i);
        const float4 q0 = *(const float4*)(qg + i), q1 = *(const float4*)(qg + i + 4);
        dot += q0.x * kv_elem(kw.x, 0, p.bf16); dot += q0.y * kv_elem(kw.x, 1, p.bf16);
        dot += q0.z * kv_elem(kw.y, 0, p.bf16); dot += q0.w * kv_elem(kw.y, 1, p.bf16);
        dot += q1.x * kv_elem(kw.z, 0, p.bf16); dot += q1.y * kv_elem(kw.z, 1, p.bf16);
        dot += q1.z * kv_elem(kw.w, 0, p.bf16); dot += q1.w * kv_elem(kw.w, 1, p.bf16);
    }
    p.scores[((size_t)r * p.n_head + hk * group + g) * p.s_stride + s] = dot * p.scale;
}

// Softmax of one (row, head)'s scores and the weighted sum of the values for 32 dimensions of that head.
// grid (hd / 32, n_head, rows); block 256: everyone on the softmax, then warp 0 walks the positions (a lane per dimension, one
// multiply-add chain each) over value tiles the other warps stage in shared memory one tile ahead.
// gate != null: times sigmoid(gate) (src/model/qwen35.rs:1216-1218); out_q != null: the result leaves quantised to Q8_0 (the
// output projection's own quantisation), else as f32 in out.
constexpr int AX_VT = 128;         // positions per staged value tile
struct AxOut {
    const float* scores; int s_stride;
    const uint16_t* vslab; size_t slab_stride; int rows_per_seq;
    const int* n_pos_dev; int n_pos_last, n_q;
    int kv_dim, hd, n_head, n_head_kv, bf16;
    const float* gate; float* out; int8_t* out_q; float* out_s;
    int weights_ready;             // the scores buffer already holds the softmax weights (k_attn_softmax_exact ran): skip the softmax here
};
__global__ void __launch_bounds__(256) k_attn_out_exact(AxOut p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float s_red[8];
    __shared__ float s_sum;
    const int j = blockIdx.x, h = blockIdx.y, r = blockIdx.z, hd = p.hd, group = p.n_head / p.n_head_kv, hk = h / group;
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    pdl_trigger(); pdl_wait();
    const int n_pos = p.n_pos_dev ? p.n_pos_dev[r] : p.n_pos_last - p.n_q + 1 + r;
    float* w = (float*)smem;                                      // [n_pos] scores -> exponentials -> weights
    uint16_t* vt = (uint16_t*)(w + ((n_pos + 3) & ~3));           // [2][AX_VT][32]
    const float* sc = p.scores + ((size_t)r * p.n_head + h) * p.s_stride;
    const uint16_t* vbase = p.vslab + (size_t)(r / max(1, p.rows_per_seq)) * p.slab_stride + hk * hd + j * 32;
    auto stage = [&](int tile) {                                  // warps 1..7: tile `tile` of the values into its buffer
        const int s0 = tile * AX_VT, ns = min(AX_VT, n_pos - s0);
        uint16_t* dst = vt + (tile & 1) * AX_VT * 32;
        for (int i = tid - 32; i < ns * 4; i += 224) {            // 4 x 16 bytes per position
            const int s = i >> 2, q = i & 3;
            *(uint4*)(dst + s * 32 + q * 8) = *(const uint4*)(vbase + (size_t)(s0 + s) * p.kv_dim + q * 8);
        }
    };
    if (wid > 0 && n_pos > 0) stage(0);
    if (p.weights_ready) {
        for (int s = tid; s < n_pos; s += 256) w[s] = sc[s];
    } else {
        float mx = -INFINITY;
        for (int s = tid; s < n_pos; s += 256) { const float v = sc[s]; w[s] = v; mx = fmaxf(mx, v); }
        mx = warp_max(mx);
        if (lane == 0) s_red[wid] = mx;
        __syncthreads();
        mx = s_red[0];
        for (int k = 1; k < 8; ++k) mx = fmaxf(mx, s_red[k]);
        for (int s = tid; s < n_pos; s += 256) w[s] = exp_f(w[s] - mx);
        __syncthreads();
        if (tid == 0) {                                               // the sum in position order
            float sum = 0.0f;
            int s = 0;
            for (; s + 4 <= n_pos; s += 4) { const float4 e = *(const float4*)(w + s); sum += e.x; sum += e.y; sum += e.z; sum += e.w; }
            for (; s < n_pos; ++s) sum += w[s];
            s_sum = sum;
        }
        __syncthreads();
        {
            const float sum = s_sum;
            for (int s = tid; s < n_pos; s += 256) w[s] /= sum;
        }
    }
    __syncthreads();
    float o = 0.0f;
    const int n_tiles = (n_pos + AX_VT - 1) / AX_VT;
    for (int t = 0; t < n_tiles; ++t) {
        if (wid > 0) { if (t + 1 < n_tiles) stage(t + 1); }
        else {
            const int s0 = t * AX_VT, ns = min(AX_VT, n_pos - s0);
            const uint16_t* src = vt + (t & 1) * AX_VT * 32 + lane;
            const float* ws = w + s0;
#pragma unroll 8
            for (int s = 0; s < ns; ++s) {
                const uint16_t hb = src[s * 32];
                o += ws[s] * (p.bf16 ? bf16_bits_to_f32(hb) : f16_bits_to_f32(hb));
            }
        }
        __syncthreads();
    }
    if (wid == 0) {
        const size_t idx = ((size_t)r * p.n_head + h) * hd + j * 32 + lane;
        if (p.gate) o *= sigmoid_f(p.gate[idx]);
        if (p.out_q) {
            float dq;
            const int8_t q = warp_quant_q8(o, &dq);
            p.out_q[idx] = q;
            if (lane == 0) p.out_s[idx / 32] = dq;
        } else p.out[idx] = o;
    }
}
// The softmax of one (row, head)'s scores on its own, in place (many-row passes: the eight blocks that share a head's weights in
// k_attn_out_exact would each recompute them, and the library-exact exponential is the expensive part): maximum, exponentials,
// the sum in position order by one thread, the division. grid (n_head, rows), block 256; dynamic shared memory n_pos_max floats.
struct AxSoft { float* scores; int s_stride; const int* n_pos_dev; int n_pos_last, n_q, n_head; };
__global__ void __launch_bounds__(256) k_attn_softmax_exact(AxSoft p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float s_red[8];
    __shared__ float s_sum;
    float* w = (float*)smem;
    const int h = blockIdx.x, r = blockIdx.y, tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    const int n_pos = p.n_pos_dev ? p.n_pos_dev[r] : p.n_pos_last - p.n_q + 1 + r;
    float* sc = p.scores + ((size_t)r * p.n_head + h) * p.s_stride;
    float mx = -INFINITY;
    for (int s = tid; s < n_pos; s += 256) { const float v = sc[s]; w[s] = v; mx = fmaxf(mx, v); }
    mx = warp_max(mx);
    if (lane == 0) s_red[wid] = mx;
    __syncthreads();
    mx = s_red[0];
    for (int k = 1; k < 8; ++k) mx = fmaxf(mx, s_red[k]);
    for (int s = tid; s < n_pos; s += 256) w[s] = exp_f(w[s] - mx);
    __syncthreads();
    if (tid == 0) {
        float sum = 0.0f;
        int s = 0;
        for (; s + 4 <= n_pos; s += 4) { const float4 e = *(const float4*)(w + s); sum += e.x; sum += e.y; sum += e.z; sum += e.w; }
        for (; s < n_pos; ++s) sum += w[s];
        s_sum = sum;
    }
    __syncthreads();
    const float sum = s_sum;
    for (int s = tid; s < n_pos; s += 256) sc[s] = w[s] / sum;
}
// ---- many query rows of a sequence: the same folds as tiled products ----
// A row of the product is a (token, head of the group) pair -- they all read the KV head's one key or value line -- and a thread owns
// MR x 4 chains of a tile of 16 * MR such lines by 64 positions (scores) or 64 dimensions (outputs), walked in the CPU path's order
// with product and sum rounded apart. What bounds them is the f32 pipe: two operations a step, 64 steps a cycle and SM; the tile
// keeps shared-memory reads (12 of 16 bytes for 256 operations at MR = 8) and conversions below that, where one chain per thread
// (above) waits on its own reads. Tiles of 32 k arrive through a 3-stage cp.async ring. Token tiles run from the last (most positions)
// to the first, so that no long one starts late.
// A 5,548-token prompt in passes of 2,048 rows (16 heads of 256 over 2 KV heads), all ten layers: scores 117 -> 47.5 ms, values
// 374 -> 50.0 ms; the operations alone take 35 ms each at 1.9 GHz.
constexpr int AT_KT = 32, AT_ST = AT_KT + 4, AT_NST = 3, AT_KST = 40;       // line strides: floats; 16-bit elements of a key line
struct AtTile { int r0, nt, seq; };            // first row, tokens, sequence
template <int MR>
__device__ __forceinline__ AtTile at_tile(int rows_per_seq, int group, int* s_lim, const int* n_pos_dev, int n_pos_last, int n_q) {
    const int tt = 16 * MR / group, per = (rows_per_seq + tt - 1) / tt, t = per - 1 - (int)blockIdx.z % per;
    AtTile a;
    a.seq = (int)blockIdx.z / per; a.r0 = a.seq * rows_per_seq + t * tt; a.nt = min(tt, rows_per_seq - t * tt);
    if (threadIdx.x == 0) { s_lim[0] = 0; s_lim[1] = 0x7fffffff; }
    __syncthreads();
    if ((int)threadIdx.x < a.nt) {
        const int np = n_pos_dev ? n_pos_dev[a.r0 + threadIdx.x] : n_pos_last - n_q + 1 + a.r0 + (int)threadIdx.x;
        atomicMax(&s_lim[0], np); atomicMin(&s_lim[1], np);
    }
    __syncthreads();
    return a;
}
template <int MR> constexpr size_t attn_scores_tile_smem() { return (size_t)AT_NST * (16 * MR * AT_ST * 4 + 64 * AT_KST * 2); }
template <int MR> constexpr size_t attn_out_tile_smem() { return (size_t)AT_NST * (16 * MR * AT_ST * 4 + AT_KT * 64 * 2); }
// grid (ceil(n_pos_max / 64), n_head_kv, sequences * token tiles), block 256; hd a multiple of 32.
template <int MR, bool BF>
__global__ void __launch_bounds__(256, 2) k_attn_scores_tile(AxScores p) {
    constexpr int TL = 16 * MR, QB = TL * AT_ST * 4, STAGE = QB + 64 * AT_KST * 2;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_lim[2];
    const int hk = blockIdx.y, hd = p.hd, group = p.n_head / p.n_head_kv, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, p0 = blockIdx.x * 64;
    pdl_trigger(); pdl_wait();
    const AtTile t = at_tile<MR>(p.rows_per_seq, group, s_lim, p.n_pos_dev, p.n_pos_last, p.n_q);
    const int mx = s_lim[0], nl = t.nt * group, nk = hd / AT_KT;
    if (p0 >= mx) return;
    const float* qb = p.q + ((size_t)t.r0 * p.n_head + hk * group) * hd;
    auto q_line = [&](int l) { l = min(l, nl - 1); return ((size_t)(l / group) * p.n_head + l % group) * hd; };
    const float* qsrc[MR / 2];
#pragma unroll
    for (int i = 0; i < MR / 2; ++i) qsrc[i] = qb + q_line((tid + 256 * i) >> 3) + (tid & 7) * 4;
    const uint16_t* ksrc = p.kslab + (size_t)t.seq * p.slab_stride + (size_t)min(p0 + (tid >> 2), mx - 1) * p.kv_dim + hk * hd + (tid & 3) * 8;
    auto fetch = [&](int k) {
        if (k < nk) {
            unsigned char* st = smem + (k % AT_NST) * STAGE;
#pragma unroll
            for (int i = 0; i < MR / 2; ++i) cp_async16((float*)st + ((tid + 256 * i) >> 3) * AT_ST + (tid & 7) * 4, qsrc[i] + k * AT_KT, true);
            cp_async16((uint16_t*)(st + QB) + (tid >> 2) * AT_KST + (tid & 3) * 8, ksrc + k * AT_KT, true);
        }
        cp_async_commit();
    };
    for (int k = 0; k < AT_NST - 1; ++k) fetch(k);
    float acc[MR][4];
#pragma unroll
    for (int i = 0; i < MR; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    for (int k = 0; k < nk; ++k) {
        cp_async_wait<AT_NST - 2>();
        __syncthreads();                           // tile k has landed for everyone; everyone is done with tile k - 1
        fetch(k + AT_NST - 1);
        const unsigned char* st = smem + (k % AT_NST) * STAGE;
        const float* qs = (const float*)st + ty * AT_ST;
        const uint16_t* ks = (const uint16_t*)(st + QB) + tx * AT_KST;
#pragma unroll
        for (int kk = 0; kk < AT_KT; kk += 8) {
            uint4 kw[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) kw[j] = *(const uint4*)(ks + 16 * j * AT_KST + kk);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float4 q[MR];
#pragma unroll
                for (int i = 0; i < MR; ++i) q[i] = *(const float4*)(qs + 16 * i * AT_ST + kk + 4 * h);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float kv[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) kv[j] = kv_elem(h == 0 ? (u < 2 ? kw[j].x : kw[j].y) : (u < 2 ? kw[j].z : kw[j].w), u & 1, BF);
#pragma unroll
                    for (int i = 0; i < MR; ++i) {
                        const float qv = u == 0 ? q[i].x : u == 1 ? q[i].y : u == 2 ? q[i].z : q[i].w;
#pragma unroll
                        for (int j = 0; j < 4; ++j) acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(qv, kv[j]));
                    }
                }
            }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < MR; ++i) {
        const int l = ty + 16 * i, r = t.r0 + l / group;
        if (l >= nl) break;
        const int np = p.n_pos_dev ? p.n_pos_dev[r] : p.n_pos_last - p.n_q + 1 + r;
        float* out = p.scores + ((size_t)r * p.n_head + hk * group + l % group) * p.s_stride + p0 + tx;
#pragma unroll
        for (int j = 0; j < 4; ++j) if (p0 + tx + 16 * j < np) out[16 * j] = acc[i][j] * p.scale;
    }
}
// The weighted values from the softmax weights (weights_ready), 64 dimensions of a head to a block; gate and Q8_0 as in k_attn_out_exact.
// Positions past a row's own take no part in its chain: the tiles that all of a block's rows span go unguarded, the few after them by
// a select. grid (hd / 64, n_head_kv, sequences * token tiles), block 256; s_stride a multiple of 4.
template <int MR, bool BF>
__global__ void __launch_bounds__(256, 2) k_attn_out_tile(AxOut p) {
    constexpr int TL = 16 * MR, WB = TL * AT_ST * 4, STAGE = WB + AT_KT * 64 * 2;
    static_assert(AT_NST * STAGE >= TL * 68 * 4, "the epilogue's tile fits the ring");
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_lim[2];
    const int d0 = blockIdx.x * 64, hk = blockIdx.y, hd = p.hd, group = p.n_head / p.n_head_kv, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    pdl_trigger(); pdl_wait();
    const AtTile t = at_tile<MR>(p.rows_per_seq, group, s_lim, p.n_pos_dev, p.n_pos_last, p.n_q);
    const int mx = s_lim[0], full = s_lim[1] / AT_KT, nl = t.nt * group, nk = (mx + AT_KT - 1) / AT_KT;
    const float* wb = p.scores + ((size_t)t.r0 * p.n_head + hk * group) * p.s_stride;
    const float* wsrc[MR / 2];
#pragma unroll
    for (int i = 0; i < MR / 2; ++i) {
        const int l = min((tid + 256 * i) >> 3, nl - 1);
        wsrc[i] = wb + ((size_t)(l / group) * p.n_head + l % group) * p.s_stride + (tid & 7) * 4;
    }
    const uint16_t* vsrc = p.vslab + (size_t)t.seq * p.slab_stride + hk * hd + d0 + (tid & 7) * 8;
    auto fetch = [&](int k) {
        if (k < nk) {
            unsigned char* st = smem + (k % AT_NST) * STAGE;
            const bool in_w = k * AT_KT + (tid & 7) * 4 < mx, in_v = k * AT_KT + (tid >> 3) < mx;
#pragma unroll
            for (int i = 0; i < MR / 2; ++i) cp_async16((float*)st + ((tid + 256 * i) >> 3) * AT_ST + (tid & 7) * 4, wsrc[i] + (in_w ? k * AT_KT : 0), in_w);
            cp_async16((uint16_t*)(st + WB) + (tid >> 3) * 64 + (tid & 7) * 8, vsrc + (size_t)(in_v ? k * AT_KT + (tid >> 3) : 0) * p.kv_dim, in_v);
        }
        cp_async_commit();
    };
    for (int k = 0; k < AT_NST - 1; ++k) fetch(k);
    float acc[MR][4];
    int np[MR];
#pragma unroll
    for (int i = 0; i < MR; ++i) {
        const int r = t.r0 + min(ty + 16 * i, nl - 1) / group;
        np[i] = p.n_pos_dev ? p.n_pos_dev[r] : p.n_pos_last - p.n_q + 1 + r;
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    }
    auto tile = [&](int k, auto guarded) {
        const unsigned char* st = smem + (k % AT_NST) * STAGE;
        const float* ws = (const float*)st + ty * AT_ST;
        const uint16_t* vs = (const uint16_t*)(st + WB) + tx * 4;
#pragma unroll
        for (int kk = 0; kk < AT_KT; kk += 4) {
            float4 w[MR];
#pragma unroll
            for (int i = 0; i < MR; ++i) w[i] = *(const float4*)(ws + 16 * i * AT_ST + kk);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint2 vw = *(const uint2*)(vs + (kk + u) * 64);
                const float v[4] = {kv_elem(vw.x, 0, BF), kv_elem(vw.x, 1, BF), kv_elem(vw.y, 0, BF), kv_elem(vw.y, 1, BF)};
#pragma unroll
                for (int i = 0; i < MR; ++i) {
                    const float wv = u == 0 ? w[i].x : u == 1 ? w[i].y : u == 2 ? w[i].z : w[i].w;
                    const bool in = !decltype(guarded)::value || k * AT_KT + kk + u < np[i];
#pragma unroll
                    for (int j = 0; j < 4; ++j) { const float n = __fadd_rn(acc[i][j], __fmul_rn(wv, v[j])); acc[i][j] = in ? n : acc[i][j]; }
                }
            }
        }
    };
    for (int k = 0; k < nk; ++k) {
        cp_async_wait<AT_NST - 2>();
        __syncthreads();
        fetch(k + AT_NST - 1);
        if (k < full) tile(k, std::false_type{}); else tile(k, std::true_type{});
    }
    cp_async_wait<0>();
    __syncthreads();
    float* ot = (float*)smem;                      // [TL][68]
#pragma unroll
    for (int i = 0; i < MR; ++i) *(float4*)(ot + (ty + 16 * i) * 68 + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();
    const int wid = tid >> 5, lane = tid & 31;
    for (int u = wid; u < 2 * nl; u += 8) {        // 32 dimensions of a line
        const int l = u >> 1, r = t.r0 + l / group;
        const size_t idx = ((size_t)r * p.n_head + hk * group + l % group) * hd + d0 + (u & 1) * 32 + lane;
        float o = ot[l * 68 + (u & 1) * 32 + lane];
        if (p.gate) o *= sigmoid_f(p.gate[idx]);
        if (p.out_q) {
            float dq;
            const int8_t q = warp_quant_q8(o, &dq);
            p.out_q[idx] = q;
            if (lane == 0) p.out_s[idx / 32] = dq;
        } else p.out[idx] = o;
    }
}
// Lines (16 * MR) of a tile, 0: a chain per thread (k_attn_scores_exact / k_attn_out_exact). A tile pays from about half of its
// smallest form's lines on; the large one where its blocks still give every SM two.
inline int attn_tile_rows(int rows_per_seq, int n_seq, int hd, int n_head, int n_head_kv, int sms) {
    const int group = n_head / n_head_kv;
    if (hd % 64 || rows_per_seq * group < 32) return 0;
    const long long blocks = (long long)(hd / 64) * n_head_kv * n_seq * ((rows_per_seq + 128 / group - 1) / (128 / group));
    return blocks >= 2 * sms ? 8 : 4;
}
// Scores, softmax and weighted values of a pass in that form. launch(kernel, grid, block, shared memory, argument).
template <class L>
static void attn_exact_tiles(const AxScores& a, const AxSoft& sm, const AxOut& o, int mr, int n_seq, int rows, int n_pos_max, L&& launch) {
    const int group = a.n_head / a.n_head_kv, tt = 16 * mr / group, z = n_seq * ((a.rows_per_seq + tt - 1) / tt);
    const size_t soft = (size_t)((n_pos_max + 3) & ~3) * 4;
    auto run = [&](auto scores, auto out, size_t scores_smem, size_t out_smem) {
        cudaFuncSetAttribute(scores, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scores_smem);
        cudaFuncSetAttribute(out, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem);
        cudaFuncSetAttribute(k_attn_softmax_exact, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        launch(scores, dim3((n_pos_max + 63) / 64, a.n_head_kv, z), dim3(256), scores_smem, a);
        launch(k_attn_softmax_exact, dim3(a.n_head, rows), dim3(256), soft, sm);
        launch(out, dim3(a.hd / 64, a.n_head_kv, z), dim3(256), out_smem, o);
    };
    if (mr == 8 && a.bf16) run(k_attn_scores_tile<8, true>, k_attn_out_tile<8, true>, attn_scores_tile_smem<8>(), attn_out_tile_smem<8>());
    else if (mr == 8) run(k_attn_scores_tile<8, false>, k_attn_out_tile<8, false>, attn_scores_tile_smem<8>(), attn_out_tile_smem<8>());
    else if (a.bf16) run(k_attn_scores_tile<4, true>, k_attn_out_tile<4, true>, attn_scores_tile_smem<4>(), attn_out_tile_smem<4>());
    else run(k_attn_scores_tile<4, false>, k_attn_out_tile<4, false>, attn_scores_tile_smem<4>(), attn_out_tile_smem<4>());
}
inline size_t attn_out_exact_smem(int n_pos_max) { return (size_t)((n_pos_max + 3) & ~3) * 4 + 2 * AX_VT * 32 * 2; }
inline size_t attn_scores_exact_smem(int hd, int group) { return (size_t)group * (hd + AX_QSTRIDE_PAD) * 4; }

}  // namespace
