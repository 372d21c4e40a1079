// Attention in the CPU path's own order (src/ops/naive.rs:420-466): per (query row, kv head) the scores are left-fold dot
// products over the head dimension, the softmax subtracts the maximum, sums its exponentials in position order and divides,
// and every output element is a left fold over the positions. None of that is reassociated here, so the result equals the
// CPU's bit for bit (the exponential is the C library's, itb_internal.cuh); the parallelism is across positions for the
// scores, across (head, dimension) for the outputs, with the inherently serial chains (head_dim adds per score, n_pos adds
// per softmax sum, n_pos multiply-adds per output) one thread each. Selected by exact=1; exact=0 keeps the split-K kernels,
// which reassociate the sums (tolerance class) and are faster at long contexts.
#pragma once
#include <algorithm>
#include <type_traits>
#include "itb_kernels.cuh"
#include "itb_tile.cuh"

namespace {

constexpr int AX_TP = 32;          // positions per tile of the scores kernel
constexpr int AX_QSTRIDE_PAD = 4;  // q rows in shared memory are head_dim + 4 floats apart: the heads of a group hit different banks
constexpr int AX_KPAD = 8;         // key rows in shared memory are head_dim + 8 elements apart: so do a warp's positions

__device__ __forceinline__ float kv_elem(uint32_t word, int hi, int bf16) {
    const uint16_t h = (uint16_t)(word >> (hi * 16));
    return bf16 ? bf16_bits_to_f32(h) : f16_bits_to_f32(h);
}

// scores[row][head][s] = (sum_i q[i] * k_s[i], i ascending) * scale for s < n_pos(row).
// grid (blocks that share a row's position tiles, n_head_kv, rows); block AX_TP * group threads: thread = (position in tile, head of
// the group). A tile's keys arrive in shared memory as one copy, the next tile's while this one's chains run (read by each chain as it
// goes they cost a memory round trip per 16 dimensions), and a row has only as many blocks as fill the machine: a block per tile of the
// whole context cost 24 us a layer at 32 sequences of 130 positions, most of it blocks that leave at once; now 8.9.
struct AxScores {
    const float* q; const uint16_t* kslab; size_t slab_stride; int rows_per_seq;   // q [rows][n_head][hd]; row r reads the slab of sequence r / rows_per_seq
    const int* n_pos_dev; int n_pos_last, n_q;                                      // per-row positions, or n_pos_last - n_q + 1 + row
    int kv_dim, hd, n_head, n_head_kv; float scale; int bf16;
    float* scores; int s_stride;                                                    // [rows][n_head][s_stride]
};
__global__ void k_attn_scores_exact(AxScores p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int hk = blockIdx.y, r = blockIdx.z, hd = p.hd, group = p.n_head / p.n_head_kv, qst = hd + AX_QSTRIDE_PAD, kst = hd + AX_KPAD;
    float* qs = (float*)smem;                                    // [group][hd + pad]
    uint16_t* ks = (uint16_t*)(qs + group * qst);                // [2][AX_TP][hd + pad]
    pdl_wait(); pdl_trigger();
    const int n_pos = p.n_pos_dev ? p.n_pos_dev[r] : p.n_pos_last - p.n_q + 1 + r;
    const int n_tiles = (n_pos + AX_TP - 1) / AX_TP, cpr = hd / 8;
    if ((int)blockIdx.x >= n_tiles) return;
    const uint16_t* kbase = p.kslab + (size_t)(r / max(1, p.rows_per_seq)) * p.slab_stride + hk * hd;
    auto fetch = [&](int t, int buf) {
        if (t < n_tiles) {
            const int p0 = t * AX_TP, np = min(AX_TP, n_pos - p0);
            for (int i = threadIdx.x; i < np * cpr; i += blockDim.x)
                cp_async16(ks + (buf * AX_TP + i / cpr) * kst + (i % cpr) * 8, kbase + (size_t)(p0 + i / cpr) * p.kv_dim + (i % cpr) * 8, true);
        }
        cp_async_commit();
    };
    fetch(blockIdx.x, 0);
    for (int i = threadIdx.x; i < group * hd; i += blockDim.x)
        qs[(i / hd) * qst + i % hd] = p.q[((size_t)r * p.n_head + hk * group) * hd + i];
    const int g = threadIdx.x % group, sl = threadIdx.x / group;
    const float* qg = qs + g * qst;
    float* out = p.scores + ((size_t)r * p.n_head + hk * group + g) * p.s_stride;
    int buf = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, buf ^= 1) {
        fetch(t + gridDim.x, buf ^ 1);
        cp_async_wait<1>();
        __syncthreads();
        const int s = t * AX_TP + sl;
        if (s < n_pos) {
            const uint16_t* key = ks + (buf * AX_TP + sl) * kst;
            float dot = 0.0f;
#pragma unroll 4
            for (int i = 0; i < hd; i += 8) {
                const uint4 kw = *(const uint4*)(key + i);
                const float4 q0 = *(const float4*)(qg + i), q1 = *(const float4*)(qg + i + 4);
                dot += q0.x * kv_elem(kw.x, 0, p.bf16); dot += q0.y * kv_elem(kw.x, 1, p.bf16);
                dot += q0.z * kv_elem(kw.y, 0, p.bf16); dot += q0.w * kv_elem(kw.y, 1, p.bf16);
                dot += q1.x * kv_elem(kw.z, 0, p.bf16); dot += q1.y * kv_elem(kw.z, 1, p.bf16);
                dot += q1.z * kv_elem(kw.w, 0, p.bf16); dot += q1.w * kv_elem(kw.w, 1, p.bf16);
            }
            out[s] = dot * p.scale;
        }
        __syncthreads();                                         // the buffer is free for the tile after the next
    }
    cp_async_wait<0>();
}
// Blocks that share a row's tiles: two to an SM over all rows and KV heads.
inline int attn_scores_blocks(int n_pos_max, int n_head_kv, int rows, int sms) {
    const long long tiles = (n_pos_max + AX_TP - 1) / AX_TP, share = (2LL * sms + (long long)n_head_kv * rows - 1) / ((long long)n_head_kv * rows);
    return (int)std::max(1LL, std::min(tiles, share));
}

// The serial sum of n floats of shared memory (16-byte aligned, zeros up to a multiple of 32), by every lane of a warp alike. Read 32
// ahead of the adds: the chain of 4-cycle adds is all there is to wait for.
__host__ __device__ constexpr int ax_pad(int n) { return (n + 31) & ~31; }
__device__ __forceinline__ float serial_sum(const float* w, int n) {
    float sum = 0.0f;
    float4 a[8];
    const int n32 = ax_pad(n);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = *(const float4*)(w + 4 * j);
#pragma unroll 1
    for (int s = 0; s < n32; s += 32) {
        const float* nx = w + (s + 32 < n32 ? s + 32 : s);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 e = a[j];
            a[j] = *(const float4*)(nx + 4 * j);
            sum += e.x; sum += e.y; sum += e.z; sum += e.w;
        }
    }
    return sum;
}
// The same sum, of terms >= 0, when there are many: a warp folds 32 segments at once, each from a guess of the sum before it, and again from
// better guesses until every segment began where the one before it ended. Then the whole is the left fold from zero, rounding for
// rounding, however the guesses were made: segment 0 begins at zero, and a segment that begins exactly ends exactly. Each round makes at
// least one more segment begin exactly (its correction is made of exact zeros), so 32 rounds always do; with terms of one sign the sum's grid
// seldom coarsens and 5 to 6 do (12 at most in 10^4 softmax rows of 300 to 6,500 terms; terms of both signs take 17, too many). A
// round is n / 32 adds and two scans: below 640 terms the plain chain is as fast. 6,500 terms: 28,000 cycles of adds -> 8,000; four steps at
// 6,500 positions 11.80 -> 11.37 ms.
constexpr int AX_FOLD_MIN = 640;
__device__ __forceinline__ float fold_sum(const float* w, int n) {
    if (n < AX_FOLD_MIN) return serial_sum(w, n);
    const int lane = threadIdx.x & 31, len = ((n + 31) / 32) | 1, lo = lane * len, cnt = min(len, n - lo);      // odd: the lanes' reads fall on distinct banks
    auto fold = [&](float sum) {
        const float* t = w + min(lo, n - 1);
        int i = 0;
#pragma unroll 1
        for (; i + 8 <= cnt; i += 8) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = t[i + k];
#pragma unroll
            for (int k = 0; k < 8; ++k) sum = __fadd_rn(sum, v[k]);
        }
        for (; i < cnt; ++i) sum = __fadd_rn(sum, t[i]);
        return sum;
    };
    auto before = [&](float v) {                     // the sum of the lanes before this one's, by a tree
        float inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += u; }
        const float ex = __shfl_up_sync(0xffffffffu, inc, 1);
        return lane ? ex : 0.0f;
    };
    float start = before(fold(0.0f)), end = 0.0f;
#pragma unroll 1
    for (int round = 0; round < 32; ++round) {
        end = fold(start);
        float left = __shfl_up_sync(0xffffffffu, end, 1);
        if (lane == 0) left = 0.0f;
        if (__all_sync(0xffffffffu, left == start)) break;
        start = left + before(left - start);
    }
    return __shfl_sync(0xffffffffu, end, 31);
}
// Softmax of one (row, head)'s scores and the weighted sum of the values for 32 dimensions of that head.
// grid (hd / 32, n_head, rows); block 288: everyone on the maximum, exponentials and divisions, warp 0 on the serial sums: of the
// exponentials, then of the weighted values, a lane per dimension. Those two chains (n_pos adds of 4 cycles each) bound the kernel, so
// the chain warp does nothing else: the other eight multiply a tile of AX_VT positions at a time into shared memory, a line per
// dimension, one tile ahead of it and with the values of AX_AHEAD tiles in flight. With the chain warp converting and multiplying
// too, and the sum read as it went, 6,500 positions took 124 us; with both chains serial 46 (31 of them the chains), now 35.
// gate != null: times sigmoid(gate) (src/model/qwen35.rs:1216-1218); out_q != null: the result leaves quantised to Q8_0 (the
// output projection's own quantisation), else as f32 in out.
// READY (the scores already hold the softmax weights: many rows, where the blocks that share a head would each redo the softmax): no
// weights in shared memory, so more blocks to an SM.
// A value line's four 16-byte pieces go to neighbouring lanes (a lane per position touched 32 lines a load); the lines of each eight
// dimensions start 8 floats further on, so that their products fall on distinct banks.
constexpr int AX_VT = 128, AX_VLD = AX_VT + 4, AX_AHEAD = 4, AX_VBUF = 32 * AX_VLD + 32;
constexpr int AX_OUT_SMEM = 226 * 1024;       // room for 49,344 positions beside the two tiles of products
struct AxOut {
    const float* scores; int s_stride;
    const uint16_t* vslab; size_t slab_stride; int rows_per_seq;
    const int* n_pos_dev; int n_pos_last, n_q;
    int kv_dim, hd, n_head, n_head_kv, bf16;
    const float* gate; float* out; int8_t* out_q; float* out_s;
};
template <bool READY>
__global__ void __launch_bounds__(288) k_attn_out_exact(AxOut p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float s_red[9];
    __shared__ float s_sum;
    const int j = blockIdx.x, h = blockIdx.y, r = blockIdx.z, hd = p.hd, group = p.n_head / p.n_head_kv, hk = h / group;
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    pdl_wait(); pdl_trigger();
    const int n_pos = p.n_pos_dev ? p.n_pos_dev[r] : p.n_pos_last - p.n_q + 1 + r;
    float* prod = (float*)smem;                                   // [2][32][AX_VLD]
    float* w = prod + 2 * AX_VBUF;                                // [n_pos] scores -> exponentials -> weights
    const float* sc = p.scores + ((size_t)r * p.n_head + h) * p.s_stride;
    const size_t idx = ((size_t)r * p.n_head + h) * hd + j * 32 + lane;
    const float gate = p.gate && wid == 0 ? p.gate[idx] : 0.0f;
    const int n_tiles = (n_pos + AX_VT - 1) / AX_VT;
    // warps 1..8: 16 positions of each tile, a lane 8 dimensions of two of them
    const int vs = (wid - 1) * 16 + (lane >> 2), q = lane & 3;
    const uint16_t* vbase = p.vslab + (size_t)(r / max(1, p.rows_per_seq)) * p.slab_stride + hk * hd + j * 32 + q * 8;
    uint4 v[AX_AHEAD][2];
    float vw[AX_AHEAD][2];
    auto load = [&](int t, uint4* to, float* wt) {
        if (t < n_tiles) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int s = min(t * AX_VT + vs + 8 * i, n_pos - 1);
                to[i] = *(const uint4*)(vbase + (size_t)s * p.kv_dim);
                if (READY) wt[i] = sc[s];
            }
        }
    };
    auto multiply = [&](int t, const uint4* x, const float* wt) {
        float* d = prod + (t & 1) * AX_VBUF + q * 8 * (AX_VLD + 1) + vs;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int s = t * AX_VT + vs + 8 * i;
            const float ws = s >= n_pos ? 0.0f : READY ? wt[i] : w[s];
            const uint32_t u[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float y = p.bf16 ? kv_elem(u[k >> 1], k & 1, 1) : kv_elem(u[k >> 1], k & 1, 0);
                d[k * AX_VLD + 8 * i] = s < n_pos ? ws * y : -0.0f;      // past the end: a term that changes no sum
            }
        }
    };
    if (wid > 0)
#pragma unroll
        for (int t = 0; t < AX_AHEAD; ++t) load(t, v[t], vw[t]);
    if (!READY) {
        float mx = -INFINITY;
#pragma unroll 4
        for (int s = tid; s < n_pos; s += 288) { const float x = sc[s]; w[s] = x; mx = fmaxf(mx, x); }
        mx = warp_max(mx);
        if (lane == 0) s_red[wid] = mx;
        __syncthreads();
        mx = s_red[0];
        for (int k = 1; k < 9; ++k) mx = fmaxf(mx, s_red[k]);
#pragma unroll 2
        for (int s = tid; s < ax_pad(n_pos); s += 288) w[s] = s < n_pos ? exp_f(w[s] - mx) : 0.0f;
        __syncthreads();
        if (wid == 0) {                                               // the sum in position order
            const float sum = fold_sum(w, n_pos);
            if (lane == 0) s_sum = sum;
        }
        __syncthreads();
        const float sum = s_sum;
#pragma unroll 2
        for (int s = tid; s < n_pos; s += 288) w[s] /= sum;
        __syncthreads();
    }
    float o = 0.0f;
    if (wid > 0 && n_pos > 0) { multiply(0, v[0], vw[0]); load(AX_AHEAD, v[0], vw[0]); }
    __syncthreads();
    for (int t0 = 0; t0 < n_tiles; t0 += AX_AHEAD) {
#pragma unroll
        for (int u = 0; u < AX_AHEAD; ++u) {
            const int t = t0 + u;
            if (t < n_tiles) {
                if (wid > 0) {
                    if (t + 1 < n_tiles) { multiply(t + 1, v[(u + 1) % AX_AHEAD], vw[(u + 1) % AX_AHEAD]); load(t + 1 + AX_AHEAD, v[(u + 1) % AX_AHEAD], vw[(u + 1) % AX_AHEAD]); }
                } else {
                    const float* x = prod + (t & 1) * AX_VBUF + lane * AX_VLD + (lane >> 3) * 8;
                    if (n_pos - t * AX_VT > AX_VT - 32) {
#pragma unroll
                        for (int s = 0; s < AX_VT; s += 4) { const float4 e = *(const float4*)(x + s); o += e.x; o += e.y; o += e.z; o += e.w; }
                    } else
#pragma unroll 1
                        for (int s0 = 0; s0 < n_pos - t * AX_VT; s0 += 32)
#pragma unroll
                            for (int s = s0; s < s0 + 32; s += 4) { const float4 e = *(const float4*)(x + s); o += e.x; o += e.y; o += e.z; o += e.w; }
                }
                __syncthreads();
            }
        }
    }
    if (wid == 0) {
        if (p.gate) o *= sigmoid_f(gate);
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
// the sum in position order by one warp (fold_sum), the division. grid (n_head, rows), block 256; dynamic shared memory n_pos_max floats.
struct AxSoft { float* scores; int s_stride; const int* n_pos_dev; int n_pos_last, n_q, n_head; };
__global__ void __launch_bounds__(256) k_attn_softmax_exact(AxSoft p) {
    pdl_wait();
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
    for (int s = tid; s < ax_pad(n_pos); s += 256) w[s] = s < n_pos ? exp_f(w[s] - mx) : 0.0f;
    __syncthreads();
    if (wid == 0) {
        const float sum = fold_sum(w, n_pos);
        if (lane == 0) s_sum = sum;
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
    pdl_wait(); pdl_trigger();
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
// The weighted values from the softmax weights, 64 dimensions of a head to a block; gate and Q8_0 as in k_attn_out_exact.
// Positions past a row's own take no part in its chain: the tiles that all of a block's rows span go unguarded, the few after them by
// a select. grid (hd / 64, n_head_kv, sequences * token tiles), block 256; s_stride a multiple of 4.
template <int MR, bool BF>
__global__ void __launch_bounds__(256, 2) k_attn_out_tile(AxOut p) {
    constexpr int TL = 16 * MR, WB = TL * AT_ST * 4, STAGE = WB + AT_KT * 64 * 2;
    static_assert(AT_NST * STAGE >= TL * 68 * 4, "the epilogue's tile fits the ring");
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_lim[2];
    const int d0 = blockIdx.x * 64, hk = blockIdx.y, hd = p.hd, group = p.n_head / p.n_head_kv, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    pdl_wait(); pdl_trigger();
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
    const size_t soft = (size_t)ax_pad(n_pos_max) * 4;
    auto run = [&](auto scores, auto out, size_t scores_smem, size_t out_smem) {
        itb_raise_smem(scores, scores_smem);
        itb_raise_smem(out, out_smem);
        itb_raise_smem(k_attn_softmax_exact, 200 * 1024);
        launch(scores, dim3((n_pos_max + 63) / 64, a.n_head_kv, z), dim3(256), scores_smem, a);
        launch(k_attn_softmax_exact, dim3(a.n_head, rows), dim3(256), soft, sm);
        launch(out, dim3(a.hd / 64, a.n_head_kv, z), dim3(256), out_smem, o);
    };
    if (mr == 8 && a.bf16) run(k_attn_scores_tile<8, true>, k_attn_out_tile<8, true>, attn_scores_tile_smem<8>(), attn_out_tile_smem<8>());
    else if (mr == 8) run(k_attn_scores_tile<8, false>, k_attn_out_tile<8, false>, attn_scores_tile_smem<8>(), attn_out_tile_smem<8>());
    else if (a.bf16) run(k_attn_scores_tile<4, true>, k_attn_out_tile<4, true>, attn_scores_tile_smem<4>(), attn_out_tile_smem<4>());
    else run(k_attn_scores_tile<4, false>, k_attn_out_tile<4, false>, attn_scores_tile_smem<4>(), attn_out_tile_smem<4>());
}
inline size_t attn_out_exact_smem(int n_pos_max, bool ready = false) { return (ready ? 0 : (size_t)ax_pad(n_pos_max) * 4) + 2 * AX_VBUF * 4; }
inline size_t attn_scores_exact_smem(int hd, int group) { return (size_t)group * (hd + AX_QSTRIDE_PAD) * 4 + (size_t)2 * AX_TP * (hd + AX_KPAD) * 2; }

}  // namespace
