// Kernels of the engine's multi-row path: several tokens at once, either one token of each of many sequences
// (batched decode) or many consecutive tokens of one sequence (prefill). Rows are token-major; row i belongs to
// sequence i / n_tok and is its token number i % n_tok of this pass. Matmuls run on the int8 MMA kernels
// (itb_mma.cuh, every weight row read once per 32 rows); the kernels here are the rest of a layer. All keep the
// CPU path's arithmetic order, so a prefill is bit-identical to feeding the tokens one at a time, which the
// reference asserts of its own backends (tests/qwen35.rs:94-139 there).
#pragma once
#include <type_traits>
#include "itb_kernels.cuh"
#include "itb_tile.cuh"

namespace {

// Sums of N values (4 or 8) over a warp's lanes, each with the additions of warp_sum: at every step a lane adds its partner's value to its
// own, but hands half of the values over and keeps the other half while there is more than one. The lane gets the sum of value warp_sums_of().
template <int N>
__device__ __forceinline__ int warp_sums_of(int lane) { return N == 8 ? (lane >> 2) & 7 : (lane >> 3) & 3; }
template <int N>
__device__ __forceinline__ float warp_sums(const float (&a)[N], int lane) {
    float v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = a[i];
    int o = 16;
#pragma unroll
    for (int n = N / 2; n >= 1; n >>= 1, o >>= 1) {
        const bool hi = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float give = hi ? v[i] : v[i + n], mine = hi ? v[i + n] : v[i];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}
// F32 matrix against many rows (router logits, alpha/beta, shared-expert gate), tree mode. A block takes 8 * MR weight rows (MR per
// warp, held in registers) and tok_blk token rows, F32_TOK at a time through shared memory, the next ones on their way meanwhile.
// Per lane the products are summed in the order of f32_rows<false> (the one-token path), then the same shuffle tree, so a row gets
// the bits it gets alone.
// What bounds it: the 16-byte reads of the token rows from shared memory, one for four products of each weight row that a warp holds (2,048
// rows, 256 outputs, 2,048 k: 60 us with two rows a warp, as much as the products and sums take, 120 with one), and, with a block for
// every F32_TOK rows, the weights, 1.07 GB from L2. That size takes 117 us; a block per token row and 32 outputs (k_matmul_f32) 307.
// grid (ceil(n_out / (8 MR)), ceil(n_rows / tok_blk)), block 256, dynamic smem (tok_blk > F32_TOK ? 2 : 1) * F32_TOK * n_in floats; n_in = 128 * NV.
constexpr int F32_TOK = 4;
template <int NV, int MR>
__global__ void __launch_bounds__(256) k_matmul_f32_rows(DevF32 w, const float* __restrict__ x, int n_rows, float* out, int tok_blk) {
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    float* xs = (float*)smem;
    constexpr int n = 128 * NV, N = F32_TOK * MR, PER = F32_TOK * n / 4 / 256;   // PER: float4 per thread of the token tile
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = (blockIdx.x * 8 + wid) * MR, t_lo = blockIdx.y * tok_blk, t_hi = min(t_lo + tok_blk, n_rows), ng = (t_hi - t_lo + F32_TOK - 1) / F32_TOK;
    auto fetch = [&](int g) {
        if (g < ng) {
            float* to = xs + (size_t)(g & 1) * F32_TOK * n;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int e = threadIdx.x + 256 * i, t = min(t_lo + g * F32_TOK + e / (n / 4), n_rows - 1);
                cp_async16(to + e * 4, x + (size_t)t * n + (e % (n / 4)) * 4, true);
            }
        }
        cp_async_commit();
    };
    fetch(0);
    float4 wv[MR][NV];
#pragma unroll
    for (int r = 0; r < MR; ++r) {
        const float* wr = w.w + (size_t)min(row0 + r, w.n_out - 1) * n;
#pragma unroll
        for (int j = 0; j < NV; ++j) wv[r][j] = __ldg((const float4*)(wr + lane * 4 + 128 * j));
    }
    for (int g = 0; g < ng; ++g) {
        fetch(g + 1);
        cp_async_wait<1>();
        __syncthreads();
        const float* xr = xs + (size_t)(g & 1) * F32_TOK * n + lane * 4;
        float s[N];
#pragma unroll
        for (int i = 0; i < N; ++i) s[i] = 0.0f;
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int t = 0; t < F32_TOK; ++t) {
                const float4 v = *(const float4*)(xr + t * n + 128 * j);
#pragma unroll
                for (int r = 0; r < MR; ++r) s[t * MR + r] += wv[r][j].x * v.x + wv[r][j].y * v.y + wv[r][j].z * v.z + wv[r][j].w * v.w;
            }
        const float sum = warp_sums<N>(s, lane);
        const int i = warp_sums_of<N>(lane), t = t_lo + g * F32_TOK + i / MR, row = row0 + i % MR;
        if ((lane & (32 / N - 1)) == 0 && t < t_hi && row < w.n_out) out[(size_t)t * w.n_out + row] = sum;
        __syncthreads();                           // everyone is done with these rows before the ones after the next take their place
    }
}
inline bool f32_tree_ok(int n_in) { return n_in % 512 == 0 && n_in <= 4096; }
// Two weight rows to a warp where their registers allow and the blocks still give every SM two; then as many tokens to a block as
// leave it two.
static void f32_tree(cudaStream_t st, int sms, const DevF32& w, const float* x, int n_rows, float* out) {
    auto blocks = [&](int mr, int tok) { return (long long)((w.n_out + 8 * mr - 1) / (8 * mr)) * ((n_rows + tok - 1) / tok); };
    const int mr = w.n_in <= 2048 && blocks(2, F32_TOK) >= 2 * sms ? 2 : 1;
    int tok = F32_TOK;
    while (tok < 32 && blocks(mr, 2 * tok) >= 2 * sms) tok *= 2;
    const dim3 g((w.n_out + 8 * mr - 1) / (8 * mr), (n_rows + tok - 1) / tok);
    const size_t sm = (size_t)(tok > F32_TOK ? 2 : 1) * F32_TOK * w.n_in * 4;
    auto run = [&](auto k) { itb_raise_smem(k, sm); itb_chain(k, g, 256, sm, st, w, x, n_rows, out, tok); };
    switch (w.n_in / 128) {
#define F32_CASE(NV) case NV: if (mr == 2) run(k_matmul_f32_rows<NV, 2>); else run(k_matmul_f32_rows<NV, 1>); break;
#define F32_CASE1(NV) case NV: run(k_matmul_f32_rows<NV, 1>); break;
        F32_CASE(4) F32_CASE(8) F32_CASE(12) F32_CASE(16) F32_CASE1(20) F32_CASE1(24) F32_CASE1(28) F32_CASE1(32)
#undef F32_CASE
#undef F32_CASE1
    }
}

// F32 matrix against many rows in the CPU path's own order (src/ops/naive.rs:49-56: a left fold over k of w[o][k] * x[r][k],
// product and sum rounded separately). With many rows there is a chain per (row, output), so no chain needs to be spread over
// lanes: a thread owns MR x MO of them and walks k in order -- a tiled SGEMM whose k loop is never reassociated or fused. Tiles of
// KT k arrive through an NST-stage cp.async ring, lines KT + 4 floats apart; a thread's outputs and rows are TO / MO and TR / MR
// apart, so the 16-byte reads of a warp fall on distinct banks. FUSED (tolerance class): the same walk with one fused multiply-add
// per step. Two matrices over the same rows in one launch (blockIdx.z picks; w1.w null: one): the router and the shared expert's
// gate, or alpha and beta -- each alone is a handful of blocks walking a 2,048-long chain.
// grid (ceil(n_out / TO), ceil(n_rows / TR), 1 or 2), block (TO / MO) * (TR / MR); n_in a multiple of KT.
// What bounds the shapes: 8 x 8, a chain to a thread, the chain itself: 4 cycles a step, and with up to four such blocks an SM a
// scheduler has the slots for its warps' reads, products and sums between them. The others shared memory: a warp's 16-byte read takes four
// of its cycles, the same data for several lanes or not, so four k of MO x MR chains are 4 (MO + MR) of those against MO MR operations
// (fused; twice that unfused) of a scheduler's; and the barrier of a tile, so tiles are 64 k or more. The next four k are read under this four's operations.
template <bool FUSED, int TO, int TR, int MO, int MR, int KT, int NST>
__global__ void __launch_bounds__((TO / MO) * (TR / MR)) k_sgemm_chain(DevF32 w0, const float* __restrict__ x, int n_rows, float* out0, DevF32 w1 = DevF32{}, float* out1 = nullptr) {
    constexpr int ST = KT + 4, NX = TO / MO, NY = TR / MR, NT = NX * NY, PIECES = (TO + TR) * (KT / 4) / NT, W_PIECES = TO * (KT / 4) / NT;      // a thread per MO x MR outputs
    static_assert((TO + TR) * (KT / 4) % NT == 0 && TO * (KT / 4) % NT == 0, "whole pieces");
    extern __shared__ __align__(16) unsigned char smem[];
    float* ring = (float*)smem;                    // [stage][TO weight lines | TR activation lines][ST]
    const DevF32 w = blockIdx.z ? w1 : w0;
    float* out = blockIdx.z ? out1 : out0;
    const int o0 = blockIdx.x * TO, r0 = blockIdx.y * TR, n = w.n_in, nk = n / KT;
    if (o0 >= w.n_out) { pdl_wait(); return; }
    const int tx = threadIdx.x % NX, ty = threadIdx.x / NX;
    const float* src[PIECES];
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        const int c = threadIdx.x + NT * i, line = c / (KT / 4), k4 = (c % (KT / 4)) * 4;
        src[i] = (line < TO ? w.w + (size_t)min(o0 + line, w.n_out - 1) * n : x + (size_t)min(r0 + line - TO, n_rows - 1) * n) + k4;
    }
    auto fetch = [&](int t, int from, int to) {
        float* st = ring + (size_t)(t % NST) * (TO + TR) * ST;
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const int c = threadIdx.x + NT * i;
            if (i >= from && i < to) cp_async16(st + (c / (KT / 4)) * ST + (c % (KT / 4)) * 4, src[i] + (size_t)t * KT, true);
        }
    };
    // the weights of the first stages are requested before the rows they will meet are there
    for (int t = 0; t < NST - 1; ++t) if (t < nk) fetch(t, 0, W_PIECES);
    pdl_wait();
    for (int t = 0; t < NST - 1; ++t) { if (t < nk) fetch(t, W_PIECES, PIECES); cp_async_commit(); }
    // ML of the thread's MO outputs exist: where a matrix has no more than one per thread (the shared expert's gate), the others are not walked
    auto walk = [&](auto live) {
        constexpr int ML = decltype(live)::value;
        float acc[MR][ML];
#pragma unroll
        for (int i = 0; i < MR; ++i)
#pragma unroll
            for (int j = 0; j < ML; ++j) acc[i][j] = 0.0f;
        for (int t = 0; t < nk; ++t) {
            cp_async_wait<NST - 2>();
            __syncthreads();                       // tile t has landed for everyone; everyone is done with tile t - 1
            if (t + NST - 1 < nk) fetch(t + NST - 1, 0, PIECES);      // into the slot tile t - 1 used
            cp_async_commit();
            const float* st = ring + (size_t)(t % NST) * (TO + TR) * ST;
            const float* wr = st + tx * ST; const float* xr = st + (TO + ty) * ST;
            float4 a[2][ML], c[2][MR];
            auto read = [&](int kk, float4 (&a)[ML], float4 (&c)[MR]) {
#pragma unroll
                for (int j = 0; j < ML; ++j) a[j] = *(const float4*)(wr + j * NX * ST + kk);
#pragma unroll
                for (int i = 0; i < MR; ++i) c[i] = *(const float4*)(xr + i * NY * ST + kk);
            };
            read(0, a[0], c[0]);
#pragma unroll(ML * MR <= 8 ? KT / 4 : 4)
            for (int kk = 0; kk < KT; kk += 4) {
                const int u = (kk >> 2) & 1;
                if (kk + 4 < KT) read(kk + 4, a[u ^ 1], c[u ^ 1]);
                auto step = [&](auto get) {
#pragma unroll
                    for (int i = 0; i < MR; ++i)
#pragma unroll
                        for (int j = 0; j < ML; ++j) acc[i][j] = FUSED ? fmaf(get(a[u][j]), get(c[u][i]), acc[i][j]) : __fadd_rn(acc[i][j], __fmul_rn(get(a[u][j]), get(c[u][i])));
                };
                step([](const float4& v) { return v.x; }); step([](const float4& v) { return v.y; });
                step([](const float4& v) { return v.z; }); step([](const float4& v) { return v.w; });
            }
        }
        cp_async_wait<0>();
#pragma unroll
        for (int i = 0; i < MR; ++i)
#pragma unroll
            for (int j = 0; j < ML; ++j)
                if (r0 + ty + i * NY < n_rows && o0 + tx + j * NX < w.n_out) out[(size_t)(r0 + ty + i * NY) * w.n_out + o0 + tx + j * NX] = acc[i][j];
    };
    if (MO > 1 && w.n_out - o0 <= NX) walk(std::integral_constant<int, 1>{}); else walk(std::integral_constant<int, MO>{});
}
constexpr int SG_KT = 64;
inline bool sgemm_chain_ok(int n_in) { return n_in % SG_KT == 0; }
template <bool FUSED, int TO, int TR, int MO, int MR, int KT, int NST>
static void sgemm_tiles(cudaStream_t st, int n_out, int nz, const DevF32& wa, const float* x, int n_rows, float* oa, const DevF32& wb, float* ob) {
    constexpr size_t smem = (size_t)NST * (TO + TR) * (KT + 4) * 4;
    itb_raise_smem(k_sgemm_chain<FUSED, TO, TR, MO, MR, KT, NST>, smem);
    itb_chain(k_sgemm_chain<FUSED, TO, TR, MO, MR, KT, NST>, dim3((n_out + TO - 1) / TO, (n_rows + TR - 1) / TR, nz), (TO / MO) * (TR / MR), smem, st, wa, x, n_rows, oa, wb, ob);
}
// One matrix, or two over the same rows. 8 x 8, a chain to a thread, is fastest as long as an SM has no more than four such blocks, but it
// reads every line once per 8 of the others; beyond that, of the tiles that read less the largest of which every SM still gets three or four.
// Measured (us, 257 outputs, 2,048 k; in parentheses the next best): 32 rows 8 x 8 11.4 (16 x 16 18.5); 256 rows 16 x 16 with 2 x 2 chains to a
// thread 30.1 (1 x 2 33.4); 512 rows the same 38.0 (43.0); 1,024 rows 16 x 32 with 2 x 2 59.9 (16 x 16 69.3, 32 x 32 90); 2,048 rows 32 x 32
// with 2 x 4 99.4 (16 x 32 116, 64 x 64 with 4 x 4 111; 32 x 32 with 2 x 2 and tiles of 32 k 145). Fused, 512 rows 16 x 32 with 2 x 4 42.6 (32 x 64
// 49.4), 2,048 rows 32 x 64 with 4 x 4 79.7 (64 x 64 with 4 x 4 88.9; tiles of 32 k 116).
template <bool FUSED>
static void sgemm_chain(cudaStream_t st, int sms, const DevF32& wa, const float* x, int n_rows, float* oa, const DevF32& wb = DevF32{}, float* ob = nullptr) {
    const int n_out = std::max(wa.n_out, wb.w ? wb.n_out : 0), nz = wb.w ? 2 : 1, n_all = wa.n_out + (wb.w ? wb.n_out : 0);
    auto blocks = [&](int to, int tr) { return (long long)((n_all + to - 1) / to) * ((n_rows + tr - 1) / tr); };
    if (blocks(8, 8) <= 4 * sms && wa.n_in % 128 == 0) sgemm_tiles<FUSED, 8, 8, 1, 1, 128, 5>(st, n_out, nz, wa, x, n_rows, oa, wb, ob);
    else if (blocks(8, 8) <= 4 * sms) sgemm_tiles<FUSED, 8, 8, 1, 1, 64, 8>(st, n_out, nz, wa, x, n_rows, oa, wb, ob);
    else if (FUSED && 2 * blocks(32, 64) >= 3 * sms) sgemm_tiles<FUSED, 32, 64, 4, 4, 64, 3>(st, n_out, nz, wa, x, n_rows, oa, wb, ob);
    else if (FUSED) sgemm_tiles<FUSED, 16, 32, 2, 4, 64, 4>(st, n_out, nz, wa, x, n_rows, oa, wb, ob);
    else if (2 * blocks(32, 32) >= 7 * sms) sgemm_tiles<FUSED, 32, 32, 2, 4, 64, 3>(st, n_out, nz, wa, x, n_rows, oa, wb, ob);
    else if (2 * blocks(16, 32) >= 7 * sms) sgemm_tiles<FUSED, 16, 32, 2, 2, 64, 4>(st, n_out, nz, wa, x, n_rows, oa, wb, ob);
    else sgemm_tiles<FUSED, 16, 16, 2, 2, 64, 6>(st, n_out, nz, wa, x, n_rows, oa, wb, ob);
}

// A dense Q8_0 matrix against n_rows >= 1 quantised rows: out[row][n_out] = or += (mode). tc: the tensor-core forms the context's
// options name may be used (eager many-token passes). False: a device error.
static bool dense_q8(itb_ctx* c, cudaStream_t st, const DevQ8& w, const QRows& x, int n_rows, float* out, size_t stride, int mode, bool tc) {
    const int k = w.n_in;
    // many rows, dense=f16tc (tolerance class): both operands dequantised to f16, one tcgen05 GEMM with f32 accumulators
    if (tc && c->f16tc && n_rows >= 64 && itb_tc_f16_shape_ok(w)) return itb_tc_f16_gemm(c, st, w, x, n_rows, out, stride, mode);
    // many rows, dense=q8tc: exact integer dots of 256 x 64 or 128 x 64 (row, token) pairs on tcgen05, scaled and summed in the CPU's order
    if (tc && c->q8tc && n_rows >= 64 && itb_tc_q8_shape_ok(w)) return itb_tc_q8_gemm(c, st, w, x, n_rows, out, stride, mode);
    for (const void* f : {(const void*)k_gemm_q8<1>, (const void*)k_gemm_q8<4>}) itb_raise_smem(f, 200 * 1024);
    const bool skinny = n_rows <= 32;
    if (k % 256 == 0) {
        Q8Multi p{};
        p.n = 1; p.w[0] = w; p.out[0] = out; p.stride[0] = stride;
        tile_q8(st, c->sm_count, p, x.q, x.s, n_rows, mode);
    }
    else if (skinny) itb_chain(k_gemm_q8<1>, dim3((w.n_out + 63) / 64, 1), 512, gemm_smem(k), st, w, x.q, x.s, n_rows, out, stride, mode);
    else itb_chain(k_gemm_q8<4>, dim3((w.n_out + MMA_ROWS - 1) / MMA_ROWS, (n_rows + MMA_TOK - 1) / MMA_TOK), 256, gemm_smem(k), st, w, x.q, x.s, n_rows, out, stride, mode);
    return true;
}

// RMSNorm + Q8_0 quantisation of each row (src/ops/naive.rs:139-152, :653-675): normalised f32 row, int8 quants,
// scales; xh (optional): the quants as f16 for the expert kernels (exp_pos order). grid = rows, block 256.
__global__ void __launch_bounds__(256) k_norm_quant(const float* x, const float* w, int n, float eps, float* xn_out, int8_t* xq, float* xs, __half* xh = nullptr) {
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    double* red = (double*)smem;
    float* xn = (float*)(red + 32);
    const size_t r = blockIdx.x;
    if (block_rms_norm(x + r * n, w, n, eps, xn, red, xq + r * n, xs + r * (n / 32), xh ? xh + r * n : nullptr)) {   // quantised in the same pass
        if (xn_out) for (int i = threadIdx.x; i < n / 4; i += blockDim.x) ((float4*)(xn_out + r * n))[i] = ((const float4*)xn)[i];
        return;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int b = wid; b < n / 32; b += nw) {
        float v = xn[b * 32 + lane], d;
        const int8_t q = warp_quant_q8(v, &d);
        xq[r * n + b * 32 + lane] = q;
        if (xh) xh[r * n + b * 32 + exp_pos(lane)] = __int2half_rn((int)q);
        if (lane == 0) xs[r * (n / 32) + b] = d;
        if (xn_out) xn_out[r * n + b * 32 + lane] = v;
    }
}

// Depthwise causal conv (src/ops/naive.rs:275-315), every (row, channel) on its own thread: the window of row t is
// the sequence's earlier rows of this pass, or the saved state where it reaches before the pass. Writes the
// PRE-activation sum to `out` (the input rows stay intact for the neighbours). grid (ceil(nc/128), rows).
__global__ void k_conv_rows(const float* state, size_t state_stride, const float* x, float* out, int n_tok, int nc, const float* w, int kernel) {
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const size_t r = blockIdx.y;
    const int s = (int)(r / n_tok), t = (int)(r % n_tok), keep = kernel - 1;
    const float* st = state + (size_t)s * state_stride + (size_t)c * keep;
    float sum = 0.0f;
    for (int k = 0; k < keep; ++k) {
        const int idx = t - keep + k;
        const float past = idx >= 0 ? x[((size_t)s * n_tok + idx) * nc + c] : st[keep + idx];
        sum += past * w[(size_t)c * kernel + k];
    }
    sum += x[r * nc + c] * w[(size_t)c * kernel + keep];
    out[r * nc + c] = sum;
}
// The same for a kernel of 4 taps, CONV_T consecutive tokens of one sequence per thread: the three earlier inputs slide along
// in registers and the channel's taps are read once, so an output costs one load and one store instead of eight loads. The sums
// are the same expressions in the same order. grid (ceil(nc/128), n_seq * ceil(n_tok / CONV_T)).
constexpr int CONV_T = 8;
__global__ void __launch_bounds__(128) k_conv_rows4(const float* state, size_t state_stride, const float* __restrict__ x, float* __restrict__ out, int n_tok, int nc, const float* __restrict__ w) {
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const int chunks = (n_tok + CONV_T - 1) / CONV_T, s = blockIdx.y / chunks, t0 = (blockIdx.y % chunks) * CONV_T;
    const float4 wv = *(const float4*)(w + (size_t)c * 4);
    const float* st = state + (size_t)s * state_stride + (size_t)c * 3;
    const float* xs = x + (size_t)s * n_tok * nc + c;
    float p0 = t0 >= 3 ? xs[(size_t)(t0 - 3) * nc] : st[t0], p1 = t0 >= 2 ? xs[(size_t)(t0 - 2) * nc] : st[t0 + 1], p2 = t0 >= 1 ? xs[(size_t)(t0 - 1) * nc] : st[t0 + 2];
    float cur[CONV_T];
#pragma unroll
    for (int i = 0; i < CONV_T; ++i) cur[i] = t0 + i < n_tok ? xs[(size_t)(t0 + i) * nc] : 0.0f;
#pragma unroll
    for (int i = 0; i < CONV_T; ++i) {
        if (t0 + i >= n_tok) break;
        float sum = 0.0f;
        sum += p0 * wv.x;
        sum += p1 * wv.y;
        sum += p2 * wv.z;
        sum += cur[i] * wv.w;
        out[((size_t)s * n_tok + t0 + i) * nc + c] = sum;
        p0 = p1; p1 = p2; p2 = cur[i];
    }
}
// The window each sequence leaves behind: its last kernel-1 inputs, oldest first. grid (ceil(nc/128), n_seq).
__global__ void k_conv_state(float* state, size_t state_stride, const float* x, int n_tok, int nc, int kernel) {
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x, s = blockIdx.y;
    if (c >= nc) return;
    const int keep = kernel - 1;
    float* st = state + (size_t)s * state_stride + (size_t)c * keep;
    float nv[8];
    for (int k = 0; k < keep; ++k) {
        const int idx = n_tok - keep + k;
        nv[k] = idx >= 0 ? x[((size_t)s * n_tok + idx) * nc + c] : st[keep + idx];
    }
    for (int k = 0; k < keep; ++k) st[k] = nv[k];
}

// Everything of the GatedDeltaNet block that does not depend on the state, per row: SiLU of the conv sums,
// l2-norm of q and k (q also scaled by 1/sqrt(sk)), the decay g and the write strength beta
// (src/model/qwen35.rs:1280-1316, src/ops/naive.rs:101-107, :254-273).
// Blocks (row, share of its jobs; row_share), a warp per head of q or k (NJ = sk / 32 elements a lane, the sum of squares in the same order
// as a warp per 32 of them), then per 128 elements of v, then per 32 heads' decays. Memory would bound it (131 MB at 2,048 rows of
// 8,192: 20 us); a block of 128 threads per head, with a block-wide sum and the decays by one lane, took 97 us, this 58: the
// library-exact exponential's f64 steps.
// Blocks that share a row's jobs (8 warps each): enough rows fill the machine on their own, few rows take a warp per job.
inline unsigned row_share(int rows, int jobs, int sms) { return (unsigned)std::max(1, std::min((jobs + 7) / 8, (8 * sms + rows - 1) / rows)); }
template <int NJ>
__global__ void __launch_bounds__(256) k_gdn_pre(const float* conv, int cd, const float* alpha, const float* beta, const float* ssm_a, const float* dt_bias,
                          int n_k, int n_v, float eps, float* qh, float* kh, float* vh, float* gb) {
    pdl_wait();
    constexpr int sk = NJ * 32;
    const size_t r = blockIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, key_dim = n_k * sk, vd = n_v * sk, vjobs = (vd + 127) / 128, jobs = 2 * n_k + vjobs + (n_v + 31) / 32;
    const float* cv = conv + r * cd;
    for (int u = blockIdx.y * 8 + wid; u < jobs; u += 8 * gridDim.y) {
        if (u < 2 * n_k) {
            const bool is_q = u < n_k;
            const int h = is_q ? u : u - n_k;
            const float* src = cv + (is_q ? 0 : key_dim) + h * sk + lane;
            float v[NJ];
            double tot = 0.0;
#pragma unroll
            for (int j = 0; j < NJ; ++j) v[j] = silu_f(src[32 * j]);
#pragma unroll
            for (int j = 0; j < NJ; ++j) tot += warp_sum_d((double)(v[j] * v[j]));
            const float sc = 1.0f / fmaxf(sqrtf((float)tot), eps), qs = 1.0f / sqrtf((float)sk);
            float* dst = (is_q ? qh : kh) + (r * n_k + h) * sk + lane;
#pragma unroll
            for (int j = 0; j < NJ; ++j) { float x = v[j] * sc; if (is_q) x = x * qs; dst[32 * j] = x; }
        } else if (u < 2 * n_k + vjobs) {
            const int i = (u - 2 * n_k) * 128 + lane * 4;
            if (i < vd) {
                const float4 x = *(const float4*)(cv + 2 * key_dim + i);
                *(float4*)(vh + r * vd + i) = make_float4(silu_f(x.x), silu_f(x.y), silu_f(x.z), silu_f(x.w));
            }
        } else {
            const int h = (u - 2 * n_k - vjobs) * 32 + lane;
            if (h < n_v) {
                const float a = alpha[r * n_v + h] + dt_bias[h];
                const float sp = a > 20.0f ? a : log_f(1.0f + exp_f(a));
                gb[(r * n_v + h) * 2] = exp_f(sp * ssm_a[h]);
                gb[(r * n_v + h) * 2 + 1] = sigmoid_f(beta[r * n_v + h]);
            }
        }
    }
}

// The recurrence itself (src/ops/naive.rs:109-132). A block is (value head, 32 value rows, sequence); a warp takes 8 of
// the rows, FOUR lanes per row, each lane holding a quarter of the row's state in registers across the pass's tokens.
// The CPU's serial sums over the 128 keys are kept to the bit: lane 0 of a row adds its quarter's products in order
// and hands the running sum to lane 1, and so on, so the chain is the CPU's chain; what the split buys is four times
// the warps and a quarter of the per-lane multiplies.
// Bound by that chain: 128 adds of 4 cycles a token, and a scheduler has about one warp, whose instructions go between them. So a
// token's read-out sum goes along with the NEXT token's prediction sum as the other half of packed adds (one instruction for both);
// the update, decay and products of a column are formed in the first quarter's steps, just ahead of the add that takes them; the
// next token's operands come during the other quarters, in straight-line code. A 512-token pass of 32 heads: 429 -> 256 us a layer
// (lines of a quarter are CW + 4 floats apart: the four lanes of a row read distinct banks, where they shared one).
template <int SK>
__global__ void __launch_bounds__(128) k_gdn_scan(const float* qh, const float* kh, const float* vh, const float* gb, int n_tok, int n_k, int n_v,
                                                  float* state, size_t state_stride, float* out) {
    pdl_wait();
    constexpr int CW = SK / 4;             // state columns per lane
    constexpr int QS = CW + 4, VEC = 4 * QS;
    constexpr int DEPTH = 5;               // tokens whose operands are in flight or in use (cp.async ring, one group per token)
    constexpr int SLOT = 2 * VEC + 8 + 4;  // floats per token and warp: k | q | v of the warp's 8 rows | g, beta, pad
    __shared__ __align__(16) float ring_all[4][DEPTH][SLOT];
    const int h = blockIdx.x, s = blockIdx.z, khd = h % n_k, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int r = lane >> 2, part = lane & 3, j0 = blockIdx.y * 32 + wid * 8, j = j0 + r;      // j: value row of the head
    float* sg = state + (size_t)s * state_stride + ((size_t)h * SK + j) * SK + part * CW;
    if (n_tok <= 0) return;
    // Straight-line on purpose: a branch would end the block of instructions that the sums' adds are spread over. pk, pq: this lane's
    // 16 bytes of k and q (two lanes copy the same at SK = 64); px: v's for lanes 0 and 1, g and beta for lane 2.
    const size_t row0 = (size_t)s * n_tok;
    const int e4 = lane * 4 % SK;
    const float* pk = kh + (row0 * n_k + khd) * SK + e4; const float* pq = qh + (row0 * n_k + khd) * SK + e4;
    const float* px = lane < 2 ? vh + (row0 * n_v + h) * SK + j0 + lane * 4 : gb + (row0 * n_v + h) * 2;
    const int step_k = n_k * SK, step_x = lane < 2 ? n_v * SK : n_v * 2;
    const uint32_t ring0 = (uint32_t)__cvta_generic_to_shared(ring_all[wid][0]), ring_z = ring0 + DEPTH * SLOT * 4;
    const uint32_t o_k = (uint32_t)(e4 / CW * QS + e4 % CW) * 4, o_x = (uint32_t)(2 * VEC + (lane < 2 ? lane * 4 : 8)) * 4;
    uint32_t put = ring0;
    auto fetch = [&](int t) {
        asm volatile("{.reg .pred p, a, b;\n setp.lt.s32 p, %0, %1;\n setp.lt.and.u32 a, %2, 2, p;\n setp.eq.and.u32 b, %2, 2, p;\n"
                     "@p cp.async.cg.shared.global [%3], [%4], 16;\n @p cp.async.cg.shared.global [%5], [%6], 16;\n"
                     "@a cp.async.cg.shared.global [%7], [%8], 16;\n @b cp.async.ca.shared.global [%7], [%8], 8;\n cp.async.commit_group;}"
                     ::"r"(t), "r"(n_tok), "r"(lane), "r"(put + o_k), "l"(pk), "r"(put + VEC * 4 + o_k), "l"(pq), "r"(put + o_x), "l"(px) : "memory");
        pk += step_k; pq += step_k; px += step_x;
        put += SLOT * 4; put = put == ring_z ? ring0 : put;
    };
    auto quarter = [](float* to, const float* from) {
#pragma unroll
        for (int i = 0; i < CW; i += 4) { const float4 v = *(const float4*)(from + i); to[i] = v.x; to[i + 1] = v.y; to[i + 2] = v.z; to[i + 3] = v.w; }
    };
    for (int t = 0; t < DEPTH - 1; ++t) fetch(t);
    float S[CW], qp[CW], k0[CW], k1[CW];
    uint64_t P[CW];                          // (prediction product, read-out product) of a column
    quarter(S, sg);
#pragma unroll
    for (int i = 0; i < CW; ++i) qp[i] = 0.0f;
    cp_async_wait<DEPTH - 2>();
    __syncwarp();
    const float* cur = ring_all[wid][0];
    quarter(k0, cur + part * QS);
    float v = cur[2 * VEC + r], g = cur[2 * VEC + 8], b = cur[2 * VEC + 9], d = 0.0f;
    float* o = out + ((size_t)s * n_tok * n_v + h) * SK + j;          // the read-out that is written next
    const int step_o = n_v * SK;
    auto write = [&](int t, float x) {
        asm volatile("{.reg .pred p;\n setp.ge.s32 p, %0, 0;\n setp.eq.and.s32 p, %1, 0, p;\n @p st.global.f32 [%2], %3;}" ::"r"(t), "r"(part), "l"(o), "f"(x) : "memory");
        o = t >= 0 ? o + step_o : o;
    };
    auto pair = [](float lo, float hi) { uint64_t p; asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi)); return p; };
    auto add2 = [](uint64_t& acc, uint64_t p) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(p)); };
    auto hand = [&](uint64_t& acc, int ph) {             // lane ph of a row hands both sums to the row's other lanes
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc));
        acc = pair(__shfl_sync(0xffffffffu, lo, (lane & ~3) | ph), __shfl_sync(0xffffffffu, hi, (lane & ~3) | ph));
    };
    auto add = [&](uint64_t& acc, int ph) {
#pragma unroll
        for (int i = 0; i < CW; ++i) add2(acc, P[i]);
        hand(acc, ph);
    };
    // Token t, its keys in kk (the token before's in kp, which takes the next token's). first: there is no token before.
    auto token = [&](int t, float* kk, float* kp, bool first) {
        uint64_t acc = pair(0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < CW; ++i) {
            float po = 0.0f;
            if (!first) { S[i] = S[i] + kp[i] * d; po = S[i] * qp[i]; }
            S[i] = S[i] * g;
            P[i] = pair(S[i] * kk[i], po);
            add2(acc, P[i]);
        }
        hand(acc, 0);
        fetch(t + DEPTH - 1);                // refills the slot token t - 1 used: every lane has its values (the shuffles)
        add(acc, 1);
        quarter(qp, cur + VEC + part * QS);
        cp_async_wait<DEPTH - 2>();          // token t + 1 is there (after the last token: stale values nothing uses)
        __syncwarp();
        cur = cur == ring_all[wid][DEPTH - 1] ? ring_all[wid][0] : cur + SLOT;
        const float vn = cur[2 * VEC + r], gn = cur[2 * VEC + 8], bn = cur[2 * VEC + 9];
        add(acc, 2);
        quarter(kp, cur + part * QS);
        add(acc, 3);
        float run, runo;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(run), "=f"(runo) : "l"(acc));
        write(t - 1, runo);
        d = b * (v - run);
        v = vn; g = gn; b = bn;
    };
    token(0, k0, k1, true);
    int t = 1;
#pragma unroll 1
    for (; t + 1 < n_tok; t += 2) { token(t, k1, k0, false); token(t + 1, k0, k1, false); }
    if (t < n_tok) {
        token(t, k1, k0, false);
#pragma unroll
        for (int i = 0; i < CW; ++i) k0[i] = k1[i];
    }
    float runo = 0.0f;                       // the last token's update and read-out
#pragma unroll
    for (int i = 0; i < CW; ++i) { S[i] = S[i] + k0[i] * d; qp[i] = S[i] * qp[i]; }
    for (int ph = 0; ph < 4; ++ph) {
#pragma unroll
        for (int i = 0; i < CW; ++i) runo += qp[i];
        runo = __shfl_sync(0xffffffffu, runo, (lane & ~3) | ph);
    }
    write(n_tok - 1, runo);
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < CW; i += 4) *(float4*)(sg + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
}
// One token per sequence (a batched decode step): the state passes through once, 8 rows (4 KB in a piece) to a warp, and memory bounds
// it -- so it moves as whole 16-byte spans in address order through shared memory (quarters CW + 4 floats apart, as above), with
// registers for several blocks an SM; the scan above, at one block's registers and 16 bytes of every 128 to a lane, took 53 us for 32
// sequences of 32 heads against 26 us here (134 MB: 20 us at copy speed). Same sums, same order.
template <int SK>
__global__ void __launch_bounds__(128, 4) k_gdn_step(const float* qh, const float* kh, const float* vh, const float* gb, int n_k, int n_v, float* state, size_t state_stride, float* out) {
    pdl_wait();
    constexpr int CW = SK / 4, QS = CW + 4, VEC = 4 * QS;
    __shared__ __align__(16) float st_all[4][8 * VEC], kq_all[4][2 * VEC];
    const int h = blockIdx.x, s = blockIdx.z, khd = h % n_k, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int r = lane >> 2, part = lane & 3, j0 = blockIdx.y * 32 + wid * 8;
    float* st = st_all[wid]; float* kq = kq_all[wid];
    float* sg = state + (size_t)s * state_stride + ((size_t)h * SK + j0) * SK;
    auto at = [](int e) { return (e / CW) * QS + e % CW; };                // element e of a warp's rows, or of k or q
#pragma unroll
    for (int i = 0; i < SK / 16; ++i) cp_async16(st + at((i * 32 + lane) * 4), sg + (i * 32 + lane) * 4, true);
    if (lane * 4 < SK) {
        cp_async16(kq + at(lane * 4), kh + ((size_t)s * n_k + khd) * SK + lane * 4, true);
        cp_async16(kq + VEC + at(lane * 4), qh + ((size_t)s * n_k + khd) * SK + lane * 4, true);
    }
    cp_async_commit();
    const float v = vh[((size_t)s * n_v + h) * SK + j0 + r], g = gb[((size_t)s * n_v + h) * 2], b = gb[((size_t)s * n_v + h) * 2 + 1];
    cp_async_wait<0>();
    __syncwarp();
    float S[CW], pr[CW];
    float* mine = st + r * VEC + part * QS; const float* k = kq + part * QS; const float* q = k + VEC;
#pragma unroll
    for (int i = 0; i < CW; i += 4) {
        const float4 x = *(const float4*)(mine + i), kv = *(const float4*)(k + i);
        S[i] = x.x * g; S[i + 1] = x.y * g; S[i + 2] = x.z * g; S[i + 3] = x.w * g;
        pr[i] = S[i] * kv.x; pr[i + 1] = S[i + 1] * kv.y; pr[i + 2] = S[i + 2] * kv.z; pr[i + 3] = S[i + 3] * kv.w;
    }
    auto fold = [&] {
        float run = 0.0f;
#pragma unroll
        for (int ph = 0; ph < 4; ++ph) {
            float a = run;
#pragma unroll
            for (int i = 0; i < CW; ++i) a += pr[i];
            run = __shfl_sync(0xffffffffu, a, (lane & ~3) | ph);
        }
        return run;
    };
    const float d = b * (v - fold());
#pragma unroll
    for (int i = 0; i < CW; i += 4) {
        const float4 kv = *(const float4*)(k + i), qv = *(const float4*)(q + i);
        float4 x;
        x.x = S[i] + kv.x * d; x.y = S[i + 1] + kv.y * d; x.z = S[i + 2] + kv.z * d; x.w = S[i + 3] + kv.w * d;
        pr[i] = x.x * qv.x; pr[i + 1] = x.y * qv.y; pr[i + 2] = x.z * qv.z; pr[i + 3] = x.w * qv.w;
        *(float4*)(mine + i) = x;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < SK / 16; ++i) *(float4*)(sg + (i * 32 + lane) * 4) = *(const float4*)(st + at((i * 32 + lane) * 4));
    const float o = fold();
    if (part == 0) out[((size_t)s * n_v + h) * SK + j0 + r] = o;
}

// Gated RMSNorm of the recurrence's output, the SiLU(z) gate and the Q8_0 quantisation of the result
// (src/model/qwen35.rs:1319-1325). Blocks and warps as in k_gdn_pre (75 MB at 2,048 rows of 4,096, 11 us; a block per head 65 us, this 42).
template <int NJ>
__global__ void __launch_bounds__(256) k_gdn_post(const float* o, const float* z, const float* norm_w, int n_v, float eps, int8_t* out_q, float* out_s) {
    pdl_wait();
    constexpr int sv = NJ * 32;
    const size_t r = blockIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float nw[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) nw[j] = norm_w[lane + 32 * j];
    for (int h = blockIdx.y * 8 + wid; h < n_v; h += 8 * gridDim.y) {
        const size_t idx = (r * n_v + h) * sv + lane;
        float v[NJ], g[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) { v[j] = o[idx + 32 * j]; g[j] = z[idx + 32 * j]; }
        double tot = 0.0;
#pragma unroll
        for (int j = 0; j < NJ; ++j) tot += warp_sum_d((double)(v[j] * v[j]));
        const float mean = (float)(tot / (double)sv);
        const float sc = 1.0f / sqrtf(mean + eps);
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const float core = v[j] * sc * nw[j];
            const float val = silu_f(g[j]) * core;
            float dq;
            const int8_t q = warp_quant_q8(val, &dq);
            out_q[idx + 32 * j] = q;
            if (lane == 0) out_s[idx / 32 + j] = dq;
        }
    }
}

// Attention prologue per (row, head): as k_attn_prep, the row's sequence and position derived from the pass
// shape: sequence = row / n_tok, position = pos[sequence] + row % n_tok.
struct AttnPrepRows {
    const float* qg; const float* k; const float* v;
    const float* q_norm; const float* k_norm;
    float* q_out; float* g_out;
    uint16_t* kslab; uint16_t* vslab; size_t slab_stride;
    const int* pos; int* npos_out; int n_tok;
    int hd, n_head, n_head_kv, n_rot; float theta, eps; int bf16;
};
// Blocks and warps as in k_gdn_pre: the row's rotations once, in double as the CPU takes them, then a warp per head (a block per (row,
// head) took each rotation 18 times: 116 us at 2,048 rows of 16 + 2 + 2 heads of 256, this 63). Dynamic shared memory: n_rot + 8 * hd floats.
__global__ void __launch_bounds__(256) k_attn_prep_rows(AttnPrepRows p) {
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    const int hd = p.hd, nj = hd / 32, half = p.n_rot / 2, kvd = p.n_head_kv * hd, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    float* cs = (float*)smem; float* sn = cs + half; float* val = sn + half + wid * hd;
    const size_t r = blockIdx.x;
    const int s = (int)(r / p.n_tok), pos = p.pos[s] + (int)(r % p.n_tok);
    if (tid == 0 && blockIdx.y == 0) p.npos_out[r] = pos + 1;
    for (int d = tid; d < half; d += 256) {
        const double freq = pow((double)p.theta, -2.0 * (double)d / (double)p.n_rot), th = (double)pos * freq;
        sn[d] = (float)sin(th); cs[d] = (float)cos(th);
    }
    __syncthreads();
    for (int job = blockIdx.y * 8 + wid; job < p.n_head + 2 * p.n_head_kv; job += 8 * gridDim.y) {
        const bool is_q = job < p.n_head, is_k = !is_q && job < p.n_head + p.n_head_kv;
        const int hk = is_q ? job : is_k ? job - p.n_head : job - p.n_head - p.n_head_kv;
        const float* src = is_q ? p.qg + r * 2 * hd * p.n_head + (size_t)hk * 2 * hd : (is_k ? p.k : p.v) + r * kvd + hk * hd;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) if (j < nj) v[j] = src[lane + 32 * j];
        if (is_q)
#pragma unroll
            for (int j = 0; j < 8; ++j) if (j < nj) p.g_out[(r * p.n_head + hk) * hd + lane + 32 * j] = src[hd + lane + 32 * j];
        if (is_q || is_k) {
            double tot = 0.0;
#pragma unroll
            for (int j = 0; j < 8; ++j) if (j < nj) tot += warp_sum_d((double)(v[j] * v[j]));
            const float mean = (float)(tot / (double)hd);
            const float sc = 1.0f / sqrtf(mean + p.eps);
            const float* nw = is_q ? p.q_norm : p.k_norm;
            __syncwarp();                              // everyone has the job before's values
#pragma unroll
            for (int j = 0; j < 8; ++j) if (j < nj) { v[j] = v[j] * sc * nw[lane + 32 * j]; val[lane + 32 * j] = v[j]; }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int d = lane + 32 * j;
                if (j < nj && d < half) v[j] = v[j] * cs[d] - val[d + half] * sn[d];
                else if (j < nj && d < 2 * half) v[j] = val[d - half] * sn[d - half] + v[j] * cs[d - half];
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j >= nj) continue;
            const int d = lane + 32 * j;
            if (is_q) p.q_out[(r * p.n_head + hk) * hd + d] = v[j];
            else (is_k ? p.kslab : p.vslab)[(size_t)s * p.slab_stride + (size_t)pos * kvd + hk * hd + d] = p.bf16 ? f32_to_bf16_bits(v[j]) : f32_to_f16_bits(v[j]);
        }
    }
}

// Combine of the attention splits per (row, head) with the sigmoid gate and Q8_0 quantisation; positions per row.
__global__ void k_attn_combine_rows(const float* part_acc, const float* part_ml, int n_split, int hd, const float* gate,
                                    const int* n_pos_row, int n_head, int8_t* out_q, float* out_s) {
    pdl_wait();
    const size_t th = blockIdx.x;
    const int d = threadIdx.x;
    const size_t r = th / n_head;
    const int n_pos = n_pos_row[r], per = max(ATTN_MIN_SPLIT, (n_pos + n_split - 1) / n_split), n_act = (n_pos + per - 1) / per;
    float M = -INFINITY;
    for (int s = 0; s < n_act; ++s) M = fmaxf(M, part_ml[(th * n_split + s) * 2]);
    float L = 0.0f, A = 0.0f;
    for (int s = 0; s < n_act; ++s) {
        float ms = part_ml[(th * n_split + s) * 2];
        float c = ms == -INFINITY ? 0.0f : __expf(ms - M);
        L += part_ml[(th * n_split + s) * 2 + 1] * c;
        A += part_acc[(th * n_split + s) * hd + d] * c;
    }
    float v = A / L;
    v *= sigmoid_f(gate[th * hd + d]);
    float dq;
    int8_t q = warp_quant_q8(v, &dq);
    out_q[th * hd + d] = q;
    if ((d & 31) == 0) out_s[(th * hd + d) / 32] = dq;
}

__global__ void k_advance_pos(int* pos, int n_seq, int by) {
    pdl_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_seq) pos[i] += by;
}
// Rows of the last token of each sequence, gathered for the LM head: out[s] = x[s*n_tok + n_tok-1].
__global__ void k_gather_last(const float* x, int n, int n_tok, float* out) {
    pdl_wait();
    const int s = blockIdx.x;
    for (int i = threadIdx.x; i < n; i += blockDim.x) out[(size_t)s * n + i] = x[((size_t)s * n_tok + n_tok - 1) * n + i];
}

}  // namespace

// =====================================================================================================
// Routed experts for many rows: route once per row, group the (row, pick) pairs by expert, and run each
// expert's rows through the int8-MMA NVFP4 kernels so an expert's weights are read once per pass
// (the reference groups the same way, kernels/moe.cuh:62-133 there; the order inside an expert is ascending
// pair index, so results do not depend on scheduling).
// =====================================================================================================
namespace {

// Softmax over all experts + top-k per row (src/model/qwen35.rs:1626-1638, src/ops/mod.rs:1191-1216). One warp per row. What bounds it is
// the one chain after another: the sum (in index order; its terms are read 32 ahead, or each add would wait for its own read) and the rounds of picks.
__global__ void __launch_bounds__(128) k_route_rows(const float* router, int n_rows, int n_expert, int n_used, int32_t* ids_out, float* w_out) {
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int ne32 = (n_expert + 31) & ~31;
    float* probs = (float*)smem + wid * ne32;
    const int r = blockIdx.x * nw + wid;
    if (r >= n_rows) return;
    const float* lg = router + (size_t)r * n_expert;
    float mx = -INFINITY;
#pragma unroll 4
    for (int i = lane; i < n_expert; i += 32) { const float v = lg[i]; probs[i] = v; mx = fmaxf(mx, v); }
    mx = warp_max(mx);
    for (int i = lane; i < ne32; i += 32) probs[i] = i < n_expert ? exp_f(probs[i] - mx) : 0.0f;       // behind the end: terms that change no sum
    __syncwarp();
    float sum = 0.0f;
#pragma unroll 1
    for (int i = 0; i < ne32; i += 32) {
        float4 a[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = *(const float4*)(probs + i + 4 * j);
#pragma unroll
        for (int j = 0; j < 8; ++j) { sum += a[j].x; sum += a[j].y; sum += a[j].z; sum += a[j].w; }
    }
    __syncwarp();                                    // every lane has read all of them
    for (int i = lane; i < n_expert; i += 32) probs[i] /= sum;
    __syncwarp();
    int32_t id; float w;
    warp_topk_any(probs, n_expert, n_used, id, w);
    if (lane < n_used) { ids_out[(size_t)r * n_used + lane] = id; w_out[(size_t)r * n_used + lane] = w; }
}

// silu(gate) * up of the shared expert per row, quantised (src/model/qwen35.rs:1669-1678). block per row.
__global__ void k_shared_act_rows(const float* sg, const float* su, int n, int8_t* q, float* s) {
    pdl_wait();
    const size_t r = blockIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int b = wid; b < n / 32; b += nw) {
        const size_t i = r * n + b * 32 + lane;
        float d;
        q[i] = warp_quant_q8(silu_f(sg[i]) * su[i], &d);
        if (lane == 0) s[r * (n / 32) + b] = d;
    }
}
// Weighted expert sum in pick order, gated shared expert, residual add (src/ops/mod.rs:1134-1171, src/model/qwen35.rs:1090).
__global__ void k_moe_finish_rows(float* x, int n, const float* o, const float* wts, int n_used, const float* shared, const float* logit, size_t total) {
    pdl_wait();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const size_t r = i / n; const int j = (int)(i % n);
    const float lg = logit[r], sh = shared[r * n + j], xv = x[i];
    float v = 0.0f;
    for (int k0 = 0; k0 < n_used; k0 += 8) {         // eight picks' loads in flight, and the exponential under the first eight's
        float wv[8], rv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k0 + k < n_used) { wv[k] = wts[r * n_used + k0 + k]; rv[k] = o[(r * n_used + k0 + k) * n + j]; }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k0 + k < n_used) v += wv[k] * rv[k];
    }
    v += sh * sigmoid_f(lg);
    x[i] = xv + v;
}

}  // namespace

namespace {

// Pairs grouped by expert without a serial scan: counts by shared-memory atomics, an exclusive scan, then each
// pair takes the next free place of its expert. The order inside an expert depends on scheduling; results do
// not, since every pair is computed on its own. One block.
// tiles (optional): the pairs cut into tiles of at most `cap` (a multiple of 8), an expert's pairs evenly over its tiles, as
// (expert, first slot, pairs, 0), largest first so that no long tile starts last; *n_tiles of them.
__global__ void __launch_bounds__(1024) k_group_pairs_fast(const int32_t* ids, int n_pairs, int n_expert, int* off, int* list, int4* tiles = nullptr, int* n_tiles = nullptr, int cap = 64) {
    pdl_wait();
    extern __shared__ int cnt[];    // [n_expert] counts, then cursors
    __shared__ int s_off[1025];
    __shared__ int s_bucket[9], s_start[9];       // tiles by groups of 8 pairs (1..8)
    if (threadIdx.x < 9) s_bucket[threadIdx.x] = 0;
    for (int e = threadIdx.x; e < n_expert; e += blockDim.x) cnt[e] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n_pairs; i += blockDim.x) atomicAdd(&cnt[ids[i]], 1);
    __syncthreads();
    if (threadIdx.x < 32) {
        // warp scan over experts in chunks of 32
        int carry = 0;
        for (int e0 = 0; e0 < n_expert; e0 += 32) {
            const int e = e0 + threadIdx.x;
            const int c = e < n_expert ? cnt[e] : 0;
            int inc = c;
            for (int o = 1; o < 32; o <<= 1) { int v = __shfl_up_sync(0xffffffffu, inc, o); if ((int)threadIdx.x >= o) inc += v; }
            if (e < n_expert) { off[e] = carry + inc - c; s_off[e] = carry + inc - c; }
            carry += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (threadIdx.x == 0) off[n_expert] = carry;
    }
    __syncthreads();
    // this thread's expert (at most 1024 of them): its tiles' size and the sizes' count
    const int te = threadIdx.x, tc = tiles && te < n_expert ? cnt[te] : 0, nt = (tc + cap - 1) / cap;
    const int per = nt ? (((tc + nt - 1) / nt) + 7) & ~7 : 8;
    for (int i = 0; i < nt; ++i) { const int m = min(per, tc - i * per); if (m > 0) atomicAdd(&s_bucket[(m + 7) >> 3], 1); }
    __syncthreads();
    if (threadIdx.x == 0 && tiles) {
        int at = 0;
        for (int b = 8; b >= 1; --b) { s_start[b] = at; at += s_bucket[b]; }
        *n_tiles = at;
    }
    for (int e = threadIdx.x; e < n_expert; e += blockDim.x) cnt[e] = 0;
    __syncthreads();
    for (int i = 0; i < nt; ++i) { const int m = min(per, tc - i * per); if (m > 0) tiles[atomicAdd(&s_start[(m + 7) >> 3], 1)] = make_int4(te, s_off[te] + i * per, m, 0); }
    for (int i = threadIdx.x; i < n_pairs; i += blockDim.x) { const int e = ids[i]; list[s_off[e] + atomicAdd(&cnt[e], 1)] = i; }
}

}  // namespace
