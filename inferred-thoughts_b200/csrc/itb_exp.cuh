// Routed experts (NVFP4 weights x Q8_0-quantised activations) for several rows at a time, in the CPU path's arithmetic, on the
// 16-bit tensor-core path (mma.sync m16n8k16, f32 accumulators).
//
// The CPU's term of one 16-element sub-block is  (dy * d) * (float)sum  with dy the activation block's f16-rounded scale, d the
// UE4M3 weight scale and sum = sum of E2M1 x int8 products (src/ops/naive.rs:714-734), added to the row's sum in sub-block order.
// dy * d has at most 15 significant bits and is exact in f32, so the term is the real number dy * d * sum rounded ONCE. Here an
// operand element is (E2M1 value * d), at most 6 significant bits between 2^-10 and 2688: exact in f16, as is an int8 activation.
// One MMA covers one sub-block; its products are integers of at most 15 bits times one power of two, so the tensor core's sum
// d * sum is exact whatever order it adds in, and dy times it rounds once: the CPU's term to the bit, for two f32 operations per
// (row, token, sub-block) instead of the five an integer MMA needs (convert twice, two scales, add). tests compare bits.
//
// Rates measured on this GPU: m16n8k16, f16 or int8, one per 2.0 cycles and SM; f32 pipe 128 lanes per cycle, so mul + add on the 128
// outputs of one are 2.0 cycles too, where the five operations behind an int8 dot would be 5.
//
// Two f32 operations go out as fma.rn.f32x2 / add.rn.f32x2 (two tokens per instruction: half the issue slots). The product is
// fma(c, dy, 0) and not mul.rn.f32x2: the assembler contracts a packed multiply and the packed add behind it into one fma
// (measured: 14 % of results lose the product's own rounding), which it cannot do to an fma. The zero comes from a register the
// compiler knows nothing about.
#pragma once
#include <cuda_fp16.h>
#include <type_traits>
#include "itb_tile.cuh"

namespace {

constexpr int EX_KC = 128;                               // elements of k per pipeline stage
constexpr int EX_XSTR = EX_KC * 2 + 64;                  // padded token stride: the fragment reads of a warp hit distinct banks
template <int NJ> struct ExpCfg {
    static constexpr int TOK = 8 * NJ;
    static constexpr int W = NJ <= 2 ? 4 : 8;            // warps
    static constexpr int WROWS = 32 * W;                 // weight rows per block: half gate and half up, or all of the down matrix
    static constexpr int BLOCKS = NJ <= 2 ? 4 : 2;       // to an SM
    static constexpr int VS = 16 * W + 4;                // floats per token of the gate and up tiles, which reuse the ring
    static constexpr int OFF_S = WROWS * EX_KC / 2;
    static constexpr int OFF_X = OFF_S + WROWS * (EX_KC / 16);
    static constexpr int STAGE = OFF_X + TOK * EX_XSTR;
    static constexpr int NST = 3;                        // stages
};
constexpr size_t EX_SMEM = 224 * 1024;
template <int NJ> static inline size_t exp_smem(int k) { return (size_t)ExpCfg<NJ>::NST * ExpCfg<NJ>::STAGE + (size_t)(k / 32) * ExpCfg<NJ>::TOK * 4; }

// Two E2M1 codes (low byte of w >> 8 * B, low nibble first) to two f16, times the scale pair: exact.
template <int B>
__device__ __forceinline__ uint32_t fp4x2_f16(uint32_t w, uint32_t d2) {
    uint32_t r;
    if (B == 0) asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %1; cvt.rn.f16x2.e2m1x2 %0, b0; }" : "=r"(r) : "r"(w));
    if (B == 1) asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %1; cvt.rn.f16x2.e2m1x2 %0, b1; }" : "=r"(r) : "r"(w));
    if (B == 2) asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %1; cvt.rn.f16x2.e2m1x2 %0, b2; }" : "=r"(r) : "r"(w));
    if (B == 3) asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %1; cvt.rn.f16x2.e2m1x2 %0, b3; }" : "=r"(r) : "r"(w));
    asm("mul.rn.f16x2 %0, %0, %1;" : "+r"(r) : "r"(d2));
    return r;
}
// Four UE4M3 codes to four f16 pairs (each scale twice).
__device__ __forceinline__ void ue4m3x4_pairs(uint32_t four, uint32_t (&d)[4]) {
    uint32_t lo, hi;
    asm("{ .reg .b16 a, b; mov.b32 {a, b}, %2; cvt.rn.f16x2.e4m3x2 %0, a; cvt.rn.f16x2.e4m3x2 %1, b; }" : "=r"(lo), "=r"(hi) : "r"(four));
    // (as half broadcasts, which the multiply can take as an operand modifier)
    auto bc = [](uint32_t v, int hi) {
        uint32_t r;
        if (hi) asm("{ .reg .b16 l, h; mov.b32 {l, h}, %1; mov.b32 %0, {h, h}; }" : "=r"(r) : "r"(v)); else asm("{ .reg .b16 l, h; mov.b32 {l, h}, %1; mov.b32 %0, {l, l}; }" : "=r"(r) : "r"(v));
        return r;
    };
    d[0] = bc(lo, 0); d[1] = bc(lo, 1); d[2] = bc(hi, 0); d[3] = bc(hi, 1);
}
// One sub-block: c = A x B (16 rows x 8 tokens, exact), then acc += round(c * dy) for the lane's four results, two at a time, product
// and sum rounded separately. a01: rows g, a23: row g + 8, tokens 2t and 2t + 1; zero2: two f32 zeros, opaque to the compiler.
__device__ __forceinline__ void exp_mma_add(unsigned long long& a01, unsigned long long& a23, const uint32_t (&A)[4], uint32_t b0, uint32_t b1, unsigned long long dy, unsigned long long zero2) {
    asm("{ .reg .f32 c0, c1, c2, c3; .reg .b64 p, q;\n"
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {c0, c1, c2, c3}, {%2, %3, %4, %5}, {%6, %7}, {%10, %10, %10, %10};\n"
        "mov.b64 p, {c0, c1}; mov.b64 q, {c2, c3};\n"
        "fma.rn.f32x2 p, p, %8, %9; fma.rn.f32x2 q, q, %8, %9;\n"
        "add.rn.f32x2 %0, %0, p; add.rn.f32x2 %1, %1, q; }"
        : "+l"(a01), "+l"(a23) : "r"(A[0]), "r"(A[1]), "r"(A[2]), "r"(A[3]), "r"(b0), "r"(b1), "l"(dy), "l"(zero2), "f"(0.0f));
}
__device__ __forceinline__ float f32_of_pair(unsigned long long v, int i) { return __uint_as_float((uint32_t)(i ? v >> 32 : v)); }

struct ExpArgs {
    DevFp4 wa, wb;                 // gate and up, or the down matrix (wb unused)
    const __half* xh;              // activation rows, f16 (int8 values), permuted inside 32-element blocks (exp_pos); [row][k]
    const float* xs;               // their block scales [row][k / 32]
    int div;                       // pair p reads row p / div
    const int4* tiles; const int* n_tiles; const int* list;   // k_group_pairs_fast
    float* out;                    // f32 results [pair][n_out]: silu(gate) * up, or the down row; null: quantised output below (gate + up only)
    __half* oh; float* os;         // the Q8_0 quantisation of the gated row as the down form reads it: f16 values [pair][n_out], scales [pair][n_out / 32]
    unsigned long long zero2;
};

// One 64-element group of k of a warp's two row tiles against NJA groups of 8 tokens. A compile-time group count: the loads, MMAs
// and f32 operations of all groups interleave, which is what hides their latencies (four warps to a scheduler).
// w0, w1: this lane's first word in the two tiles; s0, s1: its row's scales; xr: its token's row; xs: its token pair's scales.
template <int NJA, int NJ>
__device__ __forceinline__ void exp_stage(const unsigned char* w0, const unsigned char* w1, const unsigned char* s0, const unsigned char* s1, const unsigned char* xr,
                                          const float* xs, unsigned long long zero2, unsigned long long (&acc)[2][NJ][2]) {
    uint2 wv[2][2];                                  // [row tile][rows g, g + 8]: the words of both 32-element blocks
    uint32_t d[2][2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            wv[m][h] = *(const uint2*)((m ? w1 : w0) + h * 256);
            ue4m3x4_pairs(*(const uint32_t*)((m ? s1 : s0) + h * 32), d[m][h]);
        }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        uint32_t A[2][2][4];                         // [row tile][sub-block][fragment register]
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const uint32_t ra = u ? wv[m][0].y : wv[m][0].x, rb = u ? wv[m][1].y : wv[m][1].x;
            A[m][0][0] = fp4x2_f16<0>(ra, d[m][0][2 * u]); A[m][0][2] = fp4x2_f16<1>(ra, d[m][0][2 * u]);
            A[m][1][0] = fp4x2_f16<2>(ra, d[m][0][2 * u + 1]); A[m][1][2] = fp4x2_f16<3>(ra, d[m][0][2 * u + 1]);
            A[m][0][1] = fp4x2_f16<0>(rb, d[m][1][2 * u]); A[m][0][3] = fp4x2_f16<1>(rb, d[m][1][2 * u]);
            A[m][1][1] = fp4x2_f16<2>(rb, d[m][1][2 * u + 1]); A[m][1][3] = fp4x2_f16<3>(rb, d[m][1][2 * u + 1]);
        }
#pragma unroll
        for (int j = 0; j < NJA; ++j) {
            const uint4 x = *(const uint4*)(xr + j * 8 * EX_XSTR + u * 64);
            const unsigned long long dy = *(const unsigned long long*)(xs + u * 8 * NJ + 8 * j);
            exp_mma_add(acc[0][j][0], acc[0][j][1], A[0][0], x.x, x.y, dy, zero2);
            exp_mma_add(acc[1][j][0], acc[1][j][1], A[1][0], x.x, x.y, dy, zero2);
            exp_mma_add(acc[0][j][0], acc[0][j][1], A[0][1], x.z, x.w, dy, zero2);
            exp_mma_add(acc[1][j][0], acc[1][j][1], A[1][1], x.z, x.w, dy, zero2);
        }
    }
}
// grid (tiles, ceil(n_out / (GLU ? 16 W : 32 W))), block 32 W: a block is one tile of an expert's pairs; a warp owns 16 gate rows and the same
// 16 up rows, or 32 rows of the down matrix, and all tokens of the tile (up to 8 * NJ); groups of 8 tokens past the tile's last pair are
// skipped, so a tile costs what it holds. k in stages of 128 through a cp.async ring, whose first weights are asked for before the
// pair list is read (they need the expert alone). Any n_in that is a multiple of 64.
// What bounds it: with 1-2 pairs per expert (batched decode) the start of a tile -- a block serves one and begins with an empty ring -- and
// the last round of blocks: four warps to a block and four blocks to an SM leave less of both than eight and two do (256 experts of
// 2048 x 512, 8 pairs to a row, gate + up and down: 32 rows 77 us against 85, 64 rows 106 and 116, 128 rows 122 and 128; 43 us are the
// bytes at 32 rows; blocks for 8 pairs, five to an SM: 75, 103, 118, but 164 against 152 at 256 rows). With many pairs: the MMAs and
// the f32 operations behind them, which overlap only in part (3.8 cycles per MMA and SM in the loop alone, against 2.0 for the MMAs and
// as much for the f32 pipe); there four warps to a block are the slower ones (512 rows, tiles of 32 pairs: 232 us against 213).
// Feeding the stages by bulk copies from a ninth warp was slower (1 KB and 128-byte pieces: 102 us against 63 at 32 tokens).
template <int NJ, bool GLU>
__global__ void __launch_bounds__(32 * ExpCfg<NJ>::W, ExpCfg<NJ>::BLOCKS) k_exp(ExpArgs p) {
    pdl_wait();
    extern __shared__ __align__(128) unsigned char smem[];
    using C = ExpCfg<NJ>;
    const int k = p.wa.n_in, n_out = p.wa.n_out;
    if ((int)blockIdx.x >= *p.n_tiles) return;
    const int4 tile_d = p.tiles[blockIdx.x];
    const int t0 = tile_d.y, n = tile_d.z, nja = (n + 7) >> 3, el = fp4_slot(p.wa, tile_d.x);
    if (el < 0) return;
    __shared__ int s_pair[C::TOK], s_row[C::TOK];
    float* s_xs = (float*)(smem + C::NST * C::STAGE);    // [k / 32][TOK]: the tile's activation scales
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, t = lane & 3;
    constexpr int W = C::W, VS = C::VS, RB = GLU ? 16 * W : 32 * W, XP = (C::TOK + 2 * W - 1) / (2 * W);
    const int r0 = blockIdx.y * RB, nb = k / 32, kgs = k / 64, n_chunk = (kgs + 1) / 2;
    // this warp's two row tiles of 16 inside the staged rows
    const int wr0 = GLU ? wid * 16 : wid * 32, wr1 = GLU ? 16 * W + wid * 16 : wid * 32 + 16;
    const bool rows_live = r0 + (GLU ? wid * 16 : wid * 32) < n_out;
    const bool has_a = p.wa.scale2 != nullptr, has_b = GLU && p.wb.scale2 != nullptr;
    const float s2a = has_a ? p.wa.scale2[el] : 1.0f, s2b = has_b ? p.wb.scale2[el] : 1.0f;
    // source addresses of this thread's pieces, advanced by a stage's bytes per stage. Weights: 2 W tiles x 1 KB per stage (64 lanes x
    // 16 bytes to a tile), scales: 2 W tiles x 128 bytes; rows past the matrix read its last tile. Tokens past the last are not
    // staged: what stands in their place reaches only their own results, which nobody reads.
    const uint8_t* wsrc[4]; const uint8_t* ssrc; const __half* xsrc[XP];
    {
        const size_t eo = (size_t)el * n_out;
        auto tile_row = [&](int tile) { return eo + min(r0 + (GLU ? (tile & (W - 1)) : tile) * 16, n_out - 16); };
#pragma unroll
        for (int i = 0; i < 4; ++i) wsrc[i] = (GLU && i >= 2 ? p.wb.nib : p.wa.nib) + tile_row((tid >> 6) + i * (W / 2)) * (k / 2) + (tid & 63) * 16;
        ssrc = (GLU && tid >= 8 * W ? p.wb.sc : p.wa.sc) + tile_row((tid >> 3) & (2 * W - 1)) * (k / 16) + (tid & 7) * 16;
    }
    auto load_w = [&](int c) {
        unsigned char* st = smem + (c % C::NST) * C::STAGE;
        const bool half = 2 * c + 2 > kgs;           // the last stage of a row that ends with 64 elements
        if (!half || (tid & 63) < 32) {
#pragma unroll
            for (int i = 0; i < 4; ++i) cp_async16(st + tid * 16 + i * W * 512, wsrc[i] + (size_t)c * 1024, true);
        }
        if (tid < 16 * W && (!half || (tid & 7) < 4)) cp_async16(st + C::OFF_S + tid * 16, ssrc + (size_t)c * 128, true);
    };
    auto load_x = [&](int c) {
        unsigned char* st = smem + (c % C::NST) * C::STAGE;
        const bool half = 2 * c + 2 > kgs;
        if (!half || (tid & 15) < 8) {
#pragma unroll
            for (int i = 0; i < XP; ++i)
                if (xsrc[i]) cp_async16(st + C::OFF_X + ((tid >> 4) + i * 2 * W) * EX_XSTR + (tid & 15) * 16, xsrc[i] + (size_t)c * EX_KC, true);
        }
    };
    auto load = [&](int c) { load_w(c); load_x(c); };
    int pr = 0;
    if (tid < n) pr = p.list[t0 + tid];
#pragma unroll
    for (int c = 0; c < C::NST - 1; ++c) if (c < n_chunk) load_w(c);
    if (tid < n) { s_pair[tid] = pr; s_row[tid] = pr / p.div; }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < XP; ++i) {                   // activations: 2 W tokens x 16 pieces of 16 bytes
        const int tk = (tid >> 4) + i * 2 * W;
        xsrc[i] = tk < n ? p.xh + (size_t)s_row[tk] * k + (tid & 15) * 8 : nullptr;
    }
#pragma unroll
    for (int c = 0; c < C::NST - 1; ++c) { if (c < n_chunk) load_x(c); cp_async_commit(); }
    for (int tk = wid; tk < n; tk += W)               // the tile's activation scales, [block][token]
        for (int b2 = lane; b2 < nb / 2; b2 += 32) {
            const float2 v = *(const float2*)(p.xs + (size_t)s_row[tk] * nb + 2 * b2);
            s_xs[(2 * b2) * C::TOK + tk] = v.x; s_xs[(2 * b2 + 1) * C::TOK + tk] = v.y;
        }
    unsigned long long acc[2][NJ][2];                // f32 pairs
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[m][j][0] = acc[m][j][1] = 0;
    // the whole k loop per group count (not one call per stage: the accumulators then stay where they are)
    auto walk = [&](auto count) {
        constexpr int NJA = decltype(count)::value;
        for (int c = 0; c < n_chunk; ++c) {
            cp_async_wait<C::NST - 2>();
            __syncthreads();                         // stage c has landed; everyone is done with stage c - 1
            if (c + C::NST - 1 < n_chunk) load(c + C::NST - 1);
            cp_async_commit();
            if (!rows_live) continue;
            const unsigned char* st = smem + (c % C::NST) * C::STAGE;
            const unsigned char* w = st + g * 32 + t * 8; const unsigned char* sc = st + C::OFF_S + g * 4;
            const unsigned char* xr = st + C::OFF_X + g * EX_XSTR + t * 16;
            const float* xsr = s_xs + (size_t)c * 4 * C::TOK + 2 * t;
            const int n_kg = min(2, kgs - 2 * c);
#pragma unroll(NJA <= 2 ? 2 : 1)
            for (int kg = 0; kg < 2; ++kg) {
                if (kg >= n_kg) break;
                exp_stage<NJA, NJ>(w + wr0 * (EX_KC / 2) + kg * 512, w + wr1 * (EX_KC / 2) + kg * 512, sc + wr0 * (EX_KC / 16) + kg * 64, sc + wr1 * (EX_KC / 16) + kg * 64,
                                   xr + kg * 128, xsr + kg * 2 * C::TOK, p.zero2, acc);
            }
        }
    };
    switch (nja) {
#define EX_CASE(N) case N: if constexpr (N <= NJ) walk(std::integral_constant<int, N>{}); break;
        EX_CASE(1) EX_CASE(2) EX_CASE(3) EX_CASE(4) EX_CASE(5) EX_CASE(6)
#undef EX_CASE
    }
    cp_async_wait<0>();
    if (GLU) {
        // the gate and up results go to [token][16 W rows] tiles in the ring's memory; from there a warp takes a token's 32 rows:
        // silu(gate * s_g) * (up * s_u) (src/ops/mod.rs:1105-1117), quantised to Q8_0 where the consumer is the down projection (it
        // would do the same), stored in whole pieces. (The library-exact exponential is a call: made here it has no accumulators to save.)
        float* vg = (float*)smem; float* vu = vg + C::TOK * VS;
        __syncthreads();                             // every warp is done with the ring
        if (rows_live) {
            const int o = 2 * t * VS + wid * 16 + g;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                if (NJ > 1 && j >= nja) break;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int at = o + (8 * j + (i & 1)) * VS + (i >> 1) * 8;
                    vg[at] = f32_of_pair(acc[0][j][i >> 1], i & 1); vu[at] = f32_of_pair(acc[1][j][i >> 1], i & 1);
                }
            }
        }
        __syncthreads();
        const int q = wid % (W / 2), row = r0 + q * 32;    // the warp's 32 rows, every other token
        if (row < n_out)
#pragma unroll 1
            for (int tk = wid / (W / 2); tk < n; tk += 2) {
                float gv = vg[tk * VS + q * 32 + lane], uv = vu[tk * VS + q * 32 + lane];
                if (has_a) gv = gv * s2a;
                if (has_b) uv = uv * s2b;
                const float val = silu_f(gv) * uv;
                const size_t pr = (size_t)s_pair[tk];
                if (p.out) p.out[pr * n_out + row + lane] = val;
                else {
                    float d;
                    const int8_t qv = warp_quant_q8(val, &d);
                    p.oh[pr * n_out + row + exp_pos(lane)] = __int2half_rn((int)qv);
                    if (lane == 0) p.os[pr * (n_out / 32) + row / 32] = d;
                }
            }
    } else if (rows_live) {
        const int row = r0 + wid * 32 + g;           // the warp's rows: row, + 8, + 16, + 24 (n_out is a multiple of 16)
        const bool second = r0 + wid * 32 + 16 < n_out;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            if (NJ > 1 && j >= nja) break;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int tk = 8 * j + 2 * t + h;
                if (tk >= n) continue;
                float* o = p.out + (size_t)s_pair[tk] * n_out + row;
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float v = f32_of_pair(acc[m][j][i], h);
                        if (m == 0 || second) o[m * 16 + i * 8] = has_a ? v * s2a : v;
                    }
            }
        }
    }
}
template <int NJ, bool GLU>
static inline void exp_launch(const ExpArgs& a, int max_tiles, cudaStream_t st) {
    itb_raise_smem(k_exp<NJ, GLU>, EX_SMEM);
    constexpr int W = ExpCfg<NJ>::W, RB = GLU ? 16 * W : 32 * W;
    itb_chain(k_exp<NJ, GLU>, dim3((unsigned)max_tiles, (unsigned)((a.wa.n_out + RB - 1) / RB)), 32 * W, exp_smem<NJ>(a.wa.n_in), st, a);
}
// The activation scales of a tile's whole rows lie beside the ring: up to 21,312 elements of k with 48 tokens.
static inline bool exp_k_ok(int k) { return exp_smem<6>(k) <= EX_SMEM; }
// Pairs per tile: 16, 32 or 48. A larger tile decodes an expert's weights once for more of its pairs; a smaller one has fewer
// accumulators and less of shared memory in activations, and an expert's pairs are cut evenly, so tiles of 32 end less unevenly than
// tiles of 48. Gate + up and down of 256 experts (2048 x 512), 8 pairs to a row, in us with 16 / 32 / 48 pairs: 128 rows 122 / 132 /
// 138, 256 rows 152 / 156 / 162, 384 rows 188 / 187 / 192, 512 rows 233 / 213 / 218, 768 rows 321 / 278 / 279, 1,024 rows 399 / 358 /
// 334, 5,548 rows 1909 / 1606 / 1497: 16 up to 8 pairs per expert on average, 32 up to 24. (64 pairs leave room for two stages only and
// spill: 180, 214, 240, 304, 365 and 1565 us from 256 rows on.) Where that leaves SMs without a block (few experts or short rows):
// as many pairs as give every SM four blocks.
static inline int exp_tile_cap(int n_pairs, int n_expert, int ff, int sms) {
    const int cap = n_pairs <= 8 * n_expert ? 16 : n_pairs <= 24 * n_expert ? 32 : 48;
    const int want = 4 * sms / ((ff + 127) / 128);                        // tiles, at (ff / 128) blocks each
    if (n_expert >= want) return cap;
    return std::min(cap, std::max(16, (n_pairs / std::max(want, 1) + 7) & ~7));
}
static inline int exp_max_tiles(int n_pairs, int n_expert, int cap) { return std::min(n_pairs, n_expert + n_pairs / cap); }
static inline void exp_run(ExpArgs a, bool glu, int max_tiles, int cap, cudaStream_t st) {
    a.zero2 = 0;
    if (cap <= 16) { if (glu) exp_launch<2, true>(a, max_tiles, st); else exp_launch<2, false>(a, max_tiles, st); }
    else if (cap <= 32) { if (glu) exp_launch<4, true>(a, max_tiles, st); else exp_launch<4, false>(a, max_tiles, st); }
    else { if (glu) exp_launch<6, true>(a, max_tiles, st); else exp_launch<6, false>(a, max_tiles, st); }
}

// Q8_0 quantisation of f32 rows as the kernels above read them: f16 values permuted inside blocks, block scales.
__global__ void __launch_bounds__(256) k_quant_rows_h(const float* x, size_t n_blocks, __half* xh, float* xs) {
    pdl_wait();
    quant_blocks(x, n_blocks, xs, [&](size_t, size_t b, int lane, int8_t q) { xh[b * 32 + exp_pos(lane)] = __int2half_rn((int)q); });
}
// int8 rows (already quantised) to the same form; a thread per 16 bytes.
__global__ void k_q8_to_h(const int8_t* xq, size_t n16, __half* xh) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n16) return;
    const uint4 v = ((const uint4*)xq)[i];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    __half* o = xh + (i >> 1) * 32 + (i & 1) * 4;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        __half2 lo, hi;
        lo.x = __int2half_rn((int)(int8_t)(w[t] & 0xff)); lo.y = __int2half_rn((int)(int8_t)((w[t] >> 8) & 0xff));
        hi.x = __int2half_rn((int)(int8_t)((w[t] >> 16) & 0xff)); hi.y = __int2half_rn((int)(int8_t)(w[t] >> 24));
        *(uint2*)(o + t * 8) = make_uint2(*(uint32_t*)&lo, *(uint32_t*)&hi);
    }
}

}  // namespace
