// Pipelined multi-token matmuls, Q8_0 weights x Q8_0-quantised rows in the CPU path's arithmetic: a block owns 16 RG weight rows x 8 NJ TG
// tokens and walks k in chunks of 256 elements through a ring of cp.async stages (weights, their scales, the activations and theirs),
// several chunks in flight. One int8 MMA per quantisation block, its int32 sum scaled and added to an f32 accumulator in ascending
// block order (src/ops/naive.rs:691-734).
#pragma once
#include <type_traits>
#include "itb_mma.cuh"

namespace {

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = valid ? 16 : 0;   // src-size 0: the 16 bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }

constexpr int TQ_KC = 256;                       // elements of k per stage
template <int RG, int TG, int NJ> struct TileCfg {
    static constexpr int ROWS = 16 * RG, TOK = 8 * NJ * TG, THREADS = 32 * RG * TG;
    static constexpr int STR = TQ_KC + 32;           // padded line: fragment reads hit distinct banks
    static constexpr int XSF = TQ_KC / 32 + 4;       // floats per token's line of scales, padded likewise
    static constexpr int OFF_S = ROWS * STR, OFF_X = OFF_S + ROWS * 16, OFF_XS = OFF_X + TOK * STR, STAGE = OFF_XS + TOK * XSF * 4;
};
// Up to three dense Q8_0 matrices over the same quantised rows in one launch (the input projections of a layer; the shared
// expert's gate and up): grid.x runs over the matrices' row tiles one after the other. A matrix of 512 rows alone is 32 blocks.
struct Q8Multi { DevQ8 w[3]; float* out[3]; size_t stride[3]; int tiles[3]; int n; };

// RG x TG warps, each 16 rows x 8 NJ tokens; groups of 8 tokens past the last row are neither staged nor multiplied. mode 0: out = v;
// mode 1: out += v. n_in a multiple of 256. grid (row tiles of all matrices, ceil(n_tok / TOK)).
// What bounds it, at 32 tokens: with many rows shared memory and the issue slots (LM head, 248,320 x 2048: a 16 x 8 product costs 8 cycles of
// an SM's shared-memory pipe -- fragments, scales, the staging itself -- and 27 issue slots; 176 us against 82 for the bytes); with few
// the latency of a stage and of the dot -> scale -> add chain, which is why all eight blocks of a stage are unrolled (a chunk's MMAs go out
// back to back), the scales of a row are one 16-byte read per chunk, and the first stages' weights are asked for before the rows are there.
template <int RG, int TG, int NJ, int NST>
__global__ void __launch_bounds__(32 * RG * TG, 3) k_tile_q8(Q8Multi p, const int8_t* xq, const float* xs, int n_tok, int mode) {
    using C = TileCfg<RG, TG, NJ>;
    extern __shared__ __align__(16) unsigned char smem[];
    int m = 0, bx = blockIdx.x;
    while (m + 1 < p.n && bx >= p.tiles[m]) { bx -= p.tiles[m]; ++m; }
    const DevQ8 w = p.w[m];
    const int k = w.n_in, nb = k / 32, n_chunk = k / TQ_KC, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, t = lane & 3;
    const int r0 = bx * C::ROWS, t0 = blockIdx.y * C::TOK, n = min(C::TOK, n_tok - t0);
    auto load_w = [&](int c) {
        unsigned char* st = smem + (c % NST) * C::STAGE;
#pragma unroll
        for (int i0 = 0; i0 < C::ROWS * 16; i0 += C::THREADS) {
            const int i = i0 + tid, r = i >> 4, q = i & 15, row = min(r0 + r, w.n_out - 1);
            cp_async16(st + r * C::STR + q * 16, (const uint8_t*)w.q + (size_t)row * k + (size_t)c * TQ_KC + q * 16, true);
        }
        if (tid < C::ROWS) cp_async16(st + C::OFF_S + tid * 16, (const uint8_t*)w.s + (size_t)min(r0 + tid, w.n_out - 1) * nb * 2 + (size_t)c * 16, true);
    };
    auto load_x = [&](int c) {
        unsigned char* st = smem + (c % NST) * C::STAGE;
#pragma unroll
        for (int i0 = 0; i0 < C::TOK * 16; i0 += C::THREADS) {
            const int i = i0 + tid, tk = i >> 4, q = i & 15;
            if (tk < n) cp_async16(st + C::OFF_X + tk * C::STR + q * 16, xq + (size_t)(t0 + tk) * k + (size_t)c * TQ_KC + q * 16, true);
        }
#pragma unroll
        for (int i0 = 0; i0 < C::TOK * 2; i0 += C::THREADS) {
            const int i = i0 + tid, tk = i >> 1, q = i & 1;
            if (tk < n) cp_async16(st + C::OFF_XS + tk * C::XSF * 4 + q * 16, (const unsigned char*)(xs + (size_t)(t0 + tk) * nb) + (size_t)c * 32 + q * 16, true);
        }
    };
#pragma unroll
    for (int c = 0; c < NST - 1; ++c) if (c < n_chunk) load_w(c);
    pdl_wait();
#pragma unroll
    for (int c = 0; c < NST - 1; ++c) { if (c < n_chunk) load_x(c); cp_async_commit(); }
    // this warp's rows and tokens inside the tile, and how many groups of 8 of its tokens exist
    const int rw = (wid % RG) * 16, tb = (wid / RG) * NJ * 8;
    const int nja = min(NJ, (n - tb + 7) >> 3);
    float acc[NJ][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = 0.0f;
    // the whole k loop per group count (a compile-time count: the loads, MMAs and sums of all groups interleave)
    auto walk = [&](auto count) {
        constexpr int NJA = decltype(count)::value;
        for (int c = 0; c < n_chunk; ++c) {
            cp_async_wait<NST - 2>();
            __syncthreads();                         // stage c has landed; everyone is done with stage c - 1
            if (c + NST - 1 < n_chunk) { load_w(c + NST - 1); load_x(c + NST - 1); }
            cp_async_commit();
            if (NJA == 0) continue;
            const unsigned char* st = smem + (c % NST) * C::STAGE;
            const unsigned char* wa = st + (rw + g) * C::STR + 8 * t;
            const unsigned char* xr = st + C::OFF_X + (tb + g) * C::STR + 8 * t;
            const float* xsr = (const float*)(st + C::OFF_XS) + (tb + 2 * t) * C::XSF;
            const uint4 sa = *(const uint4*)(st + C::OFF_S + (rw + g) * 16), sb = *(const uint4*)(st + C::OFF_S + (rw + g + 8) * 16);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float dx[NJA > 0 ? NJA : 1][2][4];
#pragma unroll
                for (int j = 0; j < NJA; ++j)
#pragma unroll
                    for (int q = 0; q < 2; ++q) { const float4 v = *(const float4*)(xsr + (8 * j + q) * C::XSF + 4 * h); dx[j][q][0] = v.x; dx[j][q][1] = v.y; dx[j][q][2] = v.z; dx[j][q][3] = v.w; }
                const uint2 s2a = h ? make_uint2(sa.z, sa.w) : make_uint2(sa.x, sa.y), s2b = h ? make_uint2(sb.z, sb.w) : make_uint2(sb.x, sb.y);
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const uint2 va = *(const uint2*)(wa + (4 * h + b) * 32), vb = *(const uint2*)(wa + 8 * C::STR + (4 * h + b) * 32);
                    const float da = f16_bits_to_f32((uint16_t)((b < 2 ? s2a.x : s2a.y) >> (16 * (b & 1)))), db = f16_bits_to_f32((uint16_t)((b < 2 ? s2b.x : s2b.y) >> (16 * (b & 1))));
#pragma unroll
                    for (int j = 0; j < NJA; ++j) {
                        const uint2 x = *(const uint2*)(xr + 8 * j * C::STR + (4 * h + b) * 32);
                        int cc[4];
                        mma_s8_k32(cc, va.x, vb.x, va.y, vb.y, x.x, x.y);
                        acc[j][0] += i2f_small(cc[0]) * (da * dx[j][0][b]);
                        acc[j][1] += i2f_small(cc[1]) * (da * dx[j][1][b]);
                        acc[j][2] += i2f_small(cc[2]) * (db * dx[j][0][b]);
                        acc[j][3] += i2f_small(cc[3]) * (db * dx[j][1][b]);
                    }
                }
            }
        }
    };
    if (nja <= 0) walk(std::integral_constant<int, 0>{});
    else if (NJ == 1 || nja == 1) walk(std::integral_constant<int, 1>{});
    else walk(std::integral_constant<int, NJ>{});
    cp_async_wait<0>();
    float* out = p.out[m];
    const int ra = r0 + rw + g, rb = ra + 8;
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int tk = t0 + tb + 8 * j + 2 * t + (i & 1), row = i < 2 ? ra : rb;
            if (tk < n_tok && row < w.n_out) { float* o = out + (size_t)tk * p.stride[m] + row; *o = mode ? *o + acc[j][i] : acc[j][i]; }
        }
}
template <int RG, int TG, int NJ, int NST>
static void tile_q8_launch(cudaStream_t st, Q8Multi p, const int8_t* xq, const float* xs, int n_tok, int mode) {
    using C = TileCfg<RG, TG, NJ>;
    static_assert(NJ <= 2, "the group counts k_tile_q8 walks");
    int tiles = 0;
    for (int i = 0; i < p.n; ++i) { p.tiles[i] = (p.w[i].n_out + C::ROWS - 1) / C::ROWS; tiles += p.tiles[i]; }
    itb_raise_smem(k_tile_q8<RG, TG, NJ, NST>, NST * C::STAGE);
    itb_chain(k_tile_q8<RG, TG, NJ, NST>, dim3((unsigned)tiles, (unsigned)((n_tok + C::TOK - 1) / C::TOK)), C::THREADS, (size_t)NST * C::STAGE, st, p, xq, xs, n_tok, mode);
}
// Tiles by how many there are, all of 32 tokens and three blocks to an SM: 16 rows while all fit the SMs at once, then 32 rows, and 64 (half
// the reads of the activations again) where even those are several to an SM. Measured (us, 16 / 32 / 64 rows; k 2048 unless said; in
// parentheses the kernel with 32 x 32 tiles, one group of 8 tokens to a warp and 64 x 64 tiles past 32 tokens that this one replaced):
// 32 tokens: 2,048 outputs of k 4096 7.6 / 10.7 / 17.8 (17.9), 4,096 6.6 / 6.6 / 10.0 (9.8), 6,144 9.3 / 10.2 / 10.4 (13.1), 12,288 16.1 / 13.6 / 16.3
// (21.1), 24,576 28.4 / 23.8 / 22.8 (36.9), 248,320 243 / 187 / 176 (311); 8 tokens: 2,048 of k 4096 6.4 / 7.9 / 13.6 (18.1), 12,288 12.0 / 8.8 / 10.0 (21.2),
// 24,576 20.3 / 15.5 / 12.5 (36.9), 248,320 181 / 118 / 102 (311); 200 tokens: 2,048 of k 4096 28.5 / 23.6 / 29.3 (34.4), 12,288 79 / 63 / 58 (103). Passes without the
// tensor cores, under ncu, 64 rows: 512 tokens 8,192 101 (127), 4,096 53 (72); 2,048 tokens 8,192 380 (491), 4,096 195 (250).
static void tile_q8(cudaStream_t st, int sms, const Q8Multi& p, const int8_t* xq, const float* xs, int n_tok, int mode) {
    long long blocks = 0;                                 // of 16 rows x 32 tokens
    for (int i = 0; i < p.n; ++i) blocks += (p.w[i].n_out + 15) / 16;
    blocks *= (n_tok + 31) / 32;
    if (blocks <= 3 * sms) tile_q8_launch<1, 4, 1, 4>(st, p, xq, xs, n_tok, mode);
    else if (blocks <= 8 * sms) tile_q8_launch<2, 2, 2, 3>(st, p, xq, xs, n_tok, mode);
    else tile_q8_launch<4, 2, 2, 2>(st, p, xq, xs, n_tok, mode);
}

}  // namespace
