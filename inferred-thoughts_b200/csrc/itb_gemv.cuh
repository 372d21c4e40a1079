// Row-streaming GEMV cores for decode: HBM-bound, 16-byte coalesced weight loads, integer dot per
// quantisation block, and an order-preserving f32 fold so every output equals the CPU path's
// `sumf += term_b` chain to the bit (src/ops/naive.rs:691-734).
//
// Shape of the code: small loop bodies and many warps. A decode GEMV touches every instruction once per
// row, so straight-line unrolled kernels spend their time fetching instructions; here a warp loops over
// its rows RP at a time with all loads of a trip issued before the first dot.
//
// Work split inside a warp: G lanes share a row (G = power of two dividing the row's unit count),
// 32/G rows run side by side, RP such groups per pass. Each lane owns fixed K-columns, computes the
// integer sums of its 32-element units, turns them into f32 terms in shared memory; then one lane per row
// folds that row's terms in ascending order.
#pragma once
#include "itb_internal.cuh"

__device__ __forceinline__ uint4 ld_stream16(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// Where element e of a 32-element activation block stands in the f16 rows the many-row expert kernels read (itb_exp.cuh): the 8
// elements a lane of an MMA quad multiplies (4 of each 16-element half) lie together, so one 16-byte read feeds two MMAs. The
// NVFP4 nibbles lie the same way (k_repack_fp4).
__host__ __device__ __forceinline__ int exp_pos(int e) { return ((e & 15) >> 2) * 8 + (e >> 4) * 4 + (e & 3); }
__device__ __forceinline__ uint32_t f16x2_of_ints(int a, int b) {
    const __half2 h = __halves2half2(__int2half_rn(a), __int2half_rn(b));
    return *(const uint32_t*)&h;
}

// ---- activation prologues ------------------------------------------------------------------------
// RMSNorm of one row into shared memory: f32 squares, f64 accumulation (tree), (x*scale)*w
// (src/ops/naive.rs:139-152, :633-640). `red` holds blockDim.x/32 doubles.
// With xq/xs given, the vector path also quantises the normalised row to Q8_0 in the same pass (8 consecutive lanes hold
// one 32-block; src/ops/naive.rs:653-675) and returns true; otherwise the caller quantises from xn. xh: the quants also as f16
// in the order of exp_pos.
__device__ __forceinline__ bool block_rms_norm(const float* __restrict__ x, const float* __restrict__ w, int n, float eps,
                                               float* xn, double* red, int8_t* xq = nullptr, float* xs = nullptr, __half* xh = nullptr) {
    const int wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((n & 3) == 0 && n <= 16 * (int)blockDim.x && ((((uintptr_t)x) | ((uintptr_t)w) | ((uintptr_t)xn)) & 15) == 0) {
        // the row and the norm weights as float4, every load in flight before the first use: one memory round trip
        float4 xv[4], wv[4];
        const int nv = n >> 2;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = threadIdx.x + j * blockDim.x;
            if (i < nv) { xv[j] = ((const float4*)x)[i]; wv[j] = __ldg((const float4*)w + i); }
        }
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if ((int)(threadIdx.x + j * blockDim.x) < nv)
                acc += (double)(xv[j].x * xv[j].x) + (double)(xv[j].y * xv[j].y) + (double)(xv[j].z * xv[j].z) + (double)(xv[j].w * xv[j].w);
        acc = warp_sum_d(acc);
        if ((threadIdx.x & 31) == 0) red[wid] = acc;
        __syncthreads();
        // the warps' partial sums in warp order, by one lane per warp (the f64 unit is slow: every thread adding all of them
        // was most of this prologue), handed to the others by shuffle
        double tot = 0.0;
        if ((threadIdx.x & 31) == 0) for (int i = 0; i < nw; ++i) tot += red[i];
        tot = __shfl_sync(0xffffffffu, tot, 0);
        const float mean = (float)(tot / (double)n);
        const float sc = 1.0f / sqrtf(mean + eps);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = threadIdx.x + j * blockDim.x;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < nv) { o = make_float4(xv[j].x * sc * wv[j].x, xv[j].y * sc * wv[j].y, xv[j].z * sc * wv[j].z, xv[j].w * sc * wv[j].w); ((float4*)xn)[i] = o; }
            if (xq && (int)(j * blockDim.x) < nv) {      // whole warps take this branch together: nv and blockDim are multiples of 8 and 32
                float amax = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fmaxf(fabsf(o.z), fabsf(o.w)));
                amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
                amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
                amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
                const float d = amax / 127.0f, id = d != 0.0f ? 1.0f / d : 0.0f;
                if (i < nv) {
                    char4 q;
                    q.x = (signed char)fminf(127.0f, fmaxf(-128.0f, roundf(o.x * id))); q.y = (signed char)fminf(127.0f, fmaxf(-128.0f, roundf(o.y * id)));
                    q.z = (signed char)fminf(127.0f, fmaxf(-128.0f, roundf(o.z * id))); q.w = (signed char)fminf(127.0f, fmaxf(-128.0f, roundf(o.w * id)));
                    ((char4*)xq)[i] = q;
                    if (xh) *(uint2*)(xh + (size_t)(i >> 3) * 32 + exp_pos((i & 7) * 4)) = make_uint2(f16x2_of_ints(q.x, q.y), f16x2_of_ints(q.z, q.w));
                    if ((i & 7) == 0) xs[i >> 3] = __half2float(__float2half_rn(d));
                }
            }
        }
        __syncthreads();
        return xq != nullptr;
    }
    double acc = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) { float v = x[i]; xn[i] = v; acc += (double)(v * v); }
    acc = warp_sum_d(acc);
    if ((threadIdx.x & 31) == 0) red[wid] = acc;
    __syncthreads();
    double tot = 0.0;
    if ((threadIdx.x & 31) == 0) for (int i = 0; i < nw; ++i) tot += red[i];
    tot = __shfl_sync(0xffffffffu, tot, 0);
    float mean = (float)(tot / (double)n);
    float sc = 1.0f / sqrtf(mean + eps);
    for (int i = threadIdx.x; i < n; i += blockDim.x) xn[i] = xn[i] * sc * w[i];
    __syncthreads();
    return false;
}

// One Q8_0 block of 32 values held one per lane (src/ops/naive.rs:653-675): d = amax/127 through f16,
// q = roundf(v * (1/d)). Returns the lane's quant; *d_out (all lanes) the f16-rounded scale.
__device__ __forceinline__ int8_t warp_quant_q8(float v, float* d_out) {
    float amax = warp_max(fabsf(v));
    float d = amax / 127.0f;
    float id = d != 0.0f ? 1.0f / d : 0.0f;
    float r = roundf(v * id);
    *d_out = __half2float(__float2half_rn(d));
    return (int8_t)fminf(127.0f, fmaxf(-128.0f, r));
}
// Q8_0 activation quantiser over a row in shared or global memory: one warp per 32-block.
__device__ __forceinline__ void block_quant_q8(const float* xn, int n, int8_t* xq, float* xs) {
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int b = wid; b < n / 32; b += nw) {
        float d;
        xq[b * 32 + lane] = warp_quant_q8(xn[b * 32 + lane], &d);
        if (lane == 0) xs[b] = d;
    }
    __syncthreads();
}

// log2 of the lanes sharing a row: the largest power of two (<= 32) dividing the row's unit count.
__host__ __device__ __forceinline__ int lanes_shift(int units) {
    int sh = 0;
    while (sh < 5 && units % (2 << sh) == 0) sh++;
    return sh;
}
// shared-memory floats one warp needs for its term matrix
__host__ __device__ __forceinline__ int terms_floats(int rp, int gsh, int n_terms) { return rp * (32 >> gsh) * (n_terms + 1); }

// E2M1 codes to doubled integer magnitudes {0,1,2,3,4,6,8,12} (src/quant/mod.rs:265) with one byte
// permute per four codes: the selector's bit 3 asks for the sign of the selected (positive) byte, i.e. 0,
// so `prmt(pool, w)` yields the magnitudes of the positive codes and zeros elsewhere, and the same on
// `w ^ 0x8888` yields the magnitudes of the negative codes.
// (The __byte_perm intrinsic masks bit 3 of each selector, so the PTX instruction is issued directly.)
__device__ __forceinline__ uint32_t prmt_raw(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
// A 16-byte unit of 32 codes (word t: elements 4t..4t+3 of the first 16 in the low half, of the second 16 in the high half)
// against 32 int8 values (xa: the first 16, xb: the second): the two sub-blocks' integer dots.
__device__ __forceinline__ void fp4_unit_dots(const uint4& w, const uint4& xa, const uint4& xb, int& s0, int& s1) {
    const uint32_t P0 = 0x03020100u, P1 = 0x0c080604u;
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w}, a[4] = {xa.x, xa.y, xa.z, xa.w}, b[4] = {xb.x, xb.y, xb.z, xb.w};
    int p0 = 0, n0 = 0, p1 = 0, n1 = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const uint32_t v = ww[t], n = v ^ 0x88888888u;
        p0 = __dp4a((int)prmt_raw(P0, P1, v), (int)a[t], p0);
        n0 = __dp4a((int)prmt_raw(P0, P1, n), (int)a[t], n0);
        p1 = __dp4a((int)prmt_raw(P0, P1, v >> 16), (int)b[t], p1);
        n1 = __dp4a((int)prmt_raw(P0, P1, n >> 16), (int)b[t], n1);
    }
    s0 = p0 - n0; s1 = p1 - n1;
}

// One lane's 32-element unit of one Q8_0 row: 32 quants and the f16 scale.
struct UnitW { uint4 a, b; uint32_t s; };
__device__ __forceinline__ void unit_load(UnitW& w, const uint8_t* pa, const uint8_t* pb, int u) {
    w.a = ld_stream16(pa + u * 32); w.b = ld_stream16(pa + u * 32 + 16);
    w.s = __ldg((const uint16_t*)(pb + u * 2));
}
// The unit's f32 term into t (row's term array), against the activation unit xa|xb with scale dx.
__device__ __forceinline__ void unit_terms(const UnitW& w, const uint4& xa, const uint4& xb, float dx, float* t, int u) {
    int s = 0;
    s = __dp4a((int)w.a.x, (int)xa.x, s); s = __dp4a((int)w.a.y, (int)xa.y, s);
    s = __dp4a((int)w.a.z, (int)xa.z, s); s = __dp4a((int)w.a.w, (int)xa.w, s);
    s = __dp4a((int)w.b.x, (int)xb.x, s); s = __dp4a((int)w.b.y, (int)xb.y, s);
    s = __dp4a((int)w.b.z, (int)xb.z, s); s = __dp4a((int)w.b.w, (int)xb.w, s);
    t[u] = i2f_small(s) * (f16_bits_to_f32((uint16_t)w.s) * dx);           // src/ops/naive.rs:701
}
// One NVFP4 row's 64 elements (v0 | v1: its 32 bytes, s4: its 4 scale codes) against 64 int8 activations with two block scales:
// the four sub-blocks' f32 terms.
__device__ __forceinline__ void fp4_group_terms(const uint4& v0, const uint4& v1, uint32_t s4, const int8_t* xq, const float* xs, float* t) {
    const uint4* x = (const uint4*)xq;
    int a, b;
    float d0, d1;
    fp4_unit_dots(make_uint4(v0.x, v0.z, v1.x, v1.z), x[0], x[1], a, b);
    ue4m3x2_half(s4 & 0xffffu, d0, d1);
    t[0] = xs[0] * d0 * i2f_small(a); t[1] = xs[0] * d1 * i2f_small(b);           // src/ops/naive.rs:730
    fp4_unit_dots(make_uint4(v0.y, v0.w, v1.y, v1.w), x[2], x[3], a, b);
    ue4m3x2_half(s4 >> 16, d0, d1);
    t[2] = xs[1] * d0 * i2f_small(a); t[3] = xs[1] * d1 * i2f_small(b);
}
// A warp on one 16-row tile of an NVFP4 matrix (nib, sc: the tile), groups [g0, g1) of 64 elements: lane = (row, group parity), so a
// trip reads two groups, 1 KB in one piece. UB trips are loaded before the first dot. Terms go to t[row * stride + term].
template <int UB> struct Fp4Trips { uint4 v[UB][2]; uint32_t s[UB]; };
template <int UB>
__device__ __forceinline__ void fp4_trips_load(Fp4Trips<UB>& w, const uint8_t* __restrict__ nib, const uint8_t* __restrict__ sc, int k0, int g1) {
    const int r = threadIdx.x & 15;
#pragma unroll
    for (int i = 0; i < UB; ++i)
        if (k0 + 2 * i < g1) {
            const uint8_t* p = nib + (size_t)(k0 + 2 * i) * 512 + r * 32;
            w.v[i][0] = ld_stream16(p); w.v[i][1] = ld_stream16(p + 16);
            w.s[i] = __ldg((const uint32_t*)(sc + (size_t)(k0 + 2 * i) * 64 + r * 4));
        }
}
template <int UB>
__device__ __forceinline__ void fp4_trips_terms(const Fp4Trips<UB>& w, int k0, int g1, const int8_t* xq, const float* xs, float* t, int stride) {
    const int r = threadIdx.x & 15;
#pragma unroll
    for (int i = 0; i < UB; ++i)
        if (k0 + 2 * i < g1) { const int k = k0 + 2 * i; fp4_group_terms(w.v[i][0], w.v[i][1], w.s[i], xq + k * 64, xs + k * 2, t + r * stride + k * 4); }
}
template <int UB>
__device__ __forceinline__ void fp4_tile_terms(const uint8_t* __restrict__ nib, const uint8_t* __restrict__ sc, int g0, int g1, const int8_t* xq, const float* xs, float* t, int stride) {
#pragma unroll 1
    for (int k0 = g0 + ((threadIdx.x >> 4) & 1); k0 < g1; k0 += 2 * UB) {
        Fp4Trips<UB> w;
        fp4_trips_load(w, nib, sc, k0, g1);
        fp4_trips_terms(w, k0, g1, xq, xs, t, stride);
    }
}
// Ascending fold of one row's terms.
__device__ __forceinline__ float fold_terms(const float* t, int nt) {
    float sum = 0.0f;
#pragma unroll 16
    for (int b = 0; b < nt; ++b) sum += t[b];   // a deep unroll keeps the loads ahead of the dependent adds
    return sum;
}

// Rows [r0, r1) of one matrix (planes pa/pb, row 0 first) against one quantised activation (xq, xs in shared
// memory). terms: warp-private shared scratch of terms_floats(RP, gsh, row_terms) floats. epi(row, value) is
// called by one lane per row. UB units per lane and trip are loaded before the first dot.
template <int RP, int UB, class Epi>
__device__ __forceinline__ void rows_direct_ub(const uint8_t* __restrict__ pa, const uint8_t* __restrict__ pb, int n_in, int r0, int r1,
                                            const int8_t* xq, const float* xs, float* terms, int gsh, Epi epi) {
    const int G = 1 << gsh, lane = threadIdx.x & 31, sub = lane & (G - 1), slot = lane >> gsh;
    const int SLOTS = 32 >> gsh, ROWS = RP * SLOTS;
    const int nunits = n_in >> 5, nt = n_in >> 5, stride = nt + 1;
    const int arb = n_in, brb = n_in / 16;
#pragma unroll 1
    for (int r = r0; r < r1; r += ROWS) {
#pragma unroll 1
        for (int u0 = sub; u0 < nunits; u0 += UB * G) {
            UnitW w[UB][RP];
#pragma unroll
            for (int i = 0; i < RP; ++i) {
                int row = r + i * SLOTS + slot;
                if (row < r1) {
#pragma unroll
                    for (int h = 0; h < UB; ++h)
                        if (u0 + h * G < nunits) unit_load(w[h][i], pa + (size_t)row * arb, pb + (size_t)row * brb, u0 + h * G);
                }
            }
#pragma unroll
            for (int h = 0; h < UB; ++h) {
                if (u0 + h * G < nunits) {
                    const int u = u0 + h * G;
                    const uint4 xa = *(const uint4*)(xq + u * 32), xb = *(const uint4*)(xq + u * 32 + 16);
                    const float dx = xs[u];
#pragma unroll
                    for (int i = 0; i < RP; ++i)
                        if (r + i * SLOTS + slot < r1) unit_terms(w[h][i], xa, xb, dx, terms + (i * SLOTS + slot) * stride, u);
                }
            }
        }
        __syncwarp();
        if (lane < ROWS && r + lane < r1) epi(r + lane, fold_terms(terms + lane * stride, nt));
        __syncwarp();
    }
}

// One trip's weights: units u0, u0 + G, .. (UB of them) of the rows r + slot, r + slot + SLOTS, .. (RP of them) below r1.
template <int RP, int UB> struct RowTrip { UnitW w[UB][RP]; };
template <int RP, int UB>
__device__ __forceinline__ void trip_load(RowTrip<RP, UB>& t, const uint8_t* __restrict__ pa, const uint8_t* __restrict__ pb, int n_in, int r, int r1, int u0, int gsh) {
    const int G = 1 << gsh, slot = (threadIdx.x & 31) >> gsh, SLOTS = 32 >> gsh, nunits = n_in >> 5;
#pragma unroll
    for (int i = 0; i < RP; ++i) {
        const int row = r + i * SLOTS + slot;
        if (row < r1) {
#pragma unroll
            for (int h = 0; h < UB; ++h)
                if (u0 + h * G < nunits) unit_load(t.w[h][i], pa + (size_t)row * n_in, pb + (size_t)row * (n_in / 16), u0 + h * G);
        }
    }
}
// As rows_direct_ub, but the terms of up to `br` rows are collected first and then folded by `br` lanes at
// once: the fold is a serial chain per row, so folding one or two rows at a time leaves most lanes idle and
// costs as many instructions as the dots themselves. terms: br * (row_terms + 1) floats, warp-private.
// A warp has a handful of trips, each a round trip to memory: the first one's weights (cur, trip_load of r0 and the lane's first unit)
// come from the caller, who can request them before the activation is there. (A second set of registers for the next trip's as well
// took the room of the next kernel's blocks and slowed the LM head from 92 to 126 us.)
template <int RP, int UB, class Epi>
__device__ __forceinline__ void rows_batched(RowTrip<RP, UB>& cur, const uint8_t* __restrict__ pa, const uint8_t* __restrict__ pb, int n_in, int r0, int r1,
                                             const int8_t* xq, const float* xs, float* terms, int br, int gsh, Epi epi) {
    const int G = 1 << gsh, lane = threadIdx.x & 31, sub = lane & (G - 1), slot = lane >> gsh;
    const int SLOTS = 32 >> gsh, ROWS = RP * SLOTS;
    const int nunits = n_in >> 5, nt = n_in >> 5, stride = nt + 1;
    br = min(br, 32) / ROWS * ROWS;   // whole passes per batch (the caller sizes terms for at least one pass)
#pragma unroll 1
    for (int rb = r0; rb < r1; rb += br) {
        const int rend = min(r1, rb + br);
#pragma unroll 1
        for (int r = rb; r < rend; r += ROWS) {
#pragma unroll 1
            for (int u0 = sub; u0 < nunits; u0 += UB * G) {
                if (r > r0 || u0 > sub) trip_load(cur, pa, pb, n_in, r, rend, u0, gsh);
#pragma unroll
                for (int h = 0; h < UB; ++h) {
                    if (u0 + h * G < nunits) {
                        const int u = u0 + h * G;
                        const uint4 xa = *(const uint4*)(xq + u * 32), xb = *(const uint4*)(xq + u * 32 + 16);
                        const float dx = xs[u];
#pragma unroll
                        for (int i = 0; i < RP; ++i) {
                            const int row = r + i * SLOTS + slot;
                            if (row < rend) unit_terms(cur.w[h][i], xa, xb, dx, terms + (row - rb) * stride, u);
                        }
                    }
                }
            }
        }
        __syncwarp();
        if (rb + lane < rend) epi(rb + lane, fold_terms(terms + lane * stride, nt));
        __syncwarp();
    }
}

template <int RP, class Epi>
__device__ __forceinline__ void rows_direct(const uint8_t* __restrict__ pa, const uint8_t* __restrict__ pb, int n_in, int r0, int r1,
                                            const int8_t* xq, const float* xs, float* terms, int gsh, Epi epi) {
    rows_direct_ub<RP, 2>(pa, pb, n_in, r0, r1, xq, xs, terms, gsh, epi);
}
template <int RP, class Epi>
__device__ __forceinline__ void q8_rows(const DevQ8& w, int r0, int r1, const int8_t* xq, const float* xs, float* terms, int gsh, Epi epi) {
    rows_direct<RP>((const uint8_t*)w.q, (const uint8_t*)w.s, w.n_in, r0, r1, xq, xs, terms, gsh, epi);
}
// ---- F32 rows --------------------------------------------------------------------------------------
// EXACT: serial-k left fold per output like the CPU path (src/ops/naive.rs:845-849). A warp takes one row at a time: the lanes
// fetch the weights (coalesced) and put the products w[k] * x[k] of a tile of the row into the warp's shared scratch, then
// lane 0 adds the tile's terms in k order -- the adds are the only dependent chain (n_in of them, about 4 cycles each);
// chains of different warps overlap. `tile`: warp-private scratch of `tile_floats` floats (at least 128).
// Otherwise: lane-strided partial sums and a shuffle tree (order differs, value within rounding); `tile` unused.
template <bool EXACT, class Epi>
__device__ __forceinline__ void f32_rows(const float* __restrict__ w, int n_in, int r0, int r1, const float* x, float* tile, Epi epi, int tile_floats = 1024) {
    const int lane = threadIdx.x & 31;
    if (EXACT) {
        float* t16 = tile + ((4 - (int)(((uintptr_t)tile >> 2) & 3)) & 3);     // 16-byte aligned view of the scratch (still an offset from `tile`: shared-memory loads stay shared-memory loads)
        const int T = max(128, (tile_floats - 4) / 128 * 128);
#pragma unroll 1
        for (int r = r0; r < r1; ++r) {
            const float* p = w + (size_t)r * n_in;
            float sum = 0.0f;
#pragma unroll 1
            for (int t0 = 0; t0 < n_in; t0 += T) {
                const int tn = min(T, n_in - t0);
#pragma unroll 4
                for (int k = lane * 4; k < tn; k += 128) {
                    if (k + 4 <= tn) {
                        const float4 wv = __ldg((const float4*)(p + t0 + k)), xv = *(const float4*)(x + t0 + k);
                        *(float4*)(t16 + k) = make_float4(wv.x * xv.x, wv.y * xv.y, wv.z * xv.z, wv.w * xv.w);
                    } else {
                        for (int j = k; j < tn; ++j) t16[j] = __ldg(p + t0 + j) * x[t0 + j];
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    // the chain: 16 terms are in registers while the next 16 are on their way from shared memory
                    int k = 0;
                    if (tn >= 32) {
                        float4 a0 = *(const float4*)(t16), a1 = *(const float4*)(t16 + 4), a2 = *(const float4*)(t16 + 8), a3 = *(const float4*)(t16 + 12);
#pragma unroll 1
                        for (; k + 32 <= tn; k += 16) {
                            const float4 b0 = *(const float4*)(t16 + k + 16), b1 = *(const float4*)(t16 + k + 20), b2 = *(const float4*)(t16 + k + 24), b3 = *(const float4*)(t16 + k + 28);
                            sum += a0.x; sum += a0.y; sum += a0.z; sum += a0.w; sum += a1.x; sum += a1.y; sum += a1.z; sum += a1.w;
                            sum += a2.x; sum += a2.y; sum += a2.z; sum += a2.w; sum += a3.x; sum += a3.y; sum += a3.z; sum += a3.w;
                            a0 = b0; a1 = b1; a2 = b2; a3 = b3;
                        }
                        sum += a0.x; sum += a0.y; sum += a0.z; sum += a0.w; sum += a1.x; sum += a1.y; sum += a1.z; sum += a1.w;
                        sum += a2.x; sum += a2.y; sum += a2.z; sum += a2.w; sum += a3.x; sum += a3.y; sum += a3.z; sum += a3.w;
                        k += 16;
                    }
                    for (; k < tn; ++k) sum += t16[k];
                }
                __syncwarp();
            }
            if (lane == 0) epi(r, sum);
        }
    } else {
#pragma unroll 1
        for (int r = r0; r < r1; ++r) {
            const float* p = w + (size_t)r * n_in;
            float s = 0.0f;
#pragma unroll 1
            for (int k0 = lane * 4; k0 < n_in; k0 += 128 * 8) {
                float4 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) if (k0 + 128 * j < n_in) v[j] = __ldg((const float4*)(p + k0 + 128 * j));
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int k = k0 + 128 * j;
                    if (k < n_in) s += v[j].x * x[k] + v[j].y * x[k + 1] + v[j].z * x[k + 2] + v[j].w * x[k + 3];
                }
            }
            s = warp_sum(s);
            if (lane == 0) epi(r, s);
        }
    }
}

// Serial-k F32 rows, F32S_ROWS rows to a block: lane = row, every lane folds ITS row in k order (product and sum rounded separately,
// src/ops/naive.rs:49-56), so the chains run side by side at one add latency per k for all of them. The unit's weights come
// from the device copy DevF32::wt (four k of a row together, rows next to each other): a stage of 256 k is 8 KB in one piece, fetched
// by ONE bulk asynchronous copy that signals the stage's `full` mbarrier; eight stages hold a whole unit of 2,048 k, requested before
// the norm. The chain of adds bounds the unit, so the folding warp does nothing else: F32S_MULT warps multiply a stage in place by the
// activation and signal `ready`, a feeding warp issues the copies of longer rows (f32_unit_feed), and the folding warp reads 16 k ahead of
// its adds and hands slots back (`empty`). Few rows to a unit, because a stage passes through shared memory three times: at 32 that took
// as long as the adds. From norm to result, 2,048 k: 32 rows with the folding warp multiplying 11.0 cycles a k, with multiplying warps
// 7.2, 8 rows 5.7 (the adds: 4). Waits are bounded: one that runs out stores `F32S_FAIL` in *err and the
// fold goes on over whatever the slot holds (the host reads *err after the step). n_in a multiple of 256.
constexpr int F32S_ROWS = 8, F32S_K = 256, F32S_STAGES = 8, F32S_STAGE_FLOATS = F32S_ROWS * F32S_K, F32S_FLOATS = F32S_STAGES * F32S_STAGE_FLOATS, F32S_MULT = 8;
constexpr int F32S_FAIL = 0x7001;
__device__ __forceinline__ bool f32s_wait(unsigned long long* bar, uint32_t parity, int* err) {
    const uint32_t b = (uint32_t)__cvta_generic_to_shared(bar);
    auto arrived = [&] {
        uint32_t ok;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(b), "r"(parity) : "memory");
        return ok != 0;
    };
    if (arrived()) return true;
    const long long t0 = clock64();
    for (;;) {
        if (arrived()) return true;
        if (clock64() - t0 > 2000000000ll) { if (err) atomicExch(err, F32S_FAIL); return false; }
    }
}
// One lane of the feeding warp: stage t of the unit into slot t % stages; first = the stages issued before anything was folded
// (no slot to wait for), then one stage per slot the folding warp hands back.
__device__ __forceinline__ void f32_unit_issue(const float* wt_unit, int t, float* ring, unsigned long long* full) {
    const int slot = t % F32S_STAGES;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(full + slot);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ring + slot * F32S_STAGE_FLOATS);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)(F32S_STAGE_FLOATS * 4)) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(wt_unit + (size_t)t * F32S_STAGE_FLOATS), "r"((uint32_t)(F32S_STAGE_FLOATS * 4)), "r"(bar) : "memory");
}
__device__ __forceinline__ void f32_unit_feed(const float* wt_unit, int n_in, float* ring, unsigned long long* full, unsigned long long* empty, int* err) {
    const int nst = n_in / F32S_K;
    for (int t = F32S_STAGES; t < nst; ++t) {
        if (!f32s_wait(empty + t % F32S_STAGES, (uint32_t)(t / F32S_STAGES - 1) & 1u, err)) return;
        f32_unit_issue(wt_unit, t, ring, full);
    }
}
// Warp `part` of F32S_MULT: its share of every stage's products, in place.
__device__ __forceinline__ void f32_unit_multiply(int n_in, int part, const float* x, float* ring, unsigned long long* full, unsigned long long* ready, int* err) {
    const int lane = threadIdx.x & 31, nst = n_in / F32S_K;
#pragma unroll 1
    for (int t = 0; t < nst; ++t) {
        const int slot = t % F32S_STAGES;
        f32s_wait(full + slot, (uint32_t)(t / F32S_STAGES) & 1u, err);
        float4* w = (float4*)(ring + slot * F32S_STAGE_FLOATS);
        const float4* xs = (const float4*)(x + t * F32S_K);
        constexpr int N = F32S_STAGE_FLOATS / 4 / (F32S_MULT * 32);
        float4 a[N], b[N];                          // all read first: the writes go where they came from
#pragma unroll
        for (int i = 0; i < N; ++i) { const int e = (i * F32S_MULT + part) * 32 + lane; a[i] = w[e]; b[i] = xs[e / F32S_ROWS]; }
#pragma unroll
        for (int i = 0; i < N; ++i)
            w[(i * F32S_MULT + part) * 32 + lane] = make_float4(__fmul_rn(a[i].x, b[i].x), __fmul_rn(a[i].y, b[i].y), __fmul_rn(a[i].z, b[i].z), __fmul_rn(a[i].w, b[i].w));
        if (t + F32S_STAGES < nst) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // these writes come before the copy that refills the slot
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(ready + slot)) : "memory");
    }
}
template <class Epi>
__device__ __forceinline__ void f32_rows_serial(int n_in, int r0, int nr, const float* ring, unsigned long long* ready,
                                                  unsigned long long* empty, int* err, Epi epi) {
    const int lane = threadIdx.x & 31, nst = n_in / F32S_K;
    const float4* at = (const float4*)ring + lane % F32S_ROWS;
    float sum = 0.0f;
    float4 a[4], b[4];                             // the 16 k being added and the 16 after them
    auto add = [&](const float4 (&v)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { sum = __fadd_rn(sum, v[i].x); sum = __fadd_rn(sum, v[i].y); sum = __fadd_rn(sum, v[i].z); sum = __fadd_rn(sum, v[i].w); }
    };
    f32s_wait(ready, 0, err);
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = at[i * F32S_ROWS];
#pragma unroll 1
    for (int t = 0; t < nst; ++t) {
        const int nx = t + 1 < nst ? t + 1 : t;
        const float4* p = at + (t % F32S_STAGES) * (F32S_STAGE_FLOATS / 4); const float4* q = at + (nx % F32S_STAGES) * (F32S_STAGE_FLOATS / 4);
#pragma unroll
        for (int j = 0; j < F32S_K / 4; j += 8) {
#pragma unroll
            for (int i = 0; i < 4; ++i) b[i] = p[(j + 4 + i) * F32S_ROWS];
            add(a);
            if (j + 8 == F32S_K / 4) f32s_wait(ready + nx % F32S_STAGES, (uint32_t)(nx / F32S_STAGES) & 1u, err);
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = j + 8 < F32S_K / 4 ? p[(j + 8 + i) * F32S_ROWS] : q[i * F32S_ROWS];
            add(b);
        }
        if (t + F32S_STAGES >= nst) continue;       // nobody waits for this slot any more
        __syncwarp();                               // every lane has this stage's products: its slot goes back
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(empty + t % F32S_STAGES)) : "memory");
    }
    if (lane < nr) epi(r0 + lane, sum);
}

// Contiguous share [lo, hi) of n items for part `i` of `parts`.
__device__ __forceinline__ void share(int n, int parts, int i, int& lo, int& hi) {
    lo = (int)(((long long)n * i) / parts);
    hi = (int)(((long long)n * (i + 1)) / parts);
}
