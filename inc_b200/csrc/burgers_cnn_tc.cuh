// The periodic CNN corrector's hidden layers on the tensor cores: shared by the
// forward rollout and its backward.
//
// A circular convolution of 32 channels to 32 channels, kernel 5, is five matrix
// products [cells x 32] x [32 x 32], one per tap, on the same activation tile
// shifted by one cell.  Activations sit in shared memory in the core-matrix layout of
// tc.cuh, one slot (16 bytes per 8 channels and piece) per cell, with the two halo
// cells of each side stored, so a tap is a start address 16 bytes further.  The
// weights' three pieces are stacked as 96 columns: the activations' hi and mid pieces take
// all 96 in one instruction each, lo 64 (hi, mid), each 32 columns further, so the 128
// accumulator columns are the sums of orders 0 to 3 (see tc.cuh).  One instruction of
// N = 96 issues in 56 cycles, N = 64 in 48, N = 32 in 45 (measured, M = 128, K = 16):
// 1,640 cycles for a layer of 128 cells against 6,550 on the FP32 pipes at their peak.
#pragma once
#include "burgers_cnn.cuh"
#include "gelu.cuh"
#include "tc.cuh"

namespace inc {
namespace burgers {
namespace cnn {

// One thread per cell, 128 or more threads: rows of at most 128 cells have a tile of
// 128 accumulator lanes each (a row of 64 cells leaves half of its tile unused; the
// second row of the CTA uses the upper half so that its threads' warps can read it).
template <int N>
struct TcCfg {
    static constexpr int T = N < 128 ? 128 : N;
    static constexpr int R = T / N;                  // rows per CTA
    static constexpr int SLOTS = R * (N + 4);        // cells with halos
    static constexpr int PLANE = SLOTS * 16;         // bytes of 8 channels of one piece
    static constexpr int TILES = N < 128 ? R : N / 128;
    static constexpr int COLS = 128 * TILES;
    static constexpr int WARPS_PER_ROW = N / 32;
};
constexpr int W_TAP = 96 * 32 * 2;             // bytes of one tap's stacked weight pieces
constexpr int W_LAYER = KW * W_TAP;            // bytes of one layer's
constexpr int W_PLANE = 96 * 16;

// Packed FP32 weights of a hidden layer ([ci][co][k]) -> stacked pieces, tap-major:
// tap k holds rows (piece, co), contraction ci.  TRANS: the layer's adjoint, rows
// (piece, ci), contraction co, taps reversed.  Each row has a scale of its own, so that
// the products of a row of small weights lie in order 0 as well; returns 2^e / 256 with 2^e >=
// the max |w| of row threadIdx.x % 32.  Two barriers; dst is scratch before the second.
template <int T, bool TRANS>
INC_DEV float stage_weights(unsigned char* dst, const float* __restrict__ w) {
    const int row = threadIdx.x % C, warp = threadIdx.x / C;
    float* part = reinterpret_cast<float*>(dst);
    float m = 0.f;
    for (int c = warp; c < C; c += T / C)
#pragma unroll
        for (int k = 0; k < KW; ++k)
            m = fmaxf(m, fabsf(__ldg(w + ((TRANS ? row : c) * C + (TRANS ? c : row)) * KW + k)));
    part[threadIdx.x] = m;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < T / C; ++i) m = fmaxf(m, part[i * C + row]);
    __syncthreads();
    const float s = tc::pow2_above(m), inv = 256.f / s;
    // item: tap k, row r (the product's output channel), 8 contraction channels c8
    for (int i = threadIdx.x; i < KW * C * (C / 8); i += T) {
        const int k = i / (C * (C / 8)), r = i % C, c8 = (i / C) % (C / 8);
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = 8 * c8 + j;
            const int ci = TRANS ? r : c, co = TRANS ? c : r, tap = TRANS ? KW - 1 - k : k;
            v[j] = __ldg(w + (ci * C + co) * KW + tap);
        }
        uint4 hi, mid, lo;
        tc::split8(v, inv, hi, mid, lo);
        unsigned char* p = dst + k * W_TAP + c8 * W_PLANE + r * 16;
        *reinterpret_cast<uint4*>(p) = hi;
        *reinterpret_cast<uint4*>(p + 32 * 16) = mid;
        *reinterpret_cast<uint4*>(p + 64 * 16) = lo;
    }
    return s * (1.f / 256.f);
}

// This thread's 32 channels at cell g of row rl, scaled by inv, into the slot and the
// halo copies that the row's ends own.  act: [3 pieces][4 planes][SLOTS][16 bytes].
template <int N>
INC_DEV void store_cell(unsigned char* act, const float (&v)[C], float inv, int rl, int g) {
    constexpr int PL = TcCfg<N>::PLANE;
    const int slot = rl * (N + 4) + g + 2;
    const int halo = g < 2 ? N : (g >= N - 2 ? -N : 0);
#pragma unroll
    for (int c8 = 0; c8 < 4; ++c8) {
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = v[8 * c8 + j];
        uint4 q[3];
        tc::split8(x, inv, q[0], q[1], q[2]);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            unsigned char* d = act + (p * 4 + c8) * PL + slot * 16;
            *reinterpret_cast<uint4*>(d) = q[p];
            if (halo != 0) *reinterpret_cast<uint4*>(d + halo * 16) = q[p];
        }
    }
}

// One layer's products for one tile: 5 taps x 2 channel halves, accumulators at
// columns d .. d + 127 of the tile's 128 lanes; one thread issues (tc::elect).
template <int N>
INC_DEV void issue_layer(uint32_t d, const unsigned char* act, const unsigned char* w, int tile) {
    constexpr int PL = TcCfg<N>::PLANE;
    // (rows of 64 cells: the second row's tile starts 64 slots early, see TcCfg)
    const int slot0 = N < 128 ? tile * (N + 4) - tile * 64 : tile * 128;
    const uint32_t a0 = tc::smem_u32(act) + slot0 * 16, b0 = tc::smem_u32(w);
    constexpr uint32_t i96 = tc::instr_desc(128, 96), i64 = tc::instr_desc(128, 64), i32 = tc::instr_desc(128, 32);
    const uint64_t ad = tc::smem_desc(a0, PL, 128), bd = tc::smem_desc(b0, W_PLANE, 128);
#pragma unroll
    for (int k = 0; k < KW; ++k) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint64_t b = tc::desc_at(bd, k * W_TAP + 2 * h * W_PLANE);
            const uint64_t a = tc::desc_at(ad, k * 16 + 2 * h * PL);
            const uint64_t mid = tc::desc_at(a, 4 * PL), lo = tc::desc_at(a, 8 * PL);
            tc::mma(d, a, b, i96, k + h > 0);
            if (k + h > 0) {
                tc::mma(d + 32, mid, b, i96, true);
            } else {  // (the first to write the last 32 columns)
                tc::mma(d + 32, mid, b, i64, true);
                tc::mma(d + 96, mid, tc::desc_at(b, 64 * 16), i32, false);
            }
            tc::mma(d + 64, lo, b, i64, true);
        }
    }
}

// 8 channels (c0 .. c0 + 7) of this thread's cell, the four orders added up
INC_DEV void read_orders8(uint32_t d, int c0, float2 (&z)[4]) {
    const float2 down = f2s(tc::DOWN);
    float v0[8], v1[8], v2[8], v3[8];
    tc::tmem_ld8(d + c0, v0);
    tc::tmem_ld8(d + 32 + c0, v1);
    tc::tmem_ld8(d + 64 + c0, v2);
    tc::tmem_ld8(d + 96 + c0, v3);
    tc::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const float2 s = __ffma2_rn(f2(v3[i], v3[i + 1]), down, f2(v2[i], v2[i + 1]));
        z[i / 2] = __ffma2_rn(__ffma2_rn(s, down, f2(v1[i], v1[i + 1])), down, f2(v0[i], v0[i + 1]));
    }
}

// the same times f and the weight rows' scales ws, plus bias
INC_DEV void read_layer8(uint32_t d, int c0, float f, const float* ws, const float* bias, float2 (&z)[4]) {
    read_orders8(d, c0, z);
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        const float4 b = lds4(bias + c0 + 2 * i), r = lds4(ws + c0 + 2 * i);
        z[i] = __ffma2_rn(__fmul2_rn(z[i], f2(r.x, r.y)), f2s(f), f2(b.x, b.y));
        z[i + 1] = __ffma2_rn(__fmul2_rn(z[i + 1], f2(r.z, r.w)), f2s(f), f2(b.z, b.w));
    }
}

// the same times f alone
INC_DEV void read_sums8(uint32_t d, int c0, float f, float2 (&z)[4]) {
    read_orders8(d, c0, z);
#pragma unroll
    for (int i = 0; i < 4; ++i) z[i] = __fmul2_rn(z[i], f2s(f));
}

// max |v| over this thread's channels and its row, of the finite values: an infinite one or NaN
// spoils the sums it enters, not the scale of the row's others (a barrier of the CTA inside;
// fails is or-ed over the CTA)
template <int N>
INC_DEV float row_absmax(const float (&v)[C], float* red, bool& fail, int rl) {
    float m = 0.f;
#pragma unroll
    for (int c = 0; c < C; ++c) m = fmaxf(m, fabsf(v[c]));
    m = group_max_nonneg<32>(m);
    if (isinf(m)) {
        m = 0.f;
#pragma unroll
        for (int c = 0; c < C; ++c) m = fmaxf(m, isinf(v[c]) ? 0.f : fabsf(v[c]));
        m = group_max_nonneg<32>(m);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    fail = __syncthreads_or(fail);
    constexpr int WPR = TcCfg<N>::WARPS_PER_ROW;
    m = 0.f;
#pragma unroll
    for (int i = 0; i < WPR; ++i) m = fmaxf(m, red[rl * WPR + i]);
    return m;
}

}  // namespace cnn
}  // namespace burgers
}  // namespace inc
