// Backward of the hybrid Burgers rollout with the periodic CNN corrector on the tensor
// cores, from the forward's record of every step's state and of the hidden layers'
// pre-activations (z2, z3).  Same gradients as burgers_cnn_bwd.cu, which needs neither
// record and stays for rollouts whose record is too large.  Three launches:
//
//   k_cnn_adjoint  one CTA per row as in the forward (burgers_cnn.cu: one thread per cell), steps
//                  in reverse: the solver's adjoint, then the network's: the last and
//                  first layers per thread from registers, the hidden layers' input
//                  adjoints as convolutions with the transposed weights and reversed
//                  taps on the tensor cores (burgers_cnn_tc.cuh).  dL/dz2 and dL/dz3 of every
//                  step go to memory with the channels' maxima.  No replay: every u_k is
//                  recorded.  Bound by the chain of a step (the solver's adjoint, four row
//                  reductions and products waited for; issue slots half used at 16 warps an
//                  SM, all its registers taken): 920 us at 256 rows x 256 cells x 32 steps
//                  (865 with bf16 pieces, one scale per weight matrix and maxima by row).
//   k_cnn_wgrad    the hidden layers' weight gradients, dW[co][ci][k] = sum dz[co][x] a[ci][x + k -
//                  2] over all cells, steps and rows: cells are the contraction, so the
//                  same tile layout serves read by columns, a tap is again a start
//                  address one cell further.
//   k_cnn_grad_sum the blocks' partial sums in a fixed order.
//
// Splitting the weight gradients off costs a round trip of dz through memory (537 MB each way
// at 256 rows x 256 cells x 32 steps, hidden behind the products) and lets them run at the
// tensor cores' rate on all SMs: in one kernel, their five taps' accumulators (480 columns
// per layer) leave no room for the adjoints' and their operands none for a second CTA.
#include "burgers_cnn_tc.cuh"

namespace inc {
namespace burgers {
namespace cnn {

INC_DEV float2 lds2(const float* p) { return *reinterpret_cast<const float2*>(p); }

// sum over the 32 cells x0 .. x0 + 31 of row r
INC_DEV float cell_sum(const float* r, int x0) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 v = lds2(r + apad(x0 + 2 + 2 * i));
        s += v.x + v.y;
    }
    return s;
}

// acc[k] += sum over the 32 cells x0 .. x0 + 31 of dr[x] ar[x + k - 2]
INC_DEV void cell_products(float (&acc)[KW], const float* dr, const float* ar, int x0) {
    float win[36];  // cells x0 - 2 .. x0 + 33
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        const float4 v = lds4(ar + apad(x0 + 4 * i));
        win[4 * i] = v.x; win[4 * i + 1] = v.y; win[4 * i + 2] = v.z; win[4 * i + 3] = v.w;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 d = lds2(dr + apad(x0 + 2 + 2 * i));
#pragma unroll
        for (int k = 0; k < KW; ++k) {
            acc[k] = fmaf(d.x, win[2 * i + k], acc[k]);
            acc[k] = fmaf(d.y, win[2 * i + 1 + k], acc[k]);
        }
    }
}

constexpr int EDGE = 2 * C * KW + C + 3;  // dW1, dW4, db1, db4 (high and low part) of one block, 1 if it gave up
constexpr int HID = C * C * KW + C;       // one hidden layer's dW and db

struct AdjArgs {
    const float* w;        // packed weights
    const float* states;   // [rows][steps][N]
    const float* corr;     // [rows][steps][N]
    const float* g_corr;   // [rows][steps][N] or NULL
    const float* acts;     // [rows][steps][2][32][N]
    float* dz;             // [rows][steps][2][32][N]: dL/dz2, dL/dz3
    float* mx;             // [4][rows][steps][32]: max over the cells of |dL/dz2|, |dL/dz3|, |gelu(z1)|, |gelu(z2)|
    float* edge;           // [blocks][EDGE]
};

template <int N>
struct AdjSmem {
    using Cfg = TcCfg<N>;
    static constexpr int RL = row_len<N>();
    alignas(128) unsigned char w[2][W_LAYER];  // W2, W3 transposed, in pieces
    union {
        alignas(128) unsigned char act[3 * 4 * Cfg::PLANE];  // dz in pieces
        WideAdjSmem<N> sol[Cfg::R];                          // the solver's rows
        struct {
            float ch[Cfg::R][C][RL];    // a layer's values by channel (first and last layers' weight gradients)
            float part[Cfg::R][KW][N];  // the first layer's input adjoint by tap
        } o;
        float sums[Cfg::T / 32][C][2 * KW + 2];
    };
    alignas(16) float w1[KW][C], b1[C], w4[KW][C];
    alignas(16) float u[Cfg::R][RL], d[Cfg::R][RL];
    alignas(16) uint16_t cm[Cfg::T / 32][C];  // the warps' channel maxima, for layer 3 (bf16, which leaves two CTAs
                                              // per SM room); layer 2's take d's place, which layer 4 has read by then
    static_assert(Cfg::R * RL * sizeof(float) >= (Cfg::T / 32) * C * sizeof(uint16_t), "layer 2's channel maxima");
    uint64_t bar[Cfg::TILES];
    uint32_t tmem;
};

// max |v| over the warp (NaN left out)
INC_DEV float warp_absmax(float v) {
    float r;
    asm("redux.sync.max.abs.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
// the warp's max |v| of 4 channels, of the finite values (x + 0 x: an infinite one to NaN), as
// bf16 rounded down
INC_DEV void put_max4(uint16_t* out, float2 v0, float2 v1) {
    uint32_t m0, m1;
    v0 = __ffma2_rn(v0, f2s(0.f), v0);
    v1 = __ffma2_rn(v1, f2s(0.f), v1);
    asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(m0) : "f"(warp_absmax(v0.y)), "f"(warp_absmax(v0.x)));
    asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(m1) : "f"(warp_absmax(v1.y)), "f"(warp_absmax(v1.x)));
    if ((threadIdx.x & 31) == 0) *reinterpret_cast<uint2*>(out) = make_uint2(m0, m1);
}
// channel `lane`'s max over the warps of row rl (at least; at most 2^-7 above)
template <int N>
INC_DEV float channel_max(const uint16_t (*m)[C], int rl) {
    constexpr int WPR = TcCfg<N>::WARPS_PER_ROW;
    uint32_t r = 0;
#pragma unroll
    for (int i = 0; i < WPR; ++i) {
        const uint32_t e = m[rl * WPR + i][threadIdx.x & 31];
        r = e < 0x7f80u ? max(r, e) : r;  // (a warp without a finite value has NaN)
    }
    return __uint_as_float(r << 16) * 1.0078125f;
}

template <int N>
__global__ void __launch_bounds__(TcCfg<N>::T, N == 512 ? 1 : 2) k_cnn_adjoint(Args a, AdjArgs c) {
    using Cfg = TcCfg<N>;
    constexpr int T = Cfg::T, R = Cfg::R;
    extern __shared__ __align__(128) unsigned char smraw[];
    AdjSmem<N>& S = *reinterpret_cast<AdjSmem<N>*>(smraw);
    const int t = threadIdx.x, rl = t / N, g = t % N, w = t >> 5, lane = t & 31;
    const int pr = (32 * w) / N, px = (32 * w) % N;  // this warp's 32 cells: row, first cell
    const int tile = N < 128 ? rl : t / 128;
    const bool issuer = N < 128 ? g < 32 : t % 128 < 32;  // the warp that issues its tile's products
    const int row = blockIdx.x * R + rl;
    const bool valid = row < a.rows;
    const int src = valid ? row : 0;  // a row past the batch runs row 0 with zero adjoints
    if (t < 32) tc::tmem_alloc(&S.tmem, Cfg::COLS);
    if (t == 0) {
#pragma unroll
        for (int i = 0; i < Cfg::TILES; ++i) tc::mbar_init(&S.bar[i], 1);
        tc::mbar_init_fence();
    }
    for (int i = t; i < KW * C; i += T) {
        S.w1[i / C][i % C] = __ldg(c.w + OFF_W1 + (i % C) * KW + i / C);
        S.w4[i / C][i % C] = __ldg(c.w + OFF_W4 + (i % C) * KW + i / C);
    }
    if (t < C) S.b1[t] = __ldg(c.w + OFF_B1 + t);
    float ws[2];  // the weight rows' scales, lane = channel
    ws[0] = stage_weights<T, true>(S.w[0], c.w + OFF_W2);
    ws[1] = stage_weights<T, true>(S.w[1], c.w + OFF_W3);
    tc::fence_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t acc = S.tmem + 128 * tile + ((uint32_t)(t & 96) << 16);
    uint32_t phase = 0;
    bool fail = false;  // a wait for the tensor cores ran out: the gradients turn to NaN
    Ctx<1> cx;
    make_ctx<1, N>(a, src, g, true, cx);
    cx.has_s = true;
    uint16_t(*cm[2])[C] = {reinterpret_cast<uint16_t(*)[C]>(S.d), S.cm};  // by layer: of dz, then of its activations
    int parity = 0;
    float g1[KW], g4[KW], gb1 = 0.f;  // this warp's cells, lane = channel
    double gb4 = 0.0;  // this cell's share of db4: one scalar, whose terms cancel
#pragma unroll
    for (int k = 0; k < KW; ++k) g1[k] = g4[k] = 0.f;
    float gu = (a.g_final && valid) ? __ldg(a.g_final + (int64_t)row * N + g) : 0.f;
    // one hidden layer's input adjoint of v (dz): split, products, v = sums
    auto adjoint_layer = [&](float (&v)[C], int l, float m) {
        const float s = tc::pow2_above(m);
        store_cell<N>(S.act, v, 256.f / s, rl, g);
        tc::fence_smem();
        tc::fence_before();
        __syncthreads();
        if (issuer && tc::elect()) {
            tc::fence_after();
            issue_layer<N>(S.tmem + 128 * tile, S.act, S.w[l], tile);
            tc::commit(&S.bar[tile]);
        }
        return s * (1.f / 256.f);
    };
    auto wait_layer = [&] {
        if (!fail) fail = !tc::mbar_wait(&S.bar[tile], phase);
        phase ^= 1;
        tc::fence_after();
    };
    auto put_row = [&](float* r, float x) { put_cell<N>(r, g, x); };
    for (int k = a.steps - 1; k >= 0; --k) {
        const int64_t at = ((int64_t)src * a.steps + k) * N + g;
        const float u = __ldg(c.states + at);
        float v[C];  // z3
        {
            const float* p = acts_tile(const_cast<float*>(c.acts), src, a.steps, k, 1, 0, N) + g;
#pragma unroll
            for (int i = 0; i < C; ++i) v[i] = __ldg(p + i * N);
        }
        // ---- the solver step's adjoint: u_bar through S and s_bar
        float gs = 0.f;
        if (a.g_frames && valid) gu += __ldg(a.g_frames + at);
        cx.s[0] = __ldg(c.corr + at);
        advance_bwd_wide<N>(a, cx, u, gu, gs, cx.t + k * cx.dt, S.sol[rl], parity, g);
        if (c.g_corr && valid) gs += __ldg(c.g_corr + at);
        put_row(S.u[rl], u);
        put_row(S.d[rl], gs);
        gb4 += gs;
        __syncthreads();  // (also: the solver's rows are free)
        // ---- layer 4: gelu(z3) by channel for dW4; dz3 = (W4^T s_bar) gelu'(z3)
        {
            float2 dd[KW];
#pragma unroll
            for (int q = 0; q < KW; ++q) dd[q] = f2s(S.d[rl][apad(g + 4 - q)]);
#pragma unroll
            for (int i = 0; i < C; i += 2) {
                float2 y, gp, s = f2s(0.f);
                act::gelu_both2(f2(v[i], v[i + 1]), y, gp);
#pragma unroll
                for (int q = 0; q < KW; ++q) s = __ffma2_rn(*reinterpret_cast<const float2*>(&S.w4[q][i]), dd[q], s);
                put_row(S.o.ch[rl][i], y.x);
                put_row(S.o.ch[rl][i + 1], y.y);
                s = __fmul2_rn(s, gp);
                v[i] = s.x;
                v[i + 1] = s.y;
            }
        }
        __syncthreads();
        cell_products(g4, S.d[pr], S.o.ch[pr][lane], px);
        // ---- layer 3: dz3 out, dz2 = (W3^T dz3) gelu'(z2)
        float z2[C];
        {
            const float* p = acts_tile(const_cast<float*>(c.acts), src, a.steps, k, 0, 0, N) + g;
#pragma unroll
            for (int i = 0; i < C; ++i) z2[i] = __ldg(p + i * N);
        }
        auto put_mx = [&](int kind, float m) {
            if (g < 32 && valid) c.mx[(((int64_t)kind * a.rows + row) * a.steps + k) * C + lane] = m;
        };
#pragma unroll
        for (int i = 0; i < C; i += 4) put_max4(&cm[1][w][i], f2(v[i], v[i + 1]), f2(v[i + 2], v[i + 3]));
        fail = __syncthreads_or(fail);  // (also: S.o.ch is read)
        if (fail) break;
        float m = channel_max<N>(cm[1], rl);
        put_mx(1, m);
        if (valid) {
            float* p = acts_tile(c.dz, row, a.steps, k, 1, 0, N) + g;
#pragma unroll
            for (int i = 0; i < C; ++i) p[i * N] = v[i];
        }
        float f = adjoint_layer(v, 1, warp_absmax(m));
        // gelu'(z2) times the weight rows' scales, and gelu(z2)'s maxima, while the products run
        auto grad_and_max = [&](float(&z)[C], uint16_t(&out)[C], float scale) {
#pragma unroll
            for (int i = 0; i < C; i += 4) {
                float2 y0, y1, g0, g1;
                act::gelu_both2(f2(z[i], z[i + 1]), y0, g0);
                act::gelu_both2(f2(z[i + 2], z[i + 3]), y1, g1);
                put_max4(&out[i], y0, y1);
                g0 = __fmul2_rn(g0, f2(shfl<32>(scale, i), shfl<32>(scale, i + 1)));
                g1 = __fmul2_rn(g1, f2(shfl<32>(scale, i + 2), shfl<32>(scale, i + 3)));
                z[i] = g0.x; z[i + 1] = g0.y; z[i + 2] = g1.x; z[i + 3] = g1.y;
            }
        };
        grad_and_max(z2, cm[1][w], ws[1]);
        wait_layer();
#pragma unroll
        for (int i = 0; i < C; i += 8) {
            float2 s[4];
            read_sums8(acc, i, f, s);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                v[i + 2 * e] = s[e].x * z2[i + 2 * e];
                v[i + 2 * e + 1] = s[e].y * z2[i + 2 * e + 1];
            }
        }
        tc::fence_before();
        if (valid) {
            float* p = acts_tile(c.dz, row, a.steps, k, 0, 0, N) + g;
#pragma unroll
            for (int i = 0; i < C; ++i) p[i * N] = v[i];
        }
#pragma unroll
        for (int i = 0; i < C; i += 4) put_max4(&cm[0][w][i], f2(v[i], v[i + 1]), f2(v[i + 2], v[i + 3]));
        // ---- layer 2: dz1 = (W2^T dz2) gelu'(z1), z1 from u
        float z1[C];
        {
            float2 uu[KW];
#pragma unroll
            for (int q = 0; q < KW; ++q) uu[q] = f2s(S.u[rl][apad(g + q)]);
#pragma unroll
            for (int i = 0; i < C; i += 2) {
                float2 z = lds2(&S.b1[i]);
#pragma unroll
                for (int q = 0; q < KW; ++q) z = __ffma2_rn(*reinterpret_cast<const float2*>(&S.w1[q][i]), uu[q], z);
                z1[i] = z.x;
                z1[i + 1] = z.y;
            }
        }
        fail = __syncthreads_or(fail);  // (also: the products have read the tile)
        if (fail) break;
        m = channel_max<N>(cm[0], rl);
        put_mx(0, m);
        put_mx(3, channel_max<N>(cm[1], rl));
        f = adjoint_layer(v, 0, warp_absmax(m));
        grad_and_max(z1, cm[0][w], ws[0]);
        wait_layer();
#pragma unroll
        for (int i = 0; i < C; i += 8) {
            float2 s[4];
            read_sums8(acc, i, f, s);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                v[i + 2 * e] = s[e].x * z1[i + 2 * e];
                v[i + 2 * e + 1] = s[e].y * z1[i + 2 * e + 1];
            }
        }
        tc::fence_before();
        fail = __syncthreads_or(fail);  // (also: every tile's products have read the tile)
        if (fail) break;
        put_mx(2, channel_max<N>(cm[0], rl));
        // ---- layer 1: dz1 by channel for dW1, db1; the input adjoint by tap
        {
            float2 q[KW];
#pragma unroll
            for (int i = 0; i < KW; ++i) q[i] = f2s(0.f);
#pragma unroll
            for (int i = 0; i < C; i += 2) {
                put_row(S.o.ch[rl][i], v[i]);
                put_row(S.o.ch[rl][i + 1], v[i + 1]);
#pragma unroll
                for (int e = 0; e < KW; ++e)
                    q[e] = __ffma2_rn(*reinterpret_cast<const float2*>(&S.w1[e][i]), f2(v[i], v[i + 1]), q[e]);
            }
#pragma unroll
            for (int i = 0; i < KW; ++i) S.o.part[rl][i][g] = q[i].x + q[i].y;
        }
        __syncthreads();
        cell_products(g1, S.o.ch[pr][lane], S.u[pr], px);
        gb1 += cell_sum(S.o.ch[pr][lane], px);
        float du = 0.f;
#pragma unroll
        for (int i = 0; i < KW; ++i) du += S.o.part[rl][i][(g + 2 - i + N) & (N - 1)];
        gu += du;
        __syncthreads();  // the solver's rows take this memory again
    }
    if (valid) a.g_u[(int64_t)row * N + g] = fail ? __int_as_float(0x7fffffff) : gu;
    // this block's first- and last-layer gradients: one partial per warp, added in order
    __syncthreads();
    {
        float* p = S.sums[w][lane];
#pragma unroll
        for (int k = 0; k < KW; ++k) {
            p[k] = g1[k];
            p[KW + k] = g4[k];
        }
        p[2 * KW] = gb1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) gb4 += __shfl_xor_sync(0xffffffffu, gb4, o);
        const float high = (float)gb4;
        p[2 * KW + 1] = lane == 0 ? high : (float)(gb4 - high);  // (lane 1: the rest)
    }
    tc::fence_before();
    __syncthreads();
    if (t < 32) {
        float s[2 * KW + 2];
#pragma unroll
        for (int i = 0; i < 2 * KW + 2; ++i) s[i] = 0.f;
        for (int q = 0; q < T / 32; ++q)
#pragma unroll
            for (int i = 0; i < 2 * KW + 2; ++i) s[i] += S.sums[q][lane][i];
        float* e = c.edge + (int64_t)blockIdx.x * EDGE;
#pragma unroll
        for (int k = 0; k < KW; ++k) {
            e[lane * KW + k] = s[k];
            e[C * KW + lane * KW + k] = s[KW + k];
        }
        e[2 * C * KW + lane] = s[2 * KW];
        double b4 = 0.0;
        for (int q = 0; q < T / 32; ++q) b4 += (double)S.sums[q][0][2 * KW + 1] + S.sums[q][1][2 * KW + 1];
        if (lane == 0) {
            e[2 * C * KW + C] = (float)b4;
            e[2 * C * KW + C + 1] = (float)(b4 - (float)b4);
            e[2 * C * KW + C + 2] = fail ? 1.f : 0.f;
        }
        tc::tmem_free(S.tmem, Cfg::COLS);
    }
}

// ---- hidden layers' weight gradients ---------------------------------------------------
// A unit is 256 cells at one step (R rows of N <= 256 cells, or half a row of 512), a group
// GROUP steps of the same cells: its products accumulate in tensor memory with one scale per
// channel of dz and of a (the channel's maximum over the group), then the sums are read once.
// (A scale per group alone leaves a small channel's sums in the orders from 1 up, where the
// accumulator truncates at each of the 64 instructions: 1.3e-6 of the channel's gradient
// against 1.3e-7 in FP32.)  Lanes are (piece of dz, co), columns (tap, piece of a, ci); the
// nine piece pairs are added in registers, each with its order's power of two.  dz is scaled to
// 64, so that a group's 1024 terms of hi.hi stay below 2^24 (tc.cuh).
// Even blocks take layer 2 (a = gelu(z1), z1 from the recorded state), odd ones layer 3.
// The bias gradient is one more block of columns (a = 1).  16 warps prepare the two operand
// tiles (two buffers), a 17th issues.  Bound by the preparation (about 5,500 clocks a unit: two
// loads' latency, the split, GELU and the stores) and the reading of a group's sums, which
// the products of the group wait for; the products take 80 x 56 clocks.  256 rows x 256 cells x 32
// steps: 709 us in its first form; 629 with an elected issuer (tc::elect); 440 with the sums read
// without branches and the bias gradient out of the registers; 432 with the next unit's
// lines fetched to the L2; 475 with fp16 pieces (a longer split) and the channels' scales.  Not
// faster, measured against 432: 8 warps with the next values held in registers (432), 16 with
// them (478, spills), the sums kept in memory (707).
constexpr int WG = 512;
constexpr int GROUP = 4;
struct CnnWgradArgs {
    const float* w;       // packed weights (layer 1)
    const float* states;  // [rows][steps][N]
    const float* acts;
    const float* dz;
    const float* mx;
    float* part;          // [2][blocks / 2][HID]
    int rows, steps;
};
template <int N>
struct WgCfg {
    static constexpr int U = N < 256 ? N : 256;  // cells of a row in a unit
    static constexpr int R = 256 / U, H = N / U; // rows of a unit, units of a row
    static constexpr int PLANE = R * (U + 4) * 16;
};
template <int N>
struct CnnWgradSmem {
    struct Buf {
        alignas(128) unsigned char dz[3 * 4 * WgCfg<N>::PLANE];
        alignas(128) unsigned char a[(3 * 4 + 2) * WgCfg<N>::PLANE];  // two planes of ones follow the pieces
    } buf[2];  // (dz's lanes past 96 read on into a: not used)
    alignas(16) float w1[KW][C], b1[C];
    alignas(16) float up[2][2][C], down[2][2][C];  // by a group's parity, operand (dz, a), channel: scales, inverses
    uint64_t bar[2];
    uint32_t tmem;
};

INC_DEV void wg_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
INC_DEV void wg_hand_over(int buf) { asm volatile("bar.arrive %0, 544;" ::"r"(2 + buf) : "memory"); }
INC_DEV void wg_take_over(int buf) { asm volatile("bar.sync %0, 544;" ::"r"(2 + buf) : "memory"); }

// 16 channels (half of the planes) of one slot; up: the channels' scales
INC_DEV void store_half(unsigned char* tile, int plane, const float2 (&v)[8], const float* up, int slot, int half) {
#pragma unroll
    for (int c8 = 0; c8 < 2; ++c8) {
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const float4 s = lds4(up + 16 * half + 8 * c8 + 2 * j);
            tc::split2(v[4 * c8 + j], f2(s.x, s.y), h[j], m[j], l[j]);
            tc::split2(v[4 * c8 + j + 1], f2(s.z, s.w), h[j + 1], m[j + 1], l[j + 1]);
        }
        unsigned char* d = tile + (2 * half + c8) * plane + slot * 16;
        *reinterpret_cast<uint4*>(d) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(d + 4 * plane) = make_uint4(m[0], m[1], m[2], m[3]);
        *reinterpret_cast<uint4*>(d + 8 * plane) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

// accumulator columns of a tap's 96; the middle tap's are followed by 16 times dz summed (a = 1)
__host__ __device__ constexpr int tap_col(int k) { return 96 * k + (k > KW / 2 ? 16 : 0); }
constexpr int ONES = tap_col(KW / 2) + 96;

template <int N>
__global__ void __launch_bounds__(WG + 32, 1) k_cnn_wgrad(CnnWgradArgs a) {
    using Cfg = WgCfg<N>;
    constexpr int U = Cfg::U, R = Cfg::R, H = Cfg::H, PL = Cfg::PLANE;
    extern __shared__ __align__(128) unsigned char smraw[];
    CnnWgradSmem<N>& S = *reinterpret_cast<CnnWgradSmem<N>*>(smraw);
    const int tid = threadIdx.x, layer = blockIdx.x & 1;  // 0: W2, 1: W3
    const int me = blockIdx.x >> 1, blocks = gridDim.x >> 1;
    if (tid >= WG) tc::tmem_alloc(&S.tmem, 512);
    if (tid == WG) {
        tc::mbar_init(&S.bar[0], 1);
        tc::mbar_init(&S.bar[1], 1);
        tc::mbar_init_fence();
    }
    for (int i = tid; i < KW * C; i += WG + 32) S.w1[i / C][i % C] = __ldg(a.w + OFF_W1 + (i % C) * KW + i / C);
    if (tid < C) S.b1[tid] = __ldg(a.w + OFF_B1 + tid);
    for (int i = tid; i < 2 * PL / 16; i += WG + 32)
#pragma unroll
        for (int q = 0; q < 2; ++q)
            *reinterpret_cast<uint4*>(S.buf[q].a + 12 * PL + i * 16) =
                make_uint4(0x3c003c00u, 0x3c003c00u, 0x3c003c00u, 0x3c003c00u);
    tc::fence_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t d = S.tmem;
    const int places = (a.rows + R - 1) / R * H, sgroups = (a.steps + GROUP - 1) / GROUP, groups = places * sgroups;
    if (tid >= WG) {  // the issuing warp
        int n = 0;
        for (int gi = me; gi < groups; gi += blocks) {
            const int k0 = gi / places * GROUP, len = min(GROUP, a.steps - k0);
            for (int j = 0; j < len; ++j, ++n) {
                wg_take_over(n & 1);
                if (tc::elect()) {
                    tc::fence_after();
                    const uint64_t x = tc::smem_desc(tc::smem_u32(S.buf[n & 1].dz) + 32, 128, PL);
                    const uint64_t y = tc::smem_desc(tc::smem_u32(S.buf[n & 1].a), 128, PL);
                    constexpr uint32_t i96 = tc::instr_desc(128, 96, true, true), i112 = tc::instr_desc(128, 112, true, true);
#pragma unroll
                    for (int tap = 0; tap < KW; ++tap)
#pragma unroll
                        for (int r = 0; r < R; ++r)
#pragma unroll
                            for (int q = 0; q < U; q += 16)
                                tc::mma(d + tap_col(tap), tc::desc_at(x, (r * (U + 4) + q) * 16),
                                        tc::desc_at(y, (r * (U + 4) + tap + q) * 16), tap == KW / 2 ? i112 : i96,
                                        j > 0 || r > 0 || q > 0);
                    tc::commit(&S.bar[n & 1]);
                }
                __syncwarp();
            }
        }
        tc::fence_before();
        __syncthreads();
        tc::tmem_free(S.tmem, 512);
        return;
    }
    const int cell = tid & 255, half = tid >> 8, rl = cell / U, x = cell % U;  // this thread's cell, 16 channels
    const int slot = rl * (U + 4) + x + 2;
    const int halo = H > 1 ? 0 : (x < 2 ? U : (x >= U - 2 ? -U : 0));  // the copy a row's ends own
    const int lane_q = (tid >> 5) & 3, colq = tid >> 7;  // accumulator lanes' piece; 8 of the 32 input channels
    float acc[KW][8], gb = 0.f;
#pragma unroll
    for (int k = 0; k < KW; ++k)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[k][i] = 0.f;
    bool fail = false;
    uint32_t used = 0;
    bool pending = false;  // a group's sums are still in tensor memory
    // the layer's input (half of the channels) at cell xa of a row and step
    auto input = [&](int row, int k, int xa, float2(&v)[8]) {
        if (layer == 1) {
            const float* p = acts_tile(const_cast<float*>(a.acts), row, a.steps, k, 0, 16 * half, N) + xa;
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = act::gelu2(f2(__ldg(p + 2 * i * N), __ldg(p + (2 * i + 1) * N)));
        } else {
            const float* p = a.states + ((int64_t)row * a.steps + k) * N;
            float2 uu[KW];
#pragma unroll
            for (int q = 0; q < KW; ++q) uu[q] = f2s(__ldg(p + ((xa + q - 2 + N) & (N - 1))));
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float2 z = lds2(&S.b1[16 * half + 2 * i]);
#pragma unroll
                for (int q = 0; q < KW; ++q)
                    z = __ffma2_rn(*reinterpret_cast<const float2*>(&S.w1[q][16 * half + 2 * i]), uu[q], z);
                v[i] = act::gelu2(z);
            }
        }
    };
    // the lines of unit (gi, j), or of the next group's first, on their way to the L2: a 128-byte
    // line per thread (the first half dz's, the second the input's)
    auto prefetch = [&](int gi, int j) {
        if (j == min(GROUP, a.steps - gi / places * GROUP)) {
            gi += blocks;
            j = 0;
        }
        if (gi >= groups || (tid >= 256 && layer == 0)) return;
        constexpr int LINES = U / 32;  // of a row's cells in a channel
        const int e = tid & 255, line = e % LINES, ch = e / LINES % C, r = e / (LINES * C);
        const int place = gi % places, row = place / H * R + r, k = gi / places * GROUP + j;
        if (row >= a.rows) return;
        const float* p = tid < 256 ? acts_tile(const_cast<float*>(a.dz), row, a.steps, k, layer, ch, N)
                                   : acts_tile(const_cast<float*>(a.acts), row, a.steps, k, 0, ch, N);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + place % H * U + line * 32));
    };
    // a group's scales, by 64 threads: the channels' maxima over the unit's rows and the group's steps
    auto scales = [&](int gi, int par) {
        if (tid >= 64 || gi >= groups) return;
        const int op = tid >> 5, k0 = gi / places * GROUP, len = min(GROUP, a.steps - k0), first = gi % places / H * R;
        float m = 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int j = 0; j < GROUP; ++j)
                if (first + r < a.rows && j < len)
                    m = fmaxf(m, __ldg(a.mx + (((int64_t)(2 * op + layer) * a.rows + first + r) * a.steps + k0 + j) * C +
                                       (tid & 31)));
        const float s = tc::pow2_above(m), full = op == 0 ? 64.f : 256.f;
        S.up[par][op][tid & 31] = full / s;
        S.down[par][op][tid & 31] = s / full;
    };
    // the finished group's sums; `last`: the buffer of its last unit; par: its parity
    auto drain = [&](int last, int par) {
        if (!fail) fail = !tc::mbar_wait(&S.bar[last], (used >> last) & 1);
        tc::fence_after();
        // (every lane reads the same columns: loads under a branch cost a few hundred clocks each)
        const float order = lane_q == 0 ? 1.f : (lane_q == 1 ? tc::DOWN : tc::DOWN * tc::DOWN);  // of dz's piece
        const float fd = (fail ? __int_as_float(0x7fffffff) : S.down[par][0][tid & 31]) * order;
        const float4 fa0 = lds4(&S.down[par][1][8 * colq]), fa1 = lds4(&S.down[par][1][8 * colq + 4]);
        const float f[8] = {fd * fa0.x, fd * fa0.y, fd * fa0.z, fd * fa0.w, fd * fa1.x, fd * fa1.y, fd * fa1.z, fd * fa1.w};
        const uint32_t dl = d + ((uint32_t)(tid & 96) << 16) + 8 * colq;
        float ones[8];
        tc::tmem_ld8(d + ((uint32_t)(tid & 96) << 16) + ONES, ones);
#pragma unroll
        for (int k = 0; k < KW; ++k) {
            float q0[8], q1[8], q2[8];
            tc::tmem_ld8(dl + tap_col(k), q0);
            tc::tmem_ld8(dl + tap_col(k) + 32, q1);
            tc::tmem_ld8(dl + tap_col(k) + 64, q2);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i)
                acc[k][i] = fmaf(fmaf(fmaf(q2[i], tc::DOWN, q1[i]), tc::DOWN, q0[i]), f[i], acc[k][i]);
        }
        gb = fmaf(ones[0], fd, gb);
        tc::fence_before();
        wg_sync();  // read everywhere before the next group's products
    };
    int n = 0, par = 0;
    scales(me, 0);
    for (int gi = me; gi < groups; gi += blocks, par ^= 1) {
        wg_sync();  // this group's scales are there
        const int k0 = gi / places * GROUP, len = min(GROUP, a.steps - k0), place = gi % places;
        const int row = place / H * R + rl, x0 = place % H * U + x;
        const bool valid = row < a.rows;
        for (int j = 0; j < len; ++j, ++n) {
            const int buf = n & 1, k = k0 + j;
            if (n >= 2) {
                if (!fail) fail = !tc::mbar_wait(&S.bar[buf], (used >> buf) & 1);
                used ^= 1u << buf;
            }
            prefetch(gi, j + 1);
            float2 v[8];
            {
                const float* p = acts_tile(const_cast<float*>(a.dz), valid ? row : 0, a.steps, k, layer, 16 * half, N) + x0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    v[i].x = valid ? __ldg(p + 2 * i * N) : 0.f;
                    v[i].y = valid ? __ldg(p + (2 * i + 1) * N) : 0.f;
                }
            }
            store_half(S.buf[buf].dz, PL, v, S.up[par][0], slot, half);
            if (valid) {
                input(row, k, x0, v);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = f2s(0.f);
            }
            store_half(S.buf[buf].a, PL, v, S.up[par][1], slot, half);
            if (halo != 0) store_half(S.buf[buf].a, PL, v, S.up[par][1], slot + halo, half);
            if (H > 1 && x < 4) {  // half a row: the neighbours' cells on either side
                const int xh = x < 2 ? x - 2 : U + x - 2;
                input(row, k, (place % H * U + xh + N) & (N - 1), v);
                store_half(S.buf[buf].a, PL, v, S.up[par][1], xh + 2, half);
            }
            tc::fence_smem();
            tc::fence_before();
            if (j == 0 && pending) drain(buf ^ 1, par ^ 1);
            wg_hand_over(buf);
            if (j == 0) scales(gi + blocks, par ^ 1);  // (the group before this one is read: its place is free)
        }
        pending = true;
    }
    if (pending) drain((n - 1) & 1, par ^ 1);
    // the pieces of a lane's co added up, in the packed order [ci][co][k]
    float* s = reinterpret_cast<float*>(S.buf[0].dz);  // [3][32][161]; every product is done
    wg_sync();
    if (lane_q < 3) {
#pragma unroll
        for (int k = 0; k < KW; ++k)
#pragma unroll
            for (int i = 0; i < 8; ++i) s[(lane_q * 32 + (tid & 31)) * 161 + (8 * colq + i) * KW + k] = acc[k][i];
    }
    float* sb = s + 3 * 32 * 161;  // bias gradients, [3][32]
    if (lane_q < 3 && colq == 0) sb[lane_q * 32 + (tid & 31)] = gb;
    wg_sync();
    float* out = a.part + ((int64_t)layer * blocks + me) * HID;
    for (int i = tid; i < C * C * KW; i += WG) {
        const int ci = i / (C * KW), co = i / KW % C, k = i % KW;
        const float* p = s + co * 161 + ci * KW + k;
        out[i] = p[0] + (p[32 * 161] + p[64 * 161]);
    }
    if (tid < C) out[C * C * KW + tid] = sb[tid] + (sb[32 + tid] + sb[64 + tid]);
    tc::fence_before();
    __syncthreads();
}

// g[i] in the packed order from the blocks' partial sums, in FP64: 32 outputs x 32 slices per block.
// All of them are NaN when an adjoint block gave up on a wait: the weight gradients have read
// steps that it did not write.
__global__ void __launch_bounds__(1024) k_cnn_grad_sum(const float* __restrict__ edge, int edges,
                                                       const float* __restrict__ hid, int hids, float* __restrict__ g) {
    __shared__ double s[32][33];
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    const float* src = nullptr;
    int count = 0;
    int64_t stride = 0;
    if (i < OFF_B1) { src = edge + i; count = edges; }
    else if (i < OFF_W2) { src = edge + 2 * C * KW + i - OFF_B1; count = edges; }
    else if (i < OFF_W3) { src = hid + i - OFF_W2; count = hids; }
    else if (i < OFF_W4) { src = hid + (int64_t)hids * HID + i - OFF_W3; count = hids; }
    else if (i < OFF_B4) { src = edge + C * KW + i - OFF_W4; count = edges; }
    else if (i == OFF_B4) { src = edge + 2 * C * KW + C; count = edges; }
    stride = (i >= OFF_W2 && i < OFF_W4) ? HID : EDGE;
    double v = 0.0;
#pragma unroll 4
    for (int p = slice; p < count; p += 32) v += __ldg(src + p * stride);
    if (i == OFF_B4)
        for (int p = slice; p < count; p += 32) v += __ldg(src + 1 + p * stride);
    for (int p = slice; p < edges; p += 32)
        if (__ldg(edge + (int64_t)p * EDGE + 2 * C * KW + C + 2) != 0.f) v = __longlong_as_double(0x7ff8000000000000ll);
    s[slice][lane] = v;
    __syncthreads();
    if (threadIdx.x < 32 && i < W_FLOATS) {
        double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int q = 0; q < 32; ++q) t[q & 3] += s[q][lane];
        g[i] = (float)((t[0] + t[1]) + (t[2] + t[3]));
    }
}

struct BwdTcWork {
    int64_t dz, mx, edge, part, total;
    BwdTcWork(int64_t rows, int64_t n, int64_t steps) {
        int64_t at = 0;
        auto take = [&](int64_t f) {
            const int64_t r = at;
            at += (f + 31) / 32 * 32;
            return r;
        };
        dz = take(rows * steps * 2 * C * n);
        mx = take(4 * rows * steps * C);
        edge = take(rows * EDGE);
        part = take((int64_t)sm_count() * HID);
        total = at;
    }
};

template <int N>
int run_bwd_tc(const Args& a, AdjArgs c, float* g_weights, float* work, cudaStream_t st) {
    const BwdTcWork o(a.rows, N, a.steps);
    c.dz = work + o.dz;
    c.mx = work + o.mx;
    c.edge = work + o.edge;
    constexpr int R = TcCfg<N>::R;
    const int blocks = (a.rows + R - 1) / R;
    static_assert(sizeof(AdjSmem<N>) <= (N == 512 ? 227 : 113) * 1024, "shared memory");
    cudaFuncSetAttribute(k_cnn_adjoint<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AdjSmem<N>));
    k_cnn_adjoint<N><<<blocks, TcCfg<N>::T, sizeof(AdjSmem<N>), st>>>(a, c);
    int rc = check_launch("burgers_cnn_rollout_bwd (adjoint)");
    if (rc) return rc;
    const CnnWgradArgs wa{c.w, c.states, c.acts, c.dz, c.mx, work + o.part, a.rows, a.steps};
    static_assert(sizeof(CnnWgradSmem<N>) <= 227 * 1024, "shared memory");
    cudaFuncSetAttribute(k_cnn_wgrad<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CnnWgradSmem<N>));
    // as many blocks per layer as there are groups, at most half of the SMs
    const int64_t groups = (int64_t)((a.rows + WgCfg<N>::R - 1) / WgCfg<N>::R) * WgCfg<N>::H *
                           ((a.steps + GROUP - 1) / GROUP);
    const int most = sm_count() / 2 > 0 ? sm_count() / 2 : 1, per = groups < most ? (int)groups : most;
    k_cnn_wgrad<N><<<2 * per, WG + 32, sizeof(CnnWgradSmem<N>), st>>>(wa);
    rc = check_launch("burgers_cnn_rollout_bwd (weights)");
    if (rc) return rc;
    k_cnn_grad_sum<<<(W_FLOATS + 31) / 32, 1024, 0, st>>>(c.edge, blocks, wa.part, per, g_weights);
    return check_launch("burgers_cnn_rollout_bwd (sum)");
}

}  // namespace cnn
}  // namespace burgers
}  // namespace inc

using namespace inc;
using namespace inc::burgers;

extern "C" int64_t inc_burgers_cnn_rollout_bwd_states_work_size(int32_t rows, int32_t n, int32_t steps) {
    if (rows <= 0 || steps <= 0 || !(n == 64 || n == 128 || n == 256 || n == 512)) return -1;
    return cnn::BwdTcWork(rows, n, steps).total;
}

extern "C" int inc_burgers_cnn_rollout_bwd_states(const inc_burgers_desc* d, const float* weights, const float* states,
                                                  const float* corrections, const float* t_rows, double t0,
                                                  int32_t steps, const float* g_frames, const float* g_corrections,
                                                  const float* g_final, float* g_u0, float* g_weights,
                                                  const float* acts, float* work, void* stream) {
    Args a;
    int rc = fill_args(d, a);
    if (rc) return rc;
    if (!weights || !states || !corrections || !g_u0 || !g_weights || !acts || !work || steps <= 0) {
        set_error("cnn_rollout_bwd_states: bad arguments");
        return INC_E_INVALID;
    }
    a.t_rows = t_rows; a.t0 = (float)t0; a.steps = steps; a.g_frames = g_frames; a.g_final = g_final; a.g_u = g_u0;
    cnn::AdjArgs c{};
    c.w = weights; c.states = states; c.corr = corrections; c.g_corr = g_corrections; c.acts = acts;
    cudaStream_t st = as_stream(stream);
    switch (d->n) {
        case 64: return cnn::run_bwd_tc<64>(a, c, g_weights, work, st);
        case 128: return cnn::run_bwd_tc<128>(a, c, g_weights, work, st);
        case 256: return cnn::run_bwd_tc<256>(a, c, g_weights, work, st);
        case 512: return cnn::run_bwd_tc<512>(a, c, g_weights, work, st);
        default:
            set_error("cnn_rollout_bwd_states: n must be 64, 128, 256 or 512 (got %d)", d->n);
            return INC_E_UNSUPPORTED;
    }
}
