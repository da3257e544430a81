// Hybrid Burgers rollout with a periodic CNN corrector evaluated inside the
// kernel: per step s = CNN(u), then u = step(u, s) -- the per-step loop of
// trainer/trainer_1d.py:154-183 (simulate_rollout with correction "INC") for
// the convolutional corrector, forward only (evaluation rollouts).
//
// The network is the benchmark's PeriodicCNN1D: four Conv1d layers
// 1 -> 32 -> 32 -> 32 -> 1, kernel 5, circular padding 2, exact (erf) GELU
// between layers.  torch's Conv1d is a cross-correlation:
//   out[co][x] = b[co] + sum_ci sum_k W[co][ci][k] in[ci][(x + k - 2) mod N].
//
// Layout: one thread per cell, one row per CTA (two for rows of 64 cells).  The first
// layer (5 products per channel) and the last (5 partial sums per cell, exchanged once)
// run on the FP32 pipes from registers; the hidden layers are matrix products on the
// tensor cores (burgers_cnn_tc.cuh), with three-piece operands that keep every element's
// FP32 accuracy (tc.cuh).  A thread turns its cell's 32 activations into pieces with one
// power-of-two scale per row (the largest finite |a| of the row, one warp reduction and one
// barrier), one thread issues the products tile by tile, and each thread reads its
// cell's 32 sums back from tensor memory.
//
// What bounds a step: a chain.  With two rows of 256 cells on an SM a step takes about
// 28,700 clocks: the four tiles' products in turn (1,640 each, per layer), the split and its
// stores (about 2 x 2,300), reading and GELU (2 x 2,800), 2,500 in the first layer and 4,000
// in the solver's step.  256 x 256 x 32 steps: 467 us, against 1,154 with all four layers on
// the FP32 pipes.  With bf16 pieces, six products and one scale per weight matrix it was 426,
// and lost small operands' digits (tc.cuh).  Issuing a layer's products in two channel
// halves, the first beside the second's split, measured no faster (429 against 426).
#include "burgers_cnn_tc.cuh"

namespace inc {
namespace burgers {
namespace cnn {

template <int N>
struct FwdSmem {
    using Cfg = TcCfg<N>;
    alignas(128) unsigned char w[2][W_LAYER];          // W2, W3 in pieces
    union {
        alignas(128) unsigned char act[3 * 4 * Cfg::PLANE];  // activations in pieces
        struct {                                             // outside the hidden layers
            float part[Cfg::R][KW][N];  // the last layer's sums
            WideSmem<1, N> sh[Cfg::R];  // the solver's rows
        } o;
    };
    alignas(16) float w1[KW][C], b[3][C], w4[KW][C], ws[2][C];  // tap-major: channels contiguous
    float u[Cfg::R][N + 4];
    float red[2][Cfg::T / 32];
    uint64_t bar[Cfg::TILES];
    uint32_t tmem;
};

template <int N>
__global__ void __launch_bounds__(TcCfg<N>::T, N == 512 ? 1 : 2)
    k_cnn_rollout(Args a, const float* __restrict__ wts, float* __restrict__ corr, float* __restrict__ acts) {
    using Cfg = TcCfg<N>;
    constexpr int T = Cfg::T, R = Cfg::R;
    extern __shared__ __align__(128) unsigned char smraw[];
    FwdSmem<N>& S = *reinterpret_cast<FwdSmem<N>*>(smraw);
    float(*part)[KW][N] = S.o.part;
    const int t = threadIdx.x, rl = t / N, g = t % N;
    const int tile = N < 128 ? rl : t / 128;
    const bool issuer = t / 32 == T / 32 - (N < 128 ? 2 : 4);  // the warp that issues, one of the last tile's
    const int row = blockIdx.x * R + rl;
    const bool valid = row < a.rows;
    if (t < 32) tc::tmem_alloc(&S.tmem, Cfg::COLS);
    if (t == 0) {
#pragma unroll
        for (int i = 0; i < Cfg::TILES; ++i) tc::mbar_init(&S.bar[i], 1);
        tc::mbar_init_fence();
    }
    for (int i = t; i < KW * C; i += T) {
        S.w1[i / C][i % C] = __ldg(wts + OFF_W1 + (i % C) * KW + i / C);
        S.w4[i / C][i % C] = __ldg(wts + OFF_W4 + (i % C) * KW + i / C);
    }
    if (t < C) {
        S.b[0][t] = __ldg(wts + OFF_B1 + t);
        S.b[1][t] = __ldg(wts + OFF_B2 + t);
        S.b[2][t] = __ldg(wts + OFF_B3 + t);
    }
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const float s = stage_weights<T, false>(S.w[l], wts + (l == 0 ? OFF_W2 : OFF_W3));
        if (t < C) S.ws[l][t] = s;
    }
    const float b4 = __ldg(wts + OFF_B4);
    tc::fence_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    // this warp's lanes of its tile's accumulators
    const uint32_t acc = S.tmem + 128 * tile + ((uint32_t)(t & 96) << 16);
    Ctx<1> cx;
    make_ctx<1, N>(a, valid ? row : 0, g, true, cx);
    cx.has_s = true;
    float u[1], cmp[1] = {0.f};  // cmp: compensation carried from step to step (see advance)
    u[0] = valid ? __ldg(a.u + (int64_t)row * N + g) : 0.f;
    int parity = 0;
    uint32_t phase = 0;
    bool fail = false;  // a wait for the tensor cores ran out: the outputs turn to NaN
    const int nseg = a.ckpt_every > 0 ? (a.steps + a.ckpt_every - 1) / a.ckpt_every : 0;
    for (int k = 0; k < a.steps; ++k) {
        if (a.ckpts && valid && k % a.ckpt_every == 0)
            a.ckpts[((int64_t)row * nseg + k / a.ckpt_every) * N + g] = u[0];
        S.u[rl][g + 2] = u[0];
        if (g < 2) S.u[rl][N + 2 + g] = u[0];
        if (g >= N - 2) S.u[rl][g - N + 2] = u[0];
        __syncthreads();
        float v[C];
        {  // layer 1
            float2 uu[KW];
#pragma unroll
            for (int q = 0; q < KW; ++q) uu[q] = f2s(S.u[rl][g + q]);
#pragma unroll
            for (int c = 0; c < C; c += 4) {
                const float4 b = lds4(&S.b[0][c]);
                float2 z0 = f2(b.x, b.y), z1 = f2(b.z, b.w);
#pragma unroll
                for (int q = 0; q < KW; ++q) {
                    const float4 w = lds4(&S.w1[q][c]);
                    z0 = __ffma2_rn(f2(w.x, w.y), uu[q], z0);
                    z1 = __ffma2_rn(f2(w.z, w.w), uu[q], z1);
                }
                z0 = act::gelu2(z0);
                z1 = act::gelu2(z1);
                v[c] = z0.x; v[c + 1] = z0.y; v[c + 2] = z1.x; v[c + 3] = z1.y;
            }
        }
#pragma unroll 1
        for (int l = 0; l < 2; ++l) {  // layers 2 and 3
            const float m = row_absmax<N>(v, S.red[l], fail, rl);
            if (fail) break;
            const float s = tc::pow2_above(m);
            store_cell<N>(S.act, v, 256.f / s, rl, g);
            tc::fence_smem();
            tc::fence_before();
            __syncthreads();
            if (issuer && tc::elect()) {  // tile by tile: the first's sums are read while the last's products run
                tc::fence_after();
#pragma unroll
                for (int q = 0; q < Cfg::TILES; ++q) {
                    issue_layer<N>(S.tmem + 128 * q, S.act, S.w[l], q);
                    tc::commit(&S.bar[q]);
                }
            }
            fail = !tc::mbar_wait(&S.bar[tile], phase);
            phase ^= 1;
            tc::fence_after();
            const float f = s * (1.f / 256.f);
#pragma unroll
            for (int c = 0; c < C; c += 8) {
                float2 z[4];
                read_layer8(acc, c, f, S.ws[l], S.b[l + 1], z);
                if (acts && valid) {
                    float* p = acts_tile(acts, row, a.steps, k, l, c, N) + g;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        p[(int64_t)(2 * i) * N] = z[i].x;
                        p[(int64_t)(2 * i + 1) * N] = z[i].y;
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 y = act::gelu2(z[i]);
                    v[c + 2 * i] = y.x;
                    v[c + 2 * i + 1] = y.y;
                }
            }
            tc::fence_before();  // the accumulators are read before the next layer overwrites them
        }
        if (__syncthreads_or(fail)) {  // (also: every tile's products have read the activations)
            fail = true;
            break;
        }
        {  // layer 4: this cell's share of its five neighbours' sums
            float2 q[KW];
#pragma unroll
            for (int i = 0; i < KW; ++i) q[i] = f2s(0.f);
#pragma unroll
            for (int c = 0; c < C; c += 4) {
#pragma unroll
                for (int i = 0; i < KW; ++i) {
                    const float4 w = lds4(&S.w4[i][c]);
                    q[i] = __ffma2_rn(f2(w.x, w.y), f2(v[c], v[c + 1]), q[i]);
                    q[i] = __ffma2_rn(f2(w.z, w.w), f2(v[c + 2], v[c + 3]), q[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < KW; ++i) part[rl][i][g] = q[i].x + q[i].y;
        }
        __syncthreads();
        float s = b4;
#pragma unroll
        for (int i = 0; i < KW; ++i) s += part[rl][i][(g + i - 2 + N) & (N - 1)];
        cx.s[0] = s;
        const int64_t at = ((int64_t)row * a.steps + k) * N + g;
        if (corr && valid) corr[at] = s;
        // the stage's first barrier also orders these reads of the sums before the next step's writes
        advance_wide<1, N>(a, cx, u, cmp, cx.t + k * cx.dt, S.o.sh[rl], parity, g);
        if (a.frames && valid) a.frames[at] = u[0];
    }
    if (fail && valid) {
        const float nan = __int_as_float(0x7fffffff);
        u[0] = nan;
        for (int k = 0; k < a.steps; ++k) {
            const int64_t at = ((int64_t)row * a.steps + k) * N + g;
            if (corr) corr[at] = nan;
            if (a.frames) a.frames[at] = nan;
        }
    }
    if (a.out && valid) a.out[(int64_t)row * N + g] = u[0];
    tc::fence_before();
    __syncthreads();
    if (t < 32) tc::tmem_free(S.tmem, Cfg::COLS);
}

template <int N>
int launch(const Args& a, const float* w, float* corr, float* acts, cudaStream_t st) {
    constexpr int R = TcCfg<N>::R;
    const size_t smem = sizeof(FwdSmem<N>);
    static_assert(sizeof(FwdSmem<N>) <= (N == 512 ? 227 : 113) * 1024, "shared memory");
    cudaFuncSetAttribute(k_cnn_rollout<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_cnn_rollout<N><<<(a.rows + R - 1) / R, TcCfg<N>::T, smem, st>>>(a, w, corr, acts);
    return check_launch("burgers_cnn_rollout");
}

}  // namespace cnn
}  // namespace burgers
}  // namespace inc

using namespace inc;
using namespace inc::burgers;

static int cnn_rollout(const inc_burgers_desc* d, const float* weights, const float* u0, const float* t_rows,
                       double t0, int32_t steps, float* frames, float* corrections, float* u_final,
                       int32_t ckpt_every, float* ckpts, float* acts, void* stream) {
    Args a;
    int rc = fill_args(d, a);
    if (rc) return rc;
    if (!weights || !u0 || steps < 0) { set_error("cnn_rollout: bad arguments"); return INC_E_INVALID; }
    if (ckpts && ckpt_every <= 0) { set_error("cnn_rollout: ckpt_every must be positive with ckpts"); return INC_E_INVALID; }
    a.ckpt_every = ckpt_every;
    a.ckpts = ckpts;
    if (((reinterpret_cast<uintptr_t>(weights)) & 15u) != 0) {
        set_error("cnn_rollout: weights must be 16-byte aligned");
        return INC_E_INVALID;
    }
    if (acts && ((reinterpret_cast<uintptr_t>(acts)) & 15u) != 0) {
        set_error("cnn_rollout: acts must be 16-byte aligned");
        return INC_E_INVALID;
    }
    a.u = u0; a.s = nullptr; a.t_rows = t_rows; a.t0 = (float)t0; a.steps = steps; a.frames = frames; a.out = u_final;
    cudaStream_t st = as_stream(stream);
    switch (d->n) {
        case 64: return cnn::launch<64>(a, weights, corrections, acts, st);
        case 128: return cnn::launch<128>(a, weights, corrections, acts, st);
        case 256: return cnn::launch<256>(a, weights, corrections, acts, st);
        case 512: return cnn::launch<512>(a, weights, corrections, acts, st);
        default:
            set_error("cnn_rollout: n must be 64, 128, 256 or 512 (got %d)", d->n);
            return INC_E_UNSUPPORTED;
    }
}

extern "C" int inc_burgers_cnn_rollout(const inc_burgers_desc* d, const float* weights, const float* u0,
                                       const float* t_rows, double t0, int32_t steps, float* frames,
                                       float* corrections, float* u_final, int32_t ckpt_every, float* ckpts,
                                       void* stream) {
    return cnn_rollout(d, weights, u0, t_rows, t0, steps, frames, corrections, u_final, ckpt_every, ckpts, nullptr,
                       stream);
}

extern "C" int inc_burgers_cnn_rollout_acts(const inc_burgers_desc* d, const float* weights, const float* u0,
                                            const float* t_rows, double t0, int32_t steps, float* frames,
                                            float* corrections, float* u_final, int32_t ckpt_every, float* ckpts,
                                            float* acts, void* stream) {
    if (!acts) { set_error("cnn_rollout_acts: acts must not be NULL"); return INC_E_INVALID; }
    return cnn_rollout(d, weights, u0, t_rows, t0, steps, frames, corrections, u_final, ckpt_every, ckpts, acts,
                       stream);
}
