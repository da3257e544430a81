// Forward of the FNO corrector: lift, four layers and projection (FNO1D.forward,
// models/models_1d/fno.py:66-105 of tum-pbs/INC) on [batch][width][n] states.
//
//   * The lift fc0 is affine in (u, grid), so its modes come from the transforms of the
//     two input rows (k_fno_prep) and its values are formed where the first layer reads
//     them: the lifted state is never stored.
//   * A layer is three launches: the kept modes of its input (k_fno_modes), their mixing
//     (k_fno_mix) and k_fno_layer, which adds the 1x1 branch, the Fourier branch and
//     the bias and applies GELU.
//   * The projection fc1, GELU, fc2 is one launch that reads the state and writes [batch][n].
//
// What bounds it: reading and writing the state (11 passes of 67 MB at 512 x 64 x 512, 114 us
// at the measured copy rate) and, beside it, the splits and GELUs of every element and 13
// launches' starts: 359 us there, against 893 for batched FP32 matmuls, spectral-convolution
// kernels and elementwise passes on the same state.
#include "fno_tc.cuh"

namespace inc {
namespace fno {

struct ProjArgs {
    const float* x;      // [batch][W][N]
    const float* xmax;   // [tiles per row][batch]
    const unsigned char* fc1;  // image
    const float* wscale;
    const float* fc1_b;  // [128]
    const float* fc2_w;  // [128]
    const float* fc2_b;  // [1]
    float* y;            // [batch][N]
    int batch;
};

template <int W>
struct ProjSmem {
    alignas(128) unsigned char w[3 * 128 * W * 2];
    alignas(128) unsigned char x[3 * W * 128 * 2];
    alignas(16) float b1[128], w2[128];
    float y[2][128];
    uint64_t bar_images, bar;
    uint32_t tmem;
};

// y[p] = b2 + sum_j w2[j] gelu(b1[j] + sum_c w1[j][c] x[c][p]): the 128 hidden values of a
// point live in its tensor-memory lane and the registers of its two threads only.  Bound by
// those GELUs on the FMA pipe (16,384 per tile: 850 clocks per 16 columns with two CTAs) and
// the products (2,050 clocks per tile): 44 us at 512 x 64 x 512.
template <int W, int N>
__global__ void __launch_bounds__(THREADS, 2) k_fno_proj(ProjArgs a) {
    extern __shared__ __align__(128) unsigned char fno_smem[];
    ProjSmem<W>& S = *reinterpret_cast<ProjSmem<W>*>(fno_smem);
    constexpr int points = N < 128 ? N : 128, nq = N / points, C = W / 2;
    const int tid = threadIdx.x, half = (tid >> 7) & 1, t = tid & 127;
    const int tiles = a.batch * nq, step = gridDim.x;
    if (tid >= WORKERS) tc::tmem_alloc(&S.tmem, 256);
    if (tid == WORKERS) {
        tc::mbar_init(&S.bar_images, 1);
        tc::mbar_init(&S.bar, 1);
        tc::mbar_init_fence();
        tc::mbar_expect(&S.bar_images, sizeof(S.w));
        tc::bulk_load(S.w, a.fc1, sizeof(S.w), &S.bar_images);
    }
    for (int i = tid; i < 128; i += THREADS) {
        S.b1[i] = __ldg(a.fc1_b + i);
        S.w2[i] = __ldg(a.fc2_w + i);
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t d = S.tmem;
    if (tid >= WORKERS) {  // the issuing warp
        const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&S.bar_images, 0));
        for (int i = blockIdx.x; i < tiles; i += step) {
            take_over();
            if (ok && tc::elect()) {
                tc::fence_after();
                issue_product<128, W>(d, tc::smem_u32(S.x), W * 256, tc::smem_u32(S.w));
                tc::commit(&S.bar);
            }
            __syncwarp();
        }
        tc::fence_before();
        __syncthreads();
        tc::tmem_free(S.tmem, 256);
        return;
    }
    const bool on = points == 128 || t < points;
    const float ws = __ldg(a.wscale) * (1.f / 65536.f), b2 = __ldg(a.fc2_b);
    const uint32_t dl = d + ((uint32_t)(t & 96) << 16) + 64 * half;
    uint32_t phase = 0;
    bool fail = false;
    float2 v[C / 2];
    float vmax = 0.f;
    auto load_tile = [&](int i) {
        if (i >= tiles) return;
        load_channels<C, N>(a.x + ((int64_t)(i / nq) * W + half * C) * N + (i % nq) * points + t, on, v);
        vmax = __ldg(a.xmax + (int64_t)(i % nq) * a.batch + i / nq);
    };
    load_tile(blockIdx.x);
    int buf = 0;
    for (int i = blockIdx.x; i < tiles; i += step) {
        const float sx = tc::pow2_above(vmax), fs = sx * ws;
        store_point<W, C>(S.x, v, 256.f / sx, half * C, t);
        tc::fence_smem();
        tc::fence_before();
        hand_over();
        load_tile(i + step);
        if (!fail) fail = !tc::mbar_wait(&S.bar, phase);
        phase ^= 1;
        tc::fence_after();
        const float2 f = make_float2(fs, fs);
        float2 y0 = make_float2(0.f, 0.f), y1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 64; j += 16) {
            float x0[16], x1[16];
            tc::tmem_ld16(dl + j, x0);
            tc::tmem_ld16(dl + 128 + j, x1);
            tc::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
                const float4 bi = lds4(&S.b1[64 * half + j + e]), w2 = lds4(&S.w2[64 * half + j + e]);
                const float2 z0 = __ffma2_rn(join2(x0[e], x0[e + 1], x1[e], x1[e + 1]), f, make_float2(bi.x, bi.y));
                const float2 z1 =
                    __ffma2_rn(join2(x0[e + 2], x0[e + 3], x1[e + 2], x1[e + 3]), f, make_float2(bi.z, bi.w));
                y0 = __ffma2_rn(act::gelu2(z0), make_float2(w2.x, w2.y), y0);
                y1 = __ffma2_rn(act::gelu2(z1), make_float2(w2.z, w2.w), y1);
            }
        }
        tc::fence_before();
        y0 = __fadd2_rn(y0, y1);
        const float y = y0.x + y0.y;
        if (half == 1) S.y[buf][t] = y;
        worker_sync();  // (two buffers: the next tile's sums do not overwrite these)
        if (half == 0 && on)
            a.y[(int64_t)(i / nq) * N + (i % nq) * points + t] =
                fail ? __int_as_float(0x7fffffff) : (y + S.y[buf][t]) + b2;
        buf ^= 1;
    }
    tc::fence_before();
    __syncthreads();
}

template <int W, int N>
int launch_proj(const ProjArgs& a, cudaStream_t st) {
    const size_t smem = sizeof(ProjSmem<W>);
    static_assert(sizeof(ProjSmem<W>) <= 113 * 1024, "two CTAs per SM");
    cudaFuncSetAttribute(k_fno_proj<W, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int tiles = a.batch * (N < 128 ? 1 : N / 128), most = 2 * sm_count();
    k_fno_proj<W, N><<<tiles < most ? tiles : most, THREADS, smem, st>>>(a);
    return check_launch("fno projection");
}

template <int W>
int64_t work_floats(int64_t B, int64_t n, int64_t M, bool train) {
    const int64_t nq = n < 128 ? 1 : n / 128;
    return (int64_t)sizeof(Prep<W>) / 4 + 2 * (4 * M * W * W + 2 * M * B * W) + 4 * B +
           (train ? 0 : 2 * B * W * n + 4 * nq * B);
}

template <int W, bool TRAIN>
int forward_layer(const LayerArgs& a, int l, int n, cudaStream_t st) {
    return l == 0 ? run_layer<W, true, FWD, TRAIN>(a, n, st)
                  : (l < 3 ? run_layer<W, false, FWD, TRAIN>(a, n, st) : run_layer<W, false, LAST, TRAIN>(a, n, st));
}

template <int W>
int run_forward(const inc_fno_desc* d, const float* u, float* y, float* z, float* xm, float* tmax, float* work,
                cudaStream_t st) {
    const int B = d->rows, n = d->n, M = d->modes, nq = n < 128 ? 1 : n / 128;
    const int64_t state = (int64_t)B * W * n, modes = (int64_t)M * B * W;
    static_assert(sizeof(Prep<W>) % 16 == 0, "what follows the images stays aligned");
    Prep<W>* prep = reinterpret_cast<Prep<W>*>(work);
    float2* wt = reinterpret_cast<float2*>(prep + 1);          // [4][M][W][W]
    float2* part = wt + (int64_t)4 * M * W * W;                // [M][B][W]
    float2* mixed = part + modes;                              // [B][M][W]
    float* h = reinterpret_cast<float*>(mixed + modes);        // evaluation: two states,
    float* mmax = h;                                           // [4][B]
    if (!tmax) {                                               // [4][nq][B]
        tmax = h + 2 * state;
        mmax = tmax + 4 * nq * B;
    }
    PrepArgs pa{};
    for (int l = 0; l < 4; ++l) {
        pa.modes_w[l] = reinterpret_cast<const float2*>(d->modes_w[l]);
        pa.w[l] = d->w[l];
    }
    pa.fc1 = d->fc1_w;
    pa.u = u;
    pa.grid = d->grid;
    pa.fc0_w = d->fc0_w;
    pa.fc0_b = d->fc0_b;
    pa.wt = wt;
    pa.part = xm ? reinterpret_cast<float2*>(xm) : part;
    pa.zero = mmax;
    pa.grid_stride = d->grid_stride;
    pa.batch = B;
    pa.n = n;
    pa.modes = M;
    int rc = run_prep<W, false>(pa, prep, st);
    for (int l = 0; l < 4 && !rc; ++l) {
        const float* x = l == 0 ? u : (z ? z + (l - 1) * state : h + ((l - 1) & 1) * state);
        float2* im = xm ? reinterpret_cast<float2*>(xm) + l * modes : part;  // the input's modes
        if (l > 0) {
            const ModesArgs ma{x, tmax + (int64_t)(l - 1) * nq * B, prep->transform, im, B * W, B, M};
            rc = z ? run_modes<W, true>(ma, n, st) : run_modes<W, false>(ma, n, st);
            if (rc) break;
        }
        rc = run_mix<W>(im, wt + (int64_t)l * M * W * W, mixed, mmax + l * B, B, n, M, st);
        if (rc) break;
        LayerArgs a{};
        a.w = prep->w[l];
        a.inverse = prep->inverse[0];
        a.wscale = prep->scale + l;
        a.bias = d->b[l];
        a.mixed = mixed;
        a.mixed_max = mmax + l * B;
        a.tmax = tmax + (int64_t)l * nq * B;
        a.xmax = a.tmax - nq * B;  // (not read by the first layer)
        a.grid = d->grid;
        a.grid_stride = d->grid_stride;
        a.fc0_w = d->fc0_w;
        a.fc0_b = d->fc0_b;
        a.batch = B;
        a.modes = M;
        a.x = x;
        a.out = z ? z + l * state : h + (l & 1) * state;
        rc = z ? forward_layer<W, true>(a, l, n, st) : forward_layer<W, false>(a, l, n, st);
    }
    if (rc) return rc;
    const ProjArgs p{z ? z + 3 * state : h + state, tmax + 3 * nq * B, prep->fc1, prep->scale + 4, d->fc1_b, d->fc2_w,
                     d->fc2_b, y, B};
    switch (n) {
        case 64: return launch_proj<W, 64>(p, st);
        case 128: return launch_proj<W, 128>(p, st);
        case 256: return launch_proj<W, 256>(p, st);
        default: return launch_proj<W, 512>(p, st);
    }
}

int check_fno(const inc_fno_desc* d) {
    if (!d || d->rows <= 0 || !d->grid || !d->fc0_w || !d->fc0_b || !d->fc1_w || !d->fc1_b || !d->fc2_w || !d->fc2_b ||
        d->grid_stride < 0) {
        set_error("fno: bad arguments");
        return INC_E_INVALID;
    }
    for (int l = 0; l < 4; ++l)
        if (!d->modes_w[l] || !d->w[l] || !d->b[l] || (reinterpret_cast<uintptr_t>(d->modes_w[l]) & 7u) != 0) {
            set_error("fno: bad layer parameters");
            return INC_E_INVALID;
        }
    if (!supported(d->width, d->n, d->modes)) {
        set_error("fno: width 32 or 64, n 64, 128, 256 or 512, modes 1..%d (got %d, %d, %d)", KM, d->width, d->n,
                  d->modes);
        return INC_E_UNSUPPORTED;
    }
    return INC_OK;
}

}  // namespace fno
}  // namespace inc

using namespace inc;

extern "C" int64_t inc_fno_work_size(const inc_fno_desc* d, int32_t train) {
    if (!d || d->rows <= 0 || !fno::supported(d->width, d->n, d->modes)) return -1;
    return d->width == 64 ? fno::work_floats<64>(d->rows, d->n, d->modes, train != 0)
                          : fno::work_floats<32>(d->rows, d->n, d->modes, train != 0);
}

extern "C" int inc_fno_forward(const inc_fno_desc* d, const float* u, float* y, float* z, float* x_modes, float* tmax,
                               float* work, void* stream) {
    const int rc = fno::check_fno(d);
    if (rc) return rc;
    if (!u || !y || !work || (z != nullptr) != (x_modes != nullptr) || (z != nullptr) != (tmax != nullptr) ||
        (reinterpret_cast<uintptr_t>(work) & 15u) != 0 || (reinterpret_cast<uintptr_t>(x_modes) & 15u) != 0 ||
        (reinterpret_cast<uintptr_t>(z) & 15u) != 0) {  // (read four values at a time)
        set_error("fno_forward: bad arguments");
        return INC_E_INVALID;
    }
    cudaStream_t st = as_stream(stream);
    return d->width == 64 ? fno::run_forward<64>(d, u, y, z, x_modes, tmax, work, st)
                          : fno::run_forward<32>(d, u, y, z, x_modes, tmax, work, st);
}
