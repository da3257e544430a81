// The FNO corrector (FNO1D, models/models_1d/fno.py:39-105 of tum-pbs/INC) on the
// tensor cores: the parts shared by its forward (fno_fwd.cu) and backward (fno_bwd.cu).
//
// The network's contractions are products over channels (the layers' 1x1 branches, the
// projection) and, for the Fourier branch with its few kept modes, products with a
// [2 modes x points] table of cosines and sines: a transform to the modes and back is a
// thin matrix product beside the 1x1 branch's.  All of them are three-piece tcgen05
// products that keep FP32's accuracy (tc.cuh).  Two CTAs of an SM with two tiles each in
// flight leave a tile 2 W accumulator columns, so the orders of the pieces' products from 1 up
// share W of them (issue_stage).
//
// A tile of k_fno_layer is 128 points (64 for rows of 64) of one trajectory with all W
// channels.  The [W][n] state puts a point's channels n apart: two threads per point
// (half of the channels each) load them coalesced across the warp, hold them in registers
// (split and GELU without exchange) and read their outputs back from the point's
// tensor-memory lane.  The split's scale is the tile's max, recorded by the launch that
// wrote the state.  A CTA keeps one position of the row and walks over the trajectories;
// its table and weights, prepared as shared-memory images by one launch per call, arrive
// by bulk copies and stay.  8 warps do the arithmetic (in the forward a ninth only issues
// products, see layer_threads); the products of the next tile run while this one's results
// are read, and two CTAs share an SM.
//
// What bounds a layer: the loads' latency at the start of a launch (4,000 to 12,000 clocks
// until the first tile and the images are there), then the splits and GELUs beside the
// loads, and the products (2,110 clocks per tile at W = 64).  512 x 64 x 512: 47.5 us for 134 MB
// read and written (20.8 us at the copy rate; 43.5 with six products of bf16 pieces, which
// lost small operands' digits); a batched FP32 matmul, a spectral convolution and a GELU pass
// took about 150.  Programmatic launch overlap, an L2 prefetch of later tiles and 16 warps a CTA
// measured no faster.
//
// The modes of a state are a launch of their own (k_fno_modes) with the points as the
// contraction: taking them in the layer's epilogue instead (a second split and product per
// tile) made a layer of 512 x 64 x 512 75 us against 39 us without.
#pragma once
#include "gelu.cuh"
#include "tc.cuh"

namespace inc {
namespace fno {

constexpr int KM = 16;             // modes of the tables (a network with fewer has zero rows)
constexpr int WORKERS = 256;       // 128 points x 2 channel halves
constexpr int THREADS = WORKERS + 32;

// Loads of states: read once, so they leave the L1 (a few KB beside the tiles) alone
INC_DEV float ldg_na(const float* p) {
    float v;
    asm("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
INC_DEV float4 ldg_na4(const float4* p) {
    float4 v;
    asm("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
INC_DEV float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Barriers: the workers' own; and the hand-overs to the issuing warp, on which the workers
// only arrive.  A worker must not reach one hand-over barrier again before the issuing warp
// has left it: between two hand-overs on it lies a wait for products issued after the first
// (with two tile buffers in flight, each has a barrier of its own).
template <int NT = WORKERS>
INC_DEV void worker_sync() { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); }
template <int NT = WORKERS>
INC_DEV void hand_over(int buf = 0) { asm volatile("bar.arrive %0, %1;" ::"r"(2 + buf), "n"(NT + 32) : "memory"); }
template <int NT = WORKERS>
INC_DEV void take_over(int buf = 0) { asm volatile("bar.sync %0, %1;" ::"r"(2 + buf), "n"(NT + 32) : "memory"); }

// max over a warp of a non-negative value
INC_DEV float warp_max(float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v))); }

// One period of (cos, sin)(2 pi i / n), rounded from FP64 (two entries a thread; the
// tables below are look-ups in it)
INC_DEV void stage_period(float2* cs, int n) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double s, c;
        sincospi(2.0 * i / n, &s, &c);
        cs[i] = make_float2((float)c, (float)s);
    }
}

// max |w| of an array over the CTA (two barriers), as its scale
INC_DEV float cta_scale(const float* __restrict__ w, int count, float* red) {
    float m = 0.f;
#pragma unroll 4
    for (int i = threadIdx.x; i < count; i += blockDim.x) m = fmaxf(m, fabsf(__ldg(w + i)));
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    for (int i = 0; i < blockDim.x / 32; ++i) m = fmaxf(m, red[i]);
    __syncthreads();
    return tc::pow2_above(m);
}

// Weights [ROWS][K] (element (r, k) = w[r * K + k], or w[k * ROWS + r] with TRANS) as the
// stacked pieces [3 ROWS][K] of a K-major operand.
template <int ROWS, int K, bool TRANS>
INC_DEV void stage_matrix(unsigned char* dst, const float* __restrict__ w, float scale) {
    const float inv = 256.f / scale;
    for (int i = threadIdx.x; i < ROWS * (K / 8); i += blockDim.x) {
        const int r = i % ROWS, k8 = i / ROWS;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __ldg(w + (TRANS ? (8 * k8 + j) * ROWS + r : r * K + 8 * k8 + j));
        uint4 q[3];
        tc::split8(v, inv, q[0], q[1], q[2]);
#pragma unroll
        for (int p = 0; p < 3; ++p)
            *reinterpret_cast<uint4*>(dst + k8 * (3 * ROWS * 16) + (p * ROWS + r) * 16) = q[p];
    }
}

// Transform table as a K-major operand of 96 rows (piece, 2 k + {re, im}) with the points as
// the contraction: X[k] = sum_p x[p] (cos - i sin).  Planes of 8 points.  Scaled to 128 instead
// of 256: a state that hardly varies adds 512 full-scale terms into its k = 0 sum, which
// have to stay below 2^24 (tc.cuh).
constexpr int F_PLANE = 96 * 16;
constexpr float F_SCALE = 128.f;
INC_DEV void stage_transform(unsigned char* ft, const float2* cs, int n, int modes, int first, int count) {
    for (int i = first + threadIdx.x; i < first + count; i += blockDim.x) {
        const int k = i % KM, p8 = i / KM;
        float c[8], s[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float2 e = cs[(k * (8 * p8 + j)) & (n - 1)];
            c[j] = k < modes ? e.x : 0.f;
            s[j] = k < modes ? -e.y : 0.f;
        }
        uint4 q[3], r[3];
        tc::split8(c, F_SCALE, q[0], q[1], q[2]);
        tc::split8(s, F_SCALE, r[0], r[1], r[2]);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            unsigned char* d = ft + p8 * F_PLANE + (32 * p + 2 * k) * 16;
            *reinterpret_cast<uint4*>(d) = q[p];
            *reinterpret_cast<uint4*>(d + 16) = r[p];
        }
    }
}

// Inverse table of the same points: [128 points][32] K-major pieces, y[p] = sum_k g[2k] Re F
// + g[2k + 1] Im F with g = (1, 0) at k = 0 and (2 cos, -2 sin) above.  Scale 2.
INC_DEV void stage_inverse(unsigned char* gt, const float2* cs, int p0, int n, int modes) {
    for (int i = threadIdx.x; i < 128 * 4; i += blockDim.x) {
        const int p = i % 128, k4 = i / 128;
        float v[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = 4 * k4 + j;
            const float2 e = cs[(k * (p0 + p)) & (n - 1)];
            v[2 * j] = k >= modes ? 0.f : (k == 0 ? 1.f : 2.f * e.x);
            v[2 * j + 1] = (k >= modes || k == 0) ? 0.f : -2.f * e.y;
        }
        uint4 q[3];
        tc::split8(v, 128.f, q[0], q[1], q[2]);
#pragma unroll
        for (int pc = 0; pc < 3; ++pc) *reinterpret_cast<uint4*>(gt + (pc * 4 + k4) * 2048 + p * 16) = q[pc];
    }
}
constexpr int G_BYTES = 3 * 4 * 2048;

// What one preparation launch leaves in global memory for the call's other launches
// (floats; every image is the bytes of its shared-memory counterpart):
template <int W>
struct Prep {
    float scale[8];                        // of w[0..3], fc1
    unsigned char w[4][3 * W * W * 2];     // the 1x1 branches (transposed for the adjoint)
    unsigned char fc1[3 * 128 * W * 2];
    unsigned char inverse[4][G_BYTES];     // per position of the row
    unsigned char transform[64 * F_PLANE]; // the whole row (n / 8 planes)
};

// C values (channels c0 .. c0 + C - 1 of point t) as pieces in a [128 points][W] tile:
// piece-major planes of 8 channels.
template <int W, int C>
INC_DEV void store_point(unsigned char* x, const float2 (&v)[C / 2], float inv, int c0, int t) {
#pragma unroll
    for (int c8 = 0; c8 < C / 8; ++c8) {
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) tc::split2(v[4 * c8 + j], make_float2(inv, inv), h[j], m[j], l[j]);
        unsigned char* d = x + (c0 / 8 + c8) * 2048 + t * 16;
        *reinterpret_cast<uint4*>(d) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(d + (W / 8) * 2048) = make_uint4(m[0], m[1], m[2], m[3]);
        *reinterpret_cast<uint4*>(d + 2 * (W / 8) * 2048) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}
// A [128 x K] B[N x K]^T, one stage of it.  A: pieces of a point tile (planes of 2048 bytes,
// pieces a_piece apart); B: stacked pieces [3 N][K].  The stages 3, 2, 1 leave order 0 in
// columns d .. d + N - 1 and, in d + N .. d + 2N - 1, order 1 + 2^-14 (order 2 + 2^-14 order 3).  FIRST: the first
// product of the accumulators (several may add up, stage by stage).  One thread (tc::elect).
template <int N, int K, int STAGE, bool FIRST>
INC_DEV void issue_stage(uint32_t d, uint32_t a, uint32_t a_piece, uint32_t b) {
    constexpr uint32_t plane_b = 3 * N * 16;
    constexpr uint32_t i2 = tc::instr_desc(128, 2 * N), i1 = tc::instr_desc(128, N);
    const uint64_t ad = tc::smem_desc(a, 2048, 128), bd = tc::smem_desc(b, plane_b, 128);
#pragma unroll
    for (int k = 0; k < K / 16; ++k) {
        const bool first = FIRST && k == 0;
        const uint64_t a0 = tc::desc_at(ad, 2 * k * 2048), b0 = tc::desc_at(bd, 2 * k * plane_b);
        const uint64_t a1 = tc::desc_at(a0, a_piece), a2 = tc::desc_at(a0, 2 * a_piece);
        const uint64_t b1 = tc::desc_at(b0, N * 16), b2 = tc::desc_at(b0, 2 * N * 16);
        if constexpr (STAGE == 3) {
            tc::mma(d + N, a1, b2, i1, !first);  // mid.lo
            tc::mma(d + N, a2, b1, i1, true);    // lo.mid
        } else if constexpr (STAGE == 2) {
            if (first) tc::mma_scaled(d + N, a0, b2, i1);  // hi.lo
            else tc::mma(d + N, a0, b2, i1, true);
            tc::mma(d + N, a1, b1, i1, true);  // mid.mid
            tc::mma(d + N, a2, b0, i1, true);  // lo.hi
        } else {
            if (first) {  // hi.hi, hi.mid
                tc::mma(d, a0, b0, i1, false);
                tc::mma_scaled(d + N, a0, b1, i1);
            } else {
                tc::mma(d, a0, b0, i2, true);
            }
            tc::mma(d + N, a1, b0, i1, true);  // mid.hi
        }
    }
}
template <int N, int K>
INC_DEV void issue_product(uint32_t d, uint32_t a, uint32_t a_piece, uint32_t b) {
    issue_stage<N, K, 3, true>(d, a, a_piece, b);
    issue_stage<N, K, 2, true>(d, a, a_piece, b);
    issue_stage<N, K, 1, true>(d, a, a_piece, b);
}
// the two accumulators of such a product added up
INC_DEV float2 join2(float x0, float y0, float x1, float y1) {
    return __ffma2_rn(make_float2(x1, y1), make_float2(tc::DOWN, tc::DOWN), make_float2(x0, y0));
}

// sums over the warp of each of C values: lane l is left with that of channel l / (32 / C)
template <int C>
INC_DEV float warp_sums(float (&v)[C], int lane) {
    static_assert(C == 16 || C == 32, "channels per thread");
    int o = 16;
#pragma unroll
    for (int h = C / 2; h > 0; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int i = 32 / C / 2; i > 0; i >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], i);
    return v[0];
}

// this thread's C channels of its point; base = &state[b][c0][p]
template <int C, int N>
INC_DEV void load_channels(const float* __restrict__ base, bool live, float2 (&v)[C / 2]) {
#pragma unroll
    for (int c = 0; c < C; c += 2) {
        v[c / 2].x = live ? ldg_na(base + c * N) : 0.f;
        v[c / 2].y = live ? ldg_na(base + (c + 1) * N) : 0.f;
    }
}

// One FNO layer on the point tiles (forward and input adjoint):
//   z[o][p] = sum_c w[o][c] x[c][p] + sum_k (table)[p][k] mixed[k][o] + bias[o].
// MODE:
//   FWD     z stored, or gelu(z) in an evaluation;
//   LAST    z stored (the last layer: no GELU follows);
//   BWD     z gelu'(zprev) stored (x = dL/dz of this layer, w transposed, zprev the layer
//           below's z);
//   BWD0    the first layer's adjoint: nothing stored but g_u and the sums below.
// LIFT: x[c] is the lift of (u, grid); else it is read, in training's forward through GELU
// (its record holds the sums before it).  TRAIN is a parameter of the template: a test of it
// among the elements keeps their arithmetic from overlapping.
// The two products share one scale (the larger of theirs), so they accumulate together.
enum { FWD, LAST, BWD, BWD0 };

struct LayerArgs {
    const float* x;         // [batch][W][N]; LIFT: u [batch][N]
    const float* xmax;      // [tiles per row][batch]: max |x| of the tiles (a bound, after GELU)
    const unsigned char* w;        // images (Prep)
    const unsigned char* inverse;  // [tiles per row]
    const float* wscale;
    const float* bias;      // [W] (forward)
    const float2* mixed;    // [batch][modes][W]
    const float* mixed_max; // [batch]: max |mixed|
    const float* zprev;     // BWD
    float* out;             // [batch][W][N]
    float* tmax;            // [tiles per row][batch]: max |.| of the stored tile, after the GELU that follows
    const float* u;         // LIFT, BWD0: [batch][N]
    const float* grid;      // [batch][N] (row stride grid_stride)
    const float* fc0_w;     // [W][2]
    const float* fc0_b;     // [W]
    float* g_u;             // BWD0: [batch][N]
    float* sums;            // BWD0: [blocks][6][W]
    int64_t grid_stride;
    int batch, modes;
};

template <int W>
struct LayerSmem {
    alignas(128) unsigned char w[3 * W * W * 2];
    alignas(128) unsigned char gt[G_BYTES];
    alignas(128) unsigned char x[3 * W * 128 * 2];
    alignas(128) unsigned char m[3 * W * 32 * 2];
    alignas(16) float bias[W];
    alignas(16) float lift[3][W];
    alignas(16) float gu[128];
    float lift_max[3];
    alignas(16) float red[2][WORKERS / 32];
    uint64_t bar_images, bar_layer;
    uint32_t tmem;
};

// Who issues: in the forward a ninth warp; in the adjoint the last of the eight, which leaves a
// thread 128 registers in place of 96 and with them room to load zprev a tile ahead (256 x 64 x
// 512: 33.2 -> 29.6 us, the first layer's 30.1 -> 24.8; the forward with the lift 18.0 -> 20.3 that
// way, the others equal; 32.0 and 26.2 for the adjoints since the operands have fp16 pieces).
constexpr int layer_threads(int mode) { return mode >= BWD ? WORKERS : THREADS; }

template <int W, int N, bool LIFT, int MODE, bool TRAIN>
__global__ void __launch_bounds__(layer_threads(MODE), 2) k_fno_layer(LayerArgs a) {
    extern __shared__ __align__(128) unsigned char fno_smem[];
    LayerSmem<W>& S = *reinterpret_cast<LayerSmem<W>*>(fno_smem);
    constexpr bool kBwd = MODE >= BWD, kInGelu = TRAIN && !LIFT && !kBwd, kStoreGelu = !TRAIN && MODE == FWD;
    constexpr int points = N < 128 ? N : 128, nq = N / points, C = W / 2;
    constexpr int COLS = 4 * W;  // two tiles' accumulators
    const int tid = threadIdx.x, half = (tid >> 7) & 1, t = tid & 127, c0 = half * C;
    const int q = blockIdx.x % nq, p = q * points + t;
    const int step = gridDim.x / nq;  // CTAs per row position
    const int b0 = blockIdx.x / nq;
    if (tid < 32) tc::tmem_alloc(&S.tmem, COLS);
    if (tid == 0) {
        tc::mbar_init(&S.bar_images, 1);
        tc::mbar_init(&S.bar_layer, 1);
        tc::mbar_init_fence();
        tc::mbar_expect(&S.bar_images, sizeof(S.w) + G_BYTES);
        tc::bulk_load(S.w, a.w, sizeof(S.w), &S.bar_images);
        tc::bulk_load(S.gt, a.inverse + (int64_t)q * G_BYTES, G_BYTES, &S.bar_images);
    }
    for (int i = tid; i < W; i += layer_threads(MODE)) {
        S.bias[i] = kBwd ? 0.f : __ldg(a.bias + i);
        if (LIFT || MODE == BWD0) {
            S.lift[0][i] = __ldg(a.fc0_w + 2 * i);
            S.lift[1][i] = __ldg(a.fc0_w + 2 * i + 1);
            S.lift[2][i] = __ldg(a.fc0_b + i);
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t d = S.tmem;
    auto products = [&](int buf) {  // one thread
        tc::fence_after();
        const uint32_t dt = d + 2 * W * buf, x = tc::smem_u32(S.x), w = tc::smem_u32(S.w);
        const uint32_t gt = tc::smem_u32(S.gt), m = tc::smem_u32(S.m);
        issue_stage<W, W, 3, true>(dt, x, W * 256, w);
        issue_stage<W, 32, 3, false>(dt, gt, 8192, m);
        issue_stage<W, W, 2, true>(dt, x, W * 256, w);
        issue_stage<W, 32, 2, false>(dt, gt, 8192, m);
        issue_stage<W, W, 1, true>(dt, x, W * 256, w);
        issue_stage<W, 32, 1, false>(dt, gt, 8192, m);
        tc::commit(&S.bar_layer);
    };
    if (!kBwd && tid >= WORKERS) {  // ---- the issuing warp
        // (images that did not arrive: nothing is issued, and the workers' waits run out)
        const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&S.bar_images, 0));
        int buf = 0;
        for (int b = b0; b < a.batch; b += step) {
            take_over();
            if (ok && tc::elect()) products(buf);
            __syncwarp();
            buf ^= 1;
        }
        tc::fence_before();
        __syncthreads();
        return;
    }
    bool ok = true, waited = false;
    auto issue = [&](int buf) {  // the staged tile is ready
        if constexpr (!kBwd) {
            hand_over();
        } else if (tid < WORKERS - 32) {
            hand_over<WORKERS - 32>();
        } else {
            if (!waited) ok = __all_sync(0xffffffffu, tc::mbar_wait(&S.bar_images, 0));
            waited = true;
            take_over<WORKERS - 32>();
            if (ok && tc::elect()) products(buf);
            __syncwarp();
        }
    };
    // ---- the workers
    const bool on = points == 128 || t < points;  // (rows of 64 cells use half of a tile)
    const float ws = __ldg(a.wscale);
    if (LIFT) {
        if (tid < 3) {
            float m = 0.f;
            for (int i = 0; i < W; ++i) m = fmaxf(m, fabsf(S.lift[tid][i]));
            S.lift_max[tid] = m;
        }
        worker_sync();
    }
    const uint32_t dl = d + ((uint32_t)(t & 96) << 16) + c0;
    uint32_t phase = 0;
    bool fail = false;  // a wait for the tensor cores ran out: the outputs turn to NaN
    float sum[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // a tile on its way in: values (LIFT: u and grid at the point), mixed modes, magnitudes
    float2 v[C / 2];
    float lu = 0.f, lx = 0.f, vmax = 0.f, mmax = 0.f, mv[8];
    auto load_tile = [&](int b) {
        if (b >= a.batch) return;
        if constexpr (LIFT) {
            lu = on ? __ldg(a.x + (int64_t)b * N + p) : 0.f;
            lx = on ? __ldg(a.grid + (int64_t)b * a.grid_stride + p) : 0.f;
        } else {
            load_channels<C, N>(a.x + ((int64_t)b * W + c0) * N + p, on, v);
            vmax = __ldg(a.xmax + (int64_t)q * a.batch + b);
        }
        mmax = __ldg(a.mixed_max + b);
        if (tid < 4 * W) {  // channel tid / 4, four modes
            const int k0 = (tid % 4) * 4;
            const float2* mp = a.mixed + ((int64_t)b * a.modes + k0) * W + tid / 4;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 e = k0 + i < a.modes ? __ldg(mp + i * W) : make_float2(0.f, 0.f);
                mv[2 * i] = e.x;
                mv[2 * i + 1] = e.y;
            }
        }
    };
    // the loaded tile into shared memory; returns the products' scale
    auto stage_tile = [&]() -> float {
        if constexpr (LIFT) {
            // the tile's scale from the max of a bound of |lift| over its points
            const float m = warp_max(fmaf(S.lift_max[0], fabsf(lu), fmaf(S.lift_max[1], fabsf(lx), S.lift_max[2])));
            if ((tid & 31) == 0) S.red[1][tid >> 5] = m;
            worker_sync();
            const float4 r = lds4(S.red[1]);
            vmax = fmaxf(fmaxf(r.x, r.y), fmaxf(r.z, r.w));
#pragma unroll
            for (int c = 0; c < C; c += 4) {
                const float4 w0 = lds4(&S.lift[0][c0 + c]), w1 = lds4(&S.lift[1][c0 + c]), bb = lds4(&S.lift[2][c0 + c]);
                const float2 u2 = make_float2(lu, lu), x2 = make_float2(lx, lx);
                v[c / 2] = __ffma2_rn(make_float2(w0.x, w0.y), u2,
                                      __ffma2_rn(make_float2(w1.x, w1.y), x2, make_float2(bb.x, bb.y)));
                v[c / 2 + 1] = __ffma2_rn(make_float2(w0.z, w0.w), u2,
                                          __ffma2_rn(make_float2(w1.z, w1.w), x2, make_float2(bb.z, bb.w)));
            }
        } else if constexpr (kInGelu) {
#pragma unroll
            for (int i = 0; i < C / 2; ++i) v[i] = act::gelu2(v[i]);
        }
        // scales: sx ws = 2 sm (the inverse table's scale is 2), each at least its operand's max
        float sx = tc::pow2_above(vmax), sm = tc::pow2_above(mmax);
        const float scale = fmaxf(sx * ws, 2.f * sm);
        sx = fmaxf(sx, scale / ws);
        sm = fmaxf(sm, 0.5f * scale);
        store_point<W, C>(S.x, v, 256.f / sx, c0, t);
        if (tid < 4 * W) {
            uint4 r[3];
            tc::split8(mv, 256.f / sm, r[0], r[1], r[2]);
#pragma unroll
            for (int pc = 0; pc < 3; ++pc)
                *reinterpret_cast<uint4*>(S.m + (tid % 4) * (3 * W * 16) + (pc * W + tid / 4) * 16) = r[pc];
        }
        return scale * (1.f / 65536.f);
    };
    // BWD0: sums of the staged dL/dz over the points, times u, the grid and 1
    float s0 = 0.f, s1 = 0.f;
    auto point_sums = [&](const float2(&x)[C / 2], int first) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const float f = r == 0 ? s0 : (r == 1 ? s1 : 1.f);
            float e[C];
#pragma unroll
            for (int i = 0; i < C / 2; ++i) {
                e[2 * i] = x[i].x * f;
                e[2 * i + 1] = x[i].y * f;
            }
            sum[first + r] += warp_sums<C>(e, t & 31);
        }
    };
    auto load_ends = [&](int b) {
        if constexpr (MODE == BWD0) {
            s0 = on ? __ldg(a.u + (int64_t)b * N + p) : 0.f;
            s1 = on ? __ldg(a.grid + (int64_t)b * a.grid_stride + p) : 0.f;
        }
    };
    load_tile(b0);
    float f_next = stage_tile();
    tc::fence_smem();
    issue(0);
    if constexpr (MODE == BWD0) {
        load_ends(b0);
        point_sums(v, 0);
    }
    load_tile(b0 + step);
    int buf = 0;
    for (int b = b0; b < a.batch; b += step) {
        float2 zp[MODE == BWD ? C / 2 : 1];
        if constexpr (MODE == BWD) load_channels<C, N>(a.zprev + ((int64_t)b * W + c0) * N + p, on, zp);
        if (!fail) fail = !tc::mbar_wait(&S.bar_layer, phase);
        phase ^= 1;
        const float fx = fail ? __int_as_float(0x7fffffff) : f_next;
        const float u0 = s0, u1 = s1;  // (BWD0: this tile's)
        if (b + step < a.batch) {  // the tile's products are done: its buffers take the next one
            f_next = stage_tile();
            tc::fence_smem();
            tc::fence_before();
            issue(buf ^ 1);
            if constexpr (MODE == BWD0) {
                load_ends(b + step);
                point_sums(v, 0);
            }
        }
        load_tile(b + 2 * step);
        tc::fence_after();
        float m = 0.f, gu = 0.f;
        float* out = MODE == BWD0 ? nullptr : a.out + ((int64_t)b * W + c0) * N + p;
        float2 h[MODE == BWD0 ? C / 2 : 1];
        constexpr int CH = MODE == BWD ? 8 : 16;  // columns at a time (BWD holds zprev beside them)
#pragma unroll
        for (int i0 = 0; i0 < C; i0 += CH) {
            float x0[CH], x1[CH];
            tc::tmem_ld(dl + 2 * W * buf + i0, x0);
            tc::tmem_ld(dl + 2 * W * buf + W + i0, x1);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < CH; i += 4) {
                const float4 bi = kBwd ? make_float4(0.f, 0.f, 0.f, 0.f) : lds4(&S.bias[c0 + i0 + i]);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int e = i + 2 * j, ch = i0 + e;
                    float2 z = __ffma2_rn(join2(x0[e], x0[e + 1], x1[e], x1[e + 1]), make_float2(fx, fx),
                                          j == 0 ? make_float2(bi.x, bi.y) : make_float2(bi.z, bi.w));
                    if constexpr (MODE == BWD) z = __fmul2_rn(z, act::gelu_grad2(zp[ch / 2]));
                    if constexpr (MODE == FWD) {
                        m = fmaxf(m, fmaxf(z.x, z.y));  // |gelu(z)| <= max(z, 0.17)
                        if constexpr (kStoreGelu) z = act::gelu2(z);
                    } else {
                        m = fmaxf(m, fmaxf(fabsf(z.x), fabsf(z.y)));
                    }
                    if constexpr (MODE == BWD0) {
                        gu = fmaf(z.x, S.lift[0][c0 + ch], fmaf(z.y, S.lift[0][c0 + ch + 1], gu));
                        h[ch / 2] = on ? z : make_float2(0.f, 0.f);
                    } else if (on) {
                        out[ch * N] = z.x;
                        out[(ch + 1) * N] = z.y;
                    }
                }
            }
        }
        tc::fence_before();
        if constexpr (MODE == BWD0) {
            const float n0 = s0, n1 = s1;
            s0 = u0;
            s1 = u1;
            point_sums(h, 3);
            s0 = n0;
            s1 = n1;
            if (half == 1) S.gu[t] = gu;
            worker_sync();
            if (half == 0 && on && a.g_u) a.g_u[(int64_t)b * N + p] = gu + S.gu[t];
            worker_sync();
        } else {
            m = warp_max(on ? m : 0.f);
            if ((tid & 31) == 0) S.red[0][tid >> 5] = m;
            worker_sync();
            if (tid == 0) {
                const float4 r0 = lds4(S.red[0]), r1 = lds4(S.red[0] + 4);
                const float tm = fmaxf(fmaxf(fmaxf(r0.x, r0.y), fmaxf(r0.z, r0.w)),
                                       fmaxf(fmaxf(r1.x, r1.y), fmaxf(r1.z, r1.w)));
                a.tmax[(int64_t)q * a.batch + b] = MODE == FWD ? fmaxf(tm, 0.17f) : tm;
            }
            worker_sync();  // (S.red is read)
        }
        buf ^= 1;
    }
    if constexpr (MODE == BWD0) {
        // the CTA's sums: its four warps of either half added in order
        const int lane = t & 31;
        float* s = reinterpret_cast<float*>(S.x);  // [4][6][W]; every product is done
#pragma unroll
        for (int r = 0; r < 6; ++r)
            if (lane % (32 / C) == 0) s[((t >> 5) * 6 + r) * W + c0 + lane / (32 / C)] = sum[r];
        worker_sync();
        for (int i = tid; i < 6 * W; i += WORKERS)
            a.sums[(int64_t)blockIdx.x * 6 * W + i] = (s[i] + s[6 * W + i]) + (s[12 * W + i] + s[18 * W + i]);
    }
    tc::fence_before();
    __syncthreads();
    if (tid < 32) tc::tmem_free(d, COLS);
}

// CTAs of a tile kernel: at most two per SM, a multiple of the row positions
inline int tile_grid(int batch, int nq) {
    const int most = 2 * sm_count() / nq * nq, want = batch * nq;
    return want < most ? want : (most > 0 ? most : nq);
}

template <int W, int N, bool LIFT, int MODE, bool TRAIN>
int launch_layer(const LayerArgs& a, cudaStream_t st) {
    const size_t smem = sizeof(LayerSmem<W>);
    static_assert(sizeof(LayerSmem<W>) <= 113 * 1024, "two CTAs per SM");
    cudaFuncSetAttribute(k_fno_layer<W, N, LIFT, MODE, TRAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_fno_layer<W, N, LIFT, MODE, TRAIN><<<tile_grid(a.batch, N < 128 ? 1 : N / 128), layer_threads(MODE), smem, st>>>(a);
    return check_launch("fno layer");
}
template <int W, bool LIFT, int MODE, bool TRAIN>
int run_layer(const LayerArgs& a, int n, cudaStream_t st) {
    switch (n) {
        case 64: return launch_layer<W, 64, LIFT, MODE, TRAIN>(a, st);
        case 128: return launch_layer<W, 128, LIFT, MODE, TRAIN>(a, st);
        case 256: return launch_layer<W, 256, LIFT, MODE, TRAIN>(a, st);
        default: return launch_layer<W, 512, LIFT, MODE, TRAIN>(a, st);
    }
}

// ---- modes of a state ------------------------------------------------------------------
// part[k][b][c] = sum_p x[b][c][p] e^{-2 pi i k p / N}, k < modes: the [batch * W] rows are the
// accumulator lanes (128 per tile: 2 trajectories at W = 64, 4 at 32), the points the
// contraction, 64 per chunk, and the table's 96 stacked rows the columns.  A thread
// splits 8 consecutive points of a row at a time (float4 loads, 256 contiguous bytes per
// 8 lanes); the planes' pitch of 2064 bytes makes their 16-byte stores conflict-free.
// 16 warps split (and apply GELU), a 17th issues.  Bound by reading the state and the split:
// 12.8 us at 256 x 64 x 512 (33.5 MB, 5.2 us at the copy rate; 128 tiles leave 20 SMs idle),
// 14.7 with GELU, 22.1 at 512 x 64 x 512 (256 tiles on 148 SMs: a second round on 108).
constexpr int MODES_WORKERS = 512;
constexpr int A_PITCH = 2048 + 16;
struct ModesArgs {
    const float* x;      // [rows][N], with GELU through it
    const float* xmax;   // [tiles per row][batch]
    const unsigned char* table;
    float2* part;        // [modes][batch][W] = [modes][rows]
    int rows, batch, modes;
};
struct ModesSmem {
    alignas(128) unsigned char ft[64 * F_PLANE];
    alignas(128) unsigned char a[2][3 * 8 * A_PITCH];
    uint64_t bar_images, bar[2];
    uint32_t tmem;
};

template <int W, int N, bool GELU>
__global__ void __launch_bounds__(MODES_WORKERS + 32, 1) k_fno_modes(ModesArgs a) {
    extern __shared__ __align__(128) unsigned char fno_smem[];
    ModesSmem& S = *reinterpret_cast<ModesSmem*>(fno_smem);
    constexpr int nq = N < 128 ? 1 : N / 128, CHUNKS = N / 64;
    const int tid = threadIdx.x, tiles = (a.rows + 127) / 128;
    if (tid >= MODES_WORKERS) tc::tmem_alloc(&S.tmem, 128);
    if (tid == MODES_WORKERS) {
        tc::mbar_init(&S.bar_images, 1);
        tc::mbar_init(&S.bar[0], 1);
        tc::mbar_init(&S.bar[1], 1);
        tc::mbar_init_fence();
        tc::mbar_expect(&S.bar_images, N / 8 * F_PLANE);
        tc::bulk_load(S.ft, a.table, N / 8 * F_PLANE, &S.bar_images);
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t d = S.tmem;
    if (tid >= MODES_WORKERS) {  // the issuing warp
        const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&S.bar_images, 0));
        int n = 0;
        for (int i = blockIdx.x; i < tiles; i += gridDim.x)
            for (int ch = 0; ch < CHUNKS; ++ch, ++n) {
                take_over<MODES_WORKERS>(n & 1);
                if (ok && tc::elect()) {
                    tc::fence_after();
                    const uint64_t x = tc::smem_desc(tc::smem_u32(S.a[n & 1]), A_PITCH, 128);
                    const uint64_t f = tc::smem_desc(tc::smem_u32(S.ft) + ch * 8 * F_PLANE, F_PLANE, 128);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint64_t ak = tc::desc_at(x, 2 * k * A_PITCH), bd = tc::desc_at(f, 2 * k * F_PLANE);
                        const uint64_t mid = tc::desc_at(ak, 8 * A_PITCH), lo = tc::desc_at(ak, 16 * A_PITCH);
                        const bool add = ch + k > 0;
                        tc::mma(d, ak, bd, tc::instr_desc(128, 96), add);
                        if (add) {
                            tc::mma(d + 32, mid, bd, tc::instr_desc(128, 96), true);
                        } else {  // (the first to write the last 32 columns)
                            tc::mma(d + 32, mid, bd, tc::instr_desc(128, 64), true);
                            tc::mma(d + 96, mid, tc::desc_at(bd, 64 * 16), tc::instr_desc(128, 32), false);
                        }
                        tc::mma(d + 64, lo, bd, tc::instr_desc(128, 64), true);
                    }
                    tc::commit(&S.bar[n & 1]);
                }
                __syncwarp();
            }
        tc::fence_before();
        __syncthreads();
        tc::tmem_free(S.tmem, 128);
        return;
    }
    bool fail = false;
    const int c8 = tid & 7, r0 = tid >> 3;  // this thread's points of a chunk; rows r0 and r0 + 64
    // chunks are loaded two ahead, so that a load has about two chunks' time to arrive
    float4 v[2][2][2];
    const int mine = blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x * CHUNKS : 0;
    auto load = [&](int n, float4(&w)[2][2]) {
        const int i = blockIdx.x + n / CHUNKS * gridDim.x, ch = n % CHUNKS;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = i * 128 + r0 + 64 * h;
            w[h][0] = w[h][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (n < mine && row < a.rows) {
                const float4* s = reinterpret_cast<const float4*>(a.x + (int64_t)row * N + ch * 64 + 8 * c8);
                w[h][0] = ldg_na4(s);
                w[h][1] = ldg_na4(s + 1);
            }
        }
    };
    // max over the row positions of a trajectory's tiles
    auto row_scale = [&](int row) -> float {
        const int b = row < a.rows ? row / W : 0;
        float m = 0.f;
#pragma unroll
        for (int q = 0; q < nq; ++q) m = fmaxf(m, __ldg(a.xmax + (int64_t)q * a.batch + b));
        return tc::pow2_above(m);
    };
    uint32_t used = 0;  // phases of the two buffers waited for
    float inv[2] = {0.f, 0.f};
    auto chunk = [&](int n, int buf, float4(&w)[2][2]) {
        const int i = blockIdx.x + n / CHUNKS * gridDim.x, ch = n % CHUNKS;
        if (ch == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) inv[h] = 256.f / row_scale(i * 128 + r0 + 64 * h);
        }
        if (n >= 2) {  // the products of two chunks ago have read the buffer
            if (!fail) fail = !tc::mbar_wait(&S.bar[buf], (used >> buf) & 1);
            used ^= 1u << buf;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float2 e[4] = {make_float2(w[h][0].x, w[h][0].y), make_float2(w[h][0].z, w[h][0].w),
                           make_float2(w[h][1].x, w[h][1].y), make_float2(w[h][1].z, w[h][1].w)};
            uint32_t hi[4], mid[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if constexpr (GELU) e[j] = act::gelu2(e[j]);
                tc::split2(e[j], make_float2(inv[h], inv[h]), hi[j], mid[j], lo[j]);
            }
            unsigned char* s = S.a[buf] + c8 * A_PITCH + (r0 + 64 * h) * 16;
            *reinterpret_cast<uint4*>(s) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(s + 8 * A_PITCH) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
            *reinterpret_cast<uint4*>(s + 16 * A_PITCH) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
        tc::fence_smem();
        tc::fence_before();
        hand_over<MODES_WORKERS>(buf);
        load(n + 2, w);
        if (ch != CHUNKS - 1) return;
        // the tile is complete with every chunk's products: the last of either buffer
        if (CHUNKS > 1) {
            if (!fail) fail = !tc::mbar_wait(&S.bar[buf ^ 1], (used >> (buf ^ 1)) & 1);
        }
        if (!fail) fail = !tc::mbar_wait(&S.bar[buf], (used >> buf) & 1);
        tc::fence_after();
        // 4 warps per 32 lanes: 8 of the 32 columns (4 modes) each
        const int lane_row = tid & 127, part = tid >> 7, row = i * 128 + lane_row;
        const uint32_t dl = d + ((uint32_t)(tid & 96) << 16) + 8 * part;
        float q0[8], q1[8], q2[8], q3[8];
        tc::tmem_ld8(dl, q0);
        tc::tmem_ld8(dl + 32, q1);
        tc::tmem_ld8(dl + 64, q2);
        tc::tmem_ld8(dl + 96, q3);
        tc::tmem_ld_wait();
        tc::fence_before();
        worker_sync<MODES_WORKERS>();  // read everywhere before the next tile's products
        if (row < a.rows) {
            const float f = fail ? __int_as_float(0x7fffffff) : row_scale(row) * (1.f / (256.f * F_SCALE));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = 4 * part + j;
                auto sum = [&](int e) { return fmaf(fmaf(fmaf(q3[e], tc::DOWN, q2[e]), tc::DOWN, q1[e]), tc::DOWN, q0[e]); };
                if (k < a.modes) a.part[(int64_t)k * a.rows + row] = make_float2(sum(2 * j) * f, sum(2 * j + 1) * f);
            }
        }
    };
    load(0, v[0]);
    load(1, v[1]);
    for (int n = 0; n < mine; n += 2) {
        chunk(n, 0, v[0]);
        if (n + 1 < mine) chunk(n + 1, 1, v[1]);
    }
    tc::fence_before();
    __syncthreads();
}

template <int W, int N, bool GELU>
int launch_modes(const ModesArgs& a, cudaStream_t st) {
    cudaFuncSetAttribute(k_fno_modes<W, N, GELU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ModesSmem));
    static_assert(sizeof(ModesSmem) <= 227 * 1024, "shared memory");
    const int tiles = (a.rows + 127) / 128, sms = sm_count();
    k_fno_modes<W, N, GELU><<<tiles < sms ? tiles : sms, MODES_WORKERS + 32, sizeof(ModesSmem), st>>>(a);
    return check_launch("fno modes");
}
template <int W, bool GELU>
int run_modes(const ModesArgs& a, int n, cudaStream_t st) {
    switch (n) {
        case 64: return launch_modes<W, 64, GELU>(a, st);
        case 128: return launch_modes<W, 128, GELU>(a, st);
        case 256: return launch_modes<W, 256, GELU>(a, st);
        default: return launch_modes<W, 512, GELU>(a, st);
    }
}

// ---- mode mixing ---------------------------------------------------------------------
// out[b][k][r] = (1 / n) sum_j in[k][b][j] S[k][j][r]; S[k][j][r] = W[j][r][k] (forward) or
// conj(W[r][j][k]) (adjoint), laid out by the preparation.  omax[b] = max |out[b]| (zeroed by
// the preparation; a max does not depend on the order).  Block: one mode, MIX_B = 32
// trajectories; a thread has four outputs of MIX_R trajectories over half of the inputs
// (the halves are joined by shuffles), real and imaginary factors in separate packed
// accumulators (two packed operations per complex product).  The first form (all inputs
// per thread, scalar operations, 64 trajectories) took 11.5 us at 256 x 64 x 16 modes: too few
// blocks, each a long chain.
template <int W>
constexpr int mix_r() { return W == 64 ? 4 : 2; }
constexpr int MIX_B = 32;
template <int W>
__global__ void __launch_bounds__(256) k_fno_mix(const float2* __restrict__ in, const float2* __restrict__ wt,
                                                 float2* __restrict__ out, float* __restrict__ omax, int batch,
                                                 int modes, float scale) {
    constexpr int MIX_R = mix_r<W>(), TPT = W / 4, SUB = 128 / TPT;
    static_assert(SUB * MIX_R == MIX_B, "trajectories per block");
    extern __shared__ __align__(128) unsigned char fno_smem[];
    float4* S = reinterpret_cast<float4*>(fno_smem);               // [W][W / 2] pairs of complex
    float4* X = S + W * W / 2;                                     // [MIX_B][W / 2]
    const int k = blockIdx.x, b0 = blockIdx.y * MIX_B, nb = min(MIX_B, batch - b0);
    const float4* src = reinterpret_cast<const float4*>(wt + (int64_t)k * W * W);
    const float4* xin = reinterpret_cast<const float4*>(in + ((int64_t)k * batch + b0) * W);
#pragma unroll
    for (int i = threadIdx.x; i < W * W / 2; i += 256) S[i] = __ldg(src + i);
#pragma unroll
    for (int i = threadIdx.x; i < MIX_B * W / 2; i += 256)
        X[i] = 2 * i < nb * W ? __ldg(xin + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    // lanes: outputs, then the half of the inputs, then trajectories
    const int r0 = threadIdx.x % TPT, jh = threadIdx.x / TPT % 2, b = threadIdx.x / (2 * TPT);
    float2 re[MIX_R][4], im[MIX_R][4];
#pragma unroll
    for (int i = 0; i < MIX_R; ++i)
#pragma unroll
        for (int r = 0; r < 4; ++r) re[i][r] = im[i][r] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int jj = 0; jj < W / 2; ++jj) {
        const int j = jh * (W / 2) + jj;
        const float4 w0 = S[j * (W / 2) + 2 * r0], w1 = S[j * (W / 2) + 2 * r0 + 1];
        const float2 w[4] = {make_float2(w0.x, w0.y), make_float2(w0.z, w0.w), make_float2(w1.x, w1.y),
                             make_float2(w1.z, w1.w)};
#pragma unroll
        for (int i = 0; i < MIX_R; ++i) {
            const float2 x = reinterpret_cast<const float2*>(X)[(b + i * SUB) * W + j];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                re[i][r] = __ffma2_rn(make_float2(x.x, x.x), w[r], re[i][r]);
                im[i][r] = __ffma2_rn(make_float2(x.y, x.y), w[r], im[i][r]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < MIX_R; ++i) {
        float m = 0.f;
        float2 o[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            o[r] = make_float2(re[i][r].x - im[i][r].y, re[i][r].y + im[i][r].x);
            o[r].x += __shfl_xor_sync(0xffffffffu, o[r].x, TPT);
            o[r].y += __shfl_xor_sync(0xffffffffu, o[r].y, TPT);
            o[r].x *= scale;
            o[r].y *= scale;
            m = fmaxf(m, fmaxf(fabsf(o[r].x), fabsf(o[r].y)));
        }
#pragma unroll
        for (int s = TPT / 2; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
        const int bb = b + i * SUB;
        if (bb < nb && jh == 0) {
            float4* dst = reinterpret_cast<float4*>(out + ((int64_t)(b0 + bb) * modes + k) * W + 4 * r0);
            dst[0] = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
            dst[1] = make_float4(o[2].x, o[2].y, o[3].x, o[3].y);
            if (r0 == 0) atomicMax(reinterpret_cast<unsigned int*>(omax) + b0 + bb, __float_as_uint(m));
        }
    }
}

template <int W>
int run_mix(const float2* in, const float2* wt, float2* out, float* omax, int batch, int n, int modes,
            cudaStream_t st) {
    const size_t smem = (W * W + MIX_B * W) * sizeof(float2);
    cudaFuncSetAttribute(k_fno_mix<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_fno_mix<W><<<dim3(modes, (batch + MIX_B - 1) / MIX_B), 256, smem, st>>>(in, wt, out, omax, batch, modes,
                                                                           1.f / (float)n);
    return check_launch("fno mix");
}

// ---- preparation ------------------------------------------------------------------------
// One launch per call: the four layers' complex weights [c][o][k] laid out as
// [layer][k][j][r] (see k_fno_mix), the 1x1 branches, fc1 and the row positions' tables as
// shared-memory images, the zeroed magnitudes, and (forward) the modes of the lifted
// state: part[k][b][c] = w[c][0] U[k] + w[c][1] X[k] + (k == 0) n b[c] with U and X the
// transforms of u's row b and of the grid's, summed in FP64 (the ramp's are large).
struct PrepArgs {
    const float2* modes_w[4];
    const float* w[4];
    const float* fc1;
    const float* u;
    const float* grid;
    const float* fc0_w;
    const float* fc0_b;
    float2* wt;     // [4][modes][W][W]
    float2* part;   // [modes][batch][W]
    float* zero;    // [4][batch]
    int64_t grid_stride;
    int batch, n, modes;
};

template <int W, bool ADJ>
__global__ void __launch_bounds__(256) k_fno_prep(PrepArgs a, Prep<W>* __restrict__ out) {
    __shared__ float2 cs[512];
    __shared__ float su[512], sx[512], red[8];
    __shared__ double4 sums[16][KM];
    const int t = threadIdx.x, M = a.modes, n = a.n;
    const int points = n < 128 ? n : 128, nq = n / points;
    int blk = blockIdx.x;
    if (blk < nq) {
        stage_period(cs, n);
        __syncthreads();
        stage_inverse(out->inverse[blk], cs, blk * points, n, M);
        stage_transform(out->transform, cs, n, M, blk * points / 8 * KM, points / 8 * KM);
        return;
    }
    blk -= nq;
    if (blk < 4) {
        const float s = cta_scale(a.w[blk], W * W, red);
        stage_matrix<W, W, ADJ>(out->w[blk], a.w[blk], s);
        if (t == 0) out->scale[blk] = s;
        return;
    }
    blk -= 4;
    if (blk == 0) {
        const float s = cta_scale(a.fc1, 128 * W, red);
        stage_matrix<128, W, false>(out->fc1, a.fc1, s);
        if (t == 0) out->scale[4] = s;
        return;
    }
    blk -= 1;
    const int per_layer = W * W * M / 256;  // (W is 32 or 64)
    if (blk < 4 * per_layer) {
        const int l = blk / per_layer, e = (blk - l * per_layer) * 256 + t;  // e: (k * W + j) * W + r
        const int r = e % W, j = (e / W) % W, k = e / (W * W);
        const float2 v = __ldg(a.modes_w[l] + (int64_t)(ADJ ? r * W + j : j * W + r) * M + k);
        a.wt[(int64_t)l * W * W * M + e] = make_float2(v.x, ADJ ? -v.y : v.y);
        return;
    }
    blk -= 4 * per_layer;
    if (ADJ) {
        for (int i = blk * 256 + t; i < 4 * a.batch; i += (gridDim.x - (blockIdx.x - blk)) * 256) a.zero[i] = 0.f;
        return;
    }
    const int b = blk;
    if (t < 4) a.zero[t * a.batch + b] = 0.f;
    for (int i = t; i < n; i += 256) {
        su[i] = __ldg(a.u + (int64_t)b * n + i);
        sx[i] = __ldg(a.grid + (int64_t)b * a.grid_stride + i);
    }
    stage_period(cs, n);
    __syncthreads();
    const int k = t % KM, slice = t / KM;
    double4 s = make_double4(0.0, 0.0, 0.0, 0.0);
    for (int i = slice; i < n; i += 16) {
        const float2 e = cs[(k * i) & (n - 1)];
        s.x = fma((double)su[i], (double)e.x, s.x);
        s.y = fma((double)su[i], -(double)e.y, s.y);
        s.z = fma((double)sx[i], (double)e.x, s.z);
        s.w = fma((double)sx[i], -(double)e.y, s.w);
    }
    sums[slice][k] = s;
    __syncthreads();
    for (int o = 8; o > 0; o >>= 1) {
        if (slice < o) {
            const double4 e = sums[slice + o][k];
            s.x += e.x; s.y += e.y; s.z += e.z; s.w += e.w;
            sums[slice][k] = s;
        }
        __syncthreads();
    }
    for (int i = t; i < M * W; i += 256) {
        const int kk = i / W, c = i % W;
        const double4 e = sums[0][kk];
        const double w0 = __ldg(a.fc0_w + 2 * c), w1 = __ldg(a.fc0_w + 2 * c + 1);
        const double re = w0 * e.x + w1 * e.z + (kk == 0 ? (double)n * __ldg(a.fc0_b + c) : 0.0);
        a.part[((int64_t)kk * a.batch + b) * W + c] =
            make_float2((float)re, kk == 0 ? 0.f : (float)(w0 * e.y + w1 * e.w));
    }
}

template <int W, bool ADJ>
int run_prep(const PrepArgs& a, Prep<W>* out, cudaStream_t st) {
    const int nq = a.n < 128 ? 1 : a.n / 128;
    const int blocks = nq + 5 + 4 * (W * W * a.modes / 256) + (ADJ ? (4 * a.batch + 255) / 256 : a.batch);
    k_fno_prep<W, ADJ><<<blocks, 256, 0, st>>>(a, out);
    return check_launch("fno preparation");
}

inline bool supported(int width, int n, int modes) {
    return (width == 32 || width == 64) && (n == 64 || n == 128 || n == 256 || n == 512) && modes >= 1 && modes <= KM;
}

}  // namespace fno
}  // namespace inc
