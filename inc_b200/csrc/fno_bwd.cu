// Backward of the FNO corrector (fno_fwd.cu): the gradients of u and of every parameter from
// dL/dy, the layers' sums before GELU (z), the modes of the layers' inputs and the tiles'
// magnitudes that the forward recorded.
//
//   projection   k_fno_proj_bwd: the 128 hidden values again (one product), their
//                gradient g1 = dy w2 gelu'(a) (stored for fc1's weight gradient), dL/dz of
//                the last layer (a second product with the same weights read transposed)
//                and fc2's gradient;
//   layer l      modes of dL/dz_l (k_fno_modes), their adjoint mixing, and k_fno_layer with the
//                transposed weights, times gelu'(z_{l-1}): dL/dz_{l-1};
//   weights      k_fno_wgrad: dL/dz (or g1) times the layer's input, contracted over all
//                points on the tensor cores; the Fourier weights from the modes
//                (k_fno_modes_grad);
//   the lift     folded into layer 0's adjoint: the lifted state is affine in (u, grid, 1), so
//                its weight gradient and fc0's are six sums per channel.
#include "fno_tc.cuh"

namespace inc {
namespace fno {

int check_fno(const inc_fno_desc* d);  // fno_fwd.cu

// ---- projection -------------------------------------------------------------------------
// Bound, like the forward's, by the GELUs (with their derivative) and three rounds of products
// per tile, each waited for; 100 MB written.  56 us at 256 x 64 x 512 (51 with six products of bf16
// pieces; letting one of the eight warps issue, 128 registers in place of 96 and no spills,
// measured 52 then).
struct ProjBwdArgs {
    const float* x;      // z of the last layer [batch][W][N]
    const float* xmax;   // [tiles per row][batch]
    const unsigned char* fc1;  // image
    const float* wscale;
    const float* fc1_b;  // [128]
    const float* fc2_w;  // [128]
    const float* g_y;    // [batch][N]
    float* g1;           // [batch][128][N]
    float* g1max;        // [tiles per row][batch]
    float* g_x;          // [batch][W][N]
    float* gxmax;        // [tiles per row][batch]
    float* sums;         // [blocks][132]: fc2's gradient, then its bias's
    int batch;
};

template <int W>
struct ProjBwdSmem {
    alignas(128) unsigned char w[3 * 128 * W * 2];
    alignas(128) unsigned char x[3 * 64 * 128 * 2];
    alignas(16) float b1[128], w2[128];
    alignas(16) float red[2][WORKERS / 32];
    float w2max;
    uint64_t bar_images, bar;
    uint32_t tmem;
};

template <int W, int N>
__global__ void __launch_bounds__(THREADS, 2) k_fno_proj_bwd(ProjBwdArgs a) {
    extern __shared__ __align__(128) unsigned char fno_smem[];
    ProjBwdSmem<W>& S = *reinterpret_cast<ProjBwdSmem<W>*>(fno_smem);
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
    if (tid < 32) {
        float m = 0.f;
        for (int i = tid; i < 128; i += 32) m = fmaxf(m, fabsf(__ldg(a.fc2_w + i)));
        m = warp_max(m);
        if (tid == 0) S.w2max = m;
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t d = S.tmem;
    if (tid >= WORKERS) {  // the issuing warp: three products per tile
        const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&S.bar_images, 0));
        for (int i = blockIdx.x; i < tiles; i += step) {
            take_over();
            if (ok && tc::elect()) {  // hidden values: columns 0..127 and 128..255
                tc::fence_after();
                issue_product<128, W>(d, tc::smem_u32(S.x), W * 256, tc::smem_u32(S.w));
                tc::commit(&S.bar);
            }
            __syncwarp();
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {  // g1[64 h ..] w1, into columns 64 h .. and 128 + 64 h .., read by then
                take_over();
                if (ok && tc::elect()) {
                    tc::fence_after();
                    const uint64_t x = tc::smem_desc(tc::smem_u32(S.x), 2048, 128);
                    const uint64_t w = tc::smem_desc(tc::smem_u32(S.w) + 64 * h * 16, 128, 384 * 16);
                    constexpr uint32_t id = tc::instr_desc(128, W, false, true);
#pragma unroll
                    for (int stage = 3; stage > 0; --stage)  // (as issue_stage; the operand B is MN-major here)
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t c0 = d + 64 * h, c1 = c0 + 128;
                            const uint64_t a0 = tc::desc_at(x, 2 * k * 2048), a1 = tc::desc_at(a0, 8 * 2048);
                            const uint64_t a2 = tc::desc_at(a0, 16 * 2048), b0 = tc::desc_at(w, 16 * k * 16);
                            const uint64_t b1 = tc::desc_at(b0, 128 * 16), b2 = tc::desc_at(b0, 256 * 16);
                            if (stage == 3) {
                                tc::mma(c1, a1, b2, id, k > 0);
                                tc::mma(c1, a2, b1, id, true);
                            } else if (stage == 2) {
                                if (k == 0) tc::mma_scaled(c1, a0, b2, id);
                                else tc::mma(c1, a0, b2, id, true);
                                tc::mma(c1, a1, b1, id, true);
                                tc::mma(c1, a2, b0, id, true);
                            } else {
                                tc::mma(c0, a0, b0, id, k > 0);
                                if (k == 0) tc::mma_scaled(c1, a0, b1, id);
                                else tc::mma(c1, a0, b1, id, true);
                                tc::mma(c1, a1, b0, id, true);
                            }
                        }
                    tc::commit(&S.bar);
                }
                __syncwarp();
            }
        }
        tc::fence_before();
        __syncthreads();
        tc::tmem_free(S.tmem, 256);
        return;
    }
    const bool on = points == 128 || t < points;
    const float ws = __ldg(a.wscale) * (1.f / 65536.f), gbound = 1.13f * S.w2max;  // max gelu' = 1.1290
    const uint32_t dl = d + ((uint32_t)(t & 96) << 16);
    uint32_t phase = 0;
    bool fail = false;
    auto wait = [&] {
        if (!fail) fail = !tc::mbar_wait(&S.bar, phase);
        phase ^= 1;
        tc::fence_after();
    };
    float2 v[C / 2];
    float vmax = 0.f, g_next = 0.f, sum[2] = {0.f, 0.f}, sum_g = 0.f;
    auto load_tile = [&](int i) {
        if (i >= tiles) return;
        const int b = i / nq, p = (i % nq) * points + t;
        load_channels<C, N>(a.x + ((int64_t)b * W + half * C) * N + p, on, v);
        vmax = __ldg(a.xmax + (int64_t)(i % nq) * a.batch + b);
        g_next = on ? __ldg(a.g_y + (int64_t)b * N + p) : 0.f;
    };
    load_tile(blockIdx.x);
    for (int i = blockIdx.x; i < tiles; i += step) {
        const int b = i / nq, p = (i % nq) * points + t;
        const float sx = tc::pow2_above(vmax), gy = g_next;
        store_point<W, C>(S.x, v, 256.f / sx, half * C, t);
        tc::fence_smem();
        tc::fence_before();
        hand_over();
        load_tile(i + step);
        const float sg = tc::pow2_above(fabsf(gy) * gbound);  // of this point's g1
        float m1 = 0.f;
        if (half == 0) sum_g += gy;
        wait();
        const float2 f = make_float2(sx * ws, sx * ws);
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // hidden values 64 h + 32 half ..
            const int j0 = 64 * h + 32 * half;
            float2 g[16];
            float e2[32];
            float* out = a.g1 + ((int64_t)b * 128 + j0) * N + p;
#pragma unroll
            for (int c = 0; c < 32; c += 16) {
                float x0[16], x1[16];
                tc::tmem_ld16(dl + j0 + c, x0);
                tc::tmem_ld16(dl + 128 + j0 + c, x1);
                tc::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; e += 2) {
                    const int j = c + e;
                    const float2 bi = *reinterpret_cast<const float2*>(&S.b1[j0 + j]);
                    const float2 w2 = *reinterpret_cast<const float2*>(&S.w2[j0 + j]);
                    const float2 z = __ffma2_rn(join2(x0[e], x0[e + 1], x1[e], x1[e + 1]), f, bi);
                    float2 y, gp;
                    act::gelu_both2(z, y, gp);
                    const float2 gg = make_float2(gy, gy);
                    y = __fmul2_rn(y, gg);
                    e2[j] = y.x;
                    e2[j + 1] = y.y;
                    float2 r = __fmul2_rn(__fmul2_rn(gp, w2), gg);
                    if (fail) r = make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
                    g[j / 2] = r;
                    m1 = fmaxf(m1, fmaxf(fabsf(r.x), fabsf(r.y)));
                    if (on) {
                        out[j * N] = r.x;
                        out[(j + 1) * N] = r.y;
                    }
                }
            }
            sum[h] += warp_sums<32>(e2, t & 31);
            if (h == 1) wait();  // the first half's products have read the tile
            store_point<64, 32>(S.x, g, 256.f / sg, 32 * half, t);
            tc::fence_smem();
            tc::fence_before();
            hand_over();
        }
        wait();
        const float fs = sg * ws;
        float m3 = 0.f;
        float* out = a.g_x + ((int64_t)b * W + half * C) * N + p;
#pragma unroll
        for (int c = 0; c < C; c += 8) {
            float x0[8], x1[8], y0[8], y1[8];
            tc::tmem_ld8(dl + half * C + c, x0);
            tc::tmem_ld8(dl + 128 + half * C + c, x1);
            tc::tmem_ld8(dl + 64 + half * C + c, y0);
            tc::tmem_ld8(dl + 192 + half * C + c, y1);
            tc::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float r = fmaf(x1[e] + y1[e], tc::DOWN, x0[e] + y0[e]) * fs;
                m3 = fmaxf(m3, fabsf(r));
                if (on) out[(c + e) * N] = fail ? __int_as_float(0x7fffffff) : r;
            }
        }
        tc::fence_before();
        m1 = warp_max(on ? m1 : 0.f);
        m3 = warp_max(on ? m3 : 0.f);
        if ((tid & 31) == 0) {
            S.red[0][tid >> 5] = m1;
            S.red[1][tid >> 5] = m3;
        }
        worker_sync();
        if (tid < 2) {
            const float4 r0 = lds4(S.red[tid]), r1 = lds4(S.red[tid] + 4);
            (tid == 0 ? a.g1max : a.gxmax)[(int64_t)(i % nq) * a.batch + b] =
                fmaxf(fmaxf(fmaxf(r0.x, r0.y), fmaxf(r0.z, r0.w)), fmaxf(fmaxf(r1.x, r1.y), fmaxf(r1.z, r1.w)));
        }
        worker_sync();
    }
    // the CTA's sums, its four warps of either half added in order
    float* s = reinterpret_cast<float*>(S.x);  // [4][128], then [4]; every product is done
    const int w = t >> 5, lane = t & 31;
    s[w * 128 + 32 * half + lane] = sum[0];
    s[w * 128 + 64 + 32 * half + lane] = sum[1];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum_g += __shfl_xor_sync(0xffffffffu, sum_g, o);
    if (half == 0 && lane == 0) s[512 + w] = sum_g;
    worker_sync();
    float* out = a.sums + (int64_t)blockIdx.x * 132;
    if (tid < 128) out[tid] = (s[tid] + s[128 + tid]) + (s[256 + tid] + s[384 + tid]);
    if (tid == 128) out[128] = (s[512] + s[513]) + (s[514] + s[515]);
    tc::fence_before();
    __syncthreads();
}

template <int W, int N>
int launch_proj_bwd(const ProjBwdArgs& a, int* blocks, cudaStream_t st) {
    const size_t smem = sizeof(ProjBwdSmem<W>);
    static_assert(sizeof(ProjBwdSmem<W>) <= 113 * 1024, "two CTAs per SM");
    cudaFuncSetAttribute(k_fno_proj_bwd<W, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int tiles = a.batch * (N < 128 ? 1 : N / 128), most = 2 * sm_count();
    *blocks = tiles < most ? tiles : most;
    k_fno_proj_bwd<W, N><<<*blocks, THREADS, smem, st>>>(a);
    return check_launch("fno projection backward");
}

// ---- weight gradients over the points ----------------------------------------------------
// part[block][o][c] = sum over the block's units of g[b][o][p] x[b][c][p] and rows[block][o] = sum of
// g: a unit is `seg` points of one trajectory, 64 per chunk.  The rows of g in three
// stacked pieces are the accumulator lanes, those of x the columns:
//   MO = 32:  lanes (hi, mid, lo) x columns (hi, mid, lo), one product;
//   MO = 64:  lanes (hi, lo) x (hi, mid, lo), and (mid, 64 rows of zeros) x the same, one order
//             further, so that in either half of the lanes a column group is one order;
//   MO = 128: hi x (hi, mid, lo), mid x (hi, mid, lo) one order further, lo x (hi, mid) two.
// A unit's sums are read into registers (with its two scales) while the next unit's products
// run into the other half of the columns, so no chain in the tensor cores is longer than a
// row; g is scaled to 128 instead of 256, so that 512 full-scale terms stay below 2^24 (tc.cuh).
// 16 warps split; the last of them also issues (8 or 12 instructions per chunk).  A 17th warp
// for that cost every thread 32 registers (128 -> 96), and reading the sums before the next
// unit started left the tensor cores idle: 33 -> 30 us (64 x 64) and 37 -> 35 us (128 x 64) at
// 256 rows of 512 points (31.5 and 38.2 since fp16 pieces and their eight products).
struct WgradArgs {
    const float* g;      // [batch][MO][n]
    const float* gmax;   // [tiles per row][batch]
    const float* x;      // [batch][W][n], through GELU for the layers (MO = W)
    const float* xmax;   // [tiles per row][batch]
    float* part;         // [blocks][MO][W]
    float* rows;         // [blocks][MO]
    int batch, n, seg;
};
constexpr int WG_WORKERS = 512;
template <int MO, int W>
struct WgradSmem {
    static constexpr int GP = (MO == 64 ? 4 : 3) * MO * 16 + 16, XP = 3 * W * 16 + 16;  // plane pitches
    static constexpr int MID = (MO == 64 ? 2 : 1) * MO * 16, LO = (MO == 64 ? 1 : 2) * MO * 16;  // of g's rows
    struct Buf {
        alignas(128) unsigned char g[8 * GP];
        alignas(128) unsigned char x[8 * XP];
    } buf[2];
    unsigned char pad[2048];  // (lanes past the pieces read on: what they hold is not used)
    uint64_t bar[2];
    uint32_t tmem;
};

template <int MO, int W>
__global__ void __launch_bounds__(WG_WORKERS, 1) k_fno_wgrad(WgradArgs a) {
    extern __shared__ __align__(128) unsigned char fno_smem[];
    using Smem = WgradSmem<MO, W>;
    Smem& S = *reinterpret_cast<Smem*>(fno_smem);
    constexpr int GP = Smem::GP, XP = Smem::XP, COLS = W == 64 ? 256 : 128;  // (of one unit's sums)
    // pieces of 8 points of a row of g (the first MO rows) or x, per thread and chunk; the
    // last round may be half a block
    constexpr int ITEMS = (MO + W) * 8, IT = (ITEMS + WG_WORKERS - 1) / WG_WORKERS;
    const int tid = threadIdx.x;
    if (tid < 32) tc::tmem_alloc(&S.tmem, 2 * COLS);
    if (tid == 0) {
        tc::mbar_init(&S.bar[0], 1);
        tc::mbar_init(&S.bar[1], 1);
        tc::mbar_init_fence();
    }
    if (MO == 64) {  // the rows of zeros of both buffers' 8 planes
        for (int i = tid; i < 2 * 8 * 64; i += WG_WORKERS)
            *reinterpret_cast<uint4*>(S.buf[i >> 9].g + (i >> 6 & 7) * GP + (192 + (i & 63)) * 16) = make_uint4(0, 0, 0, 0);
        tc::fence_smem();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t d = S.tmem;
    const int per_row = a.n / a.seg, units = a.batch * per_row, chunks = a.seg / 64;
    const int mine = blockIdx.x < units ? (units - blockIdx.x + gridDim.x - 1) / gridDim.x * chunks : 0;
    auto issue = [&](int n) {  // chunk n's products (one thread)
        const uint64_t g = tc::smem_desc(tc::smem_u32(S.buf[n & 1].g), GP, 128);
        const uint64_t x = tc::smem_desc(tc::smem_u32(S.buf[n & 1].x), XP, 128);
        const uint32_t du = d + (n / chunks & 1) * COLS;
        const bool first = n % chunks == 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t b = tc::desc_at(x, 2 * k * XP), gk = tc::desc_at(g, 2 * k * GP);
            const bool add = !first || k > 0;
            constexpr uint32_t i3 = tc::instr_desc(128, 3 * W), i2 = tc::instr_desc(128, 2 * W);
            tc::mma(du, gk, b, i3, add);
            if (MO >= 64) {
                const uint64_t mid = tc::desc_at(gk, Smem::MID);
                if (add) {
                    tc::mma(du + W, mid, b, i3, true);
                } else {  // (the first to write the last W columns)
                    tc::mma(du + W, mid, b, i2, true);
                    tc::mma(du + 3 * W, mid, tc::desc_at(b, 2 * W * 16), tc::instr_desc(128, W), false);
                }
            }
            if (MO == 128) tc::mma(du + 2 * W, tc::desc_at(gk, Smem::LO), b, i2, true);
        }
        tc::commit(&S.bar[n & 1]);
    };
    const int c8 = tid & 7, r0 = tid >> 3;
    constexpr bool full = (MO + W) % 64 == 0;
    bool fail = false;
    uint32_t used = 0;
    // lane, quarter of the columns, piece of the lane
    constexpr int CQ = W / 4;
    const int t = tid & 127, quarter = tid >> 7, group = t / MO;
    // of the lane's piece (MO = 64: the upper half is lo)
    const float order = group == 0 ? 1.f : (MO == 32 && group == 1 ? tc::DOWN : tc::DOWN * tc::DOWN);
    float acc[CQ], rs[IT];
#pragma unroll
    for (int i = 0; i < CQ; ++i) acc[i] = 0.f;
#pragma unroll
    for (int i = 0; i < IT; ++i) rs[i] = 0.f;
    // chunks are loaded two ahead (one where a thread's share is large: registers)
    constexpr int DEPTH = IT <= 2 ? 2 : 1;
    float4 v[DEPTH][IT][2];
    auto load = [&](int n, float4(&w)[IT][2]) {
        if (n >= mine) return;
        const int u = blockIdx.x + n / chunks * gridDim.x, b = u / per_row;
        const int p = (u % per_row) * a.seg + (n % chunks) * 64 + 8 * c8;
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int r = r0 + 64 * i;
            if (full || r < MO + W) {
                const float4* s = reinterpret_cast<const float4*>(
                    (MO % 64 == 0 ? 64 * i < MO : r < MO) ? a.g + ((int64_t)b * MO + r) * a.n + p : a.x + ((int64_t)b * W + r - MO) * a.n + p);
                w[i][0] = ldg_na4(s);
                w[i][1] = ldg_na4(s + 1);
            }
        }
    };
    float sg = 1.f, sx = 1.f;
    const int nq = a.n < 128 ? 1 : a.n / 128;
    // the sums of the unit that ended with chunk n (in buffer `buf`)
    auto drain = [&](int n, int buf, float f) {
        if (!fail) fail = !tc::mbar_wait(&S.bar[buf], (used >> buf) & 1);
        tc::fence_after();
        if (fail) f = __int_as_float(0x7fffffff);
        const uint32_t dl = d + (n / chunks & 1) * COLS + ((uint32_t)(t & 96) << 16) + quarter * CQ;
        f *= order;
#pragma unroll
        for (int c = 0; c < CQ; c += 8) {
            float q0[8], q1[8], q2[8], q3[8];
            tc::tmem_ld8(dl + c, q0);
            tc::tmem_ld8(dl + c + W, q1);
            tc::tmem_ld8(dl + c + 2 * W, q2);
            if (MO >= 64) tc::tmem_ld8(dl + c + 3 * W, q3);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float s = MO >= 64 ? fmaf(q3[i], tc::DOWN, q2[i]) : q2[i];
                acc[c + i] += fmaf(fmaf(s, tc::DOWN, q1[i]), tc::DOWN, q0[i]) * f;
            }
        }
    };
    auto chunk = [&](int n, int buf, float4(&w)[IT][2]) {
        const float f_prev = sg * (1.f / 128.f) * (sx * (1.f / 256.f));
        if (n % chunks == 0) {  // the unit's scales: the max over its tiles
            const int u = blockIdx.x + n / chunks * gridDim.x, b = u / per_row;
            const int q0 = a.n < 128 ? 0 : (u % per_row) * a.seg / 128, q1 = a.seg < 128 ? q0 + 1 : q0 + a.seg / 128;
            float mg = 0.f, mx = 0.f;
            for (int q = q0; q < q1 && q < nq; ++q) {
                mg = fmaxf(mg, __ldg(a.gmax + (int64_t)q * a.batch + b));
                mx = fmaxf(mx, __ldg(a.xmax + (int64_t)q * a.batch + b));
            }
            sg = tc::pow2_above(mg);
            sx = tc::pow2_above(mx);
        }
        if (n >= 2) {
            if (!fail) fail = !tc::mbar_wait(&S.bar[buf], (used >> buf) & 1);
            used ^= 1u << buf;
        }
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int r = r0 + 64 * i;  // (a warp's rows are all of g or all of x: known here where MO is 64 or 128)
            if (full || r < MO + W) {
                const bool is_g = MO % 64 == 0 ? 64 * i < MO : r < MO;
                float2 e[4] = {make_float2(w[i][0].x, w[i][0].y), make_float2(w[i][0].z, w[i][0].w),
                               make_float2(w[i][1].x, w[i][1].y), make_float2(w[i][1].z, w[i][1].w)};
                if (is_g) {
                    rs[i] += ((e[0].x + e[0].y) + (e[1].x + e[1].y)) + ((e[2].x + e[2].y) + (e[3].x + e[3].y));
                } else if (MO == W) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) e[j] = act::gelu2(e[j]);
                }
                const float inv = is_g ? 128.f / sg : 256.f / sx;
                uint32_t hi[4], mid[4], lo[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) tc::split2(e[j], make_float2(inv, inv), hi[j], mid[j], lo[j]);
                unsigned char* s = is_g ? S.buf[buf].g + c8 * GP + r * 16 : S.buf[buf].x + c8 * XP + (r - MO) * 16;
                *reinterpret_cast<uint4*>(s) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(s + (is_g ? Smem::MID : W * 16)) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
                *reinterpret_cast<uint4*>(s + (is_g ? Smem::LO : 2 * W * 16)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
        load(n + DEPTH, w);
        tc::fence_smem();
        tc::fence_before();
        if (tid < WG_WORKERS - 32) {
            hand_over<WG_WORKERS - 32>(buf);
        } else {
            take_over<WG_WORKERS - 32>(buf);
            if (tc::elect()) {
                tc::fence_after();
                issue(n);
            }
            __syncwarp();
        }
        // the unit before this one, while this one's products run into the other columns
        if (n > 0 && n % chunks == 0) drain(n - 1, buf ^ 1, f_prev);
    };
    load(0, v[0]);
    if (DEPTH == 2) load(1, v[DEPTH - 1]);
#pragma unroll 1
    for (int n = 0; n < mine; n += 2) {
        chunk(n, 0, v[0]);
        if (n + 1 < mine) chunk(n + 1, 1, v[DEPTH - 1]);
    }
    if (mine > 0) drain(mine - 1, (mine - 1) & 1, sg * (1.f / 128.f) * (sx * (1.f / 256.f)));
    tc::fence_before();
    // the lanes' pieces added up (hi, then mid and lo), then the block's slot
    float* s = reinterpret_cast<float*>(S.buf[0].g);  // [128][W + 1]; every product is done
    static_assert(sizeof(float) * 128 * (W + 1) <= sizeof(S.buf), "scratch");
    worker_sync<WG_WORKERS>();
#pragma unroll
    for (int i = 0; i < CQ; ++i) s[t * (W + 1) + quarter * CQ + i] = acc[i];
    worker_sync<WG_WORKERS>();
    float* out = a.part + (int64_t)blockIdx.x * MO * W;
    for (int i = tid; i < MO * W; i += WG_WORKERS) {
        const int o = i / W, c = i % W;
        float r = s[o * (W + 1) + c];
        if (MO == 32) r += s[(32 + o) * (W + 1) + c] + s[(64 + o) * (W + 1) + c];
        if (MO == 64) r += s[(64 + o) * (W + 1) + c];
        out[i] = r;
    }
#pragma unroll
    for (int i = 0; i < IT; ++i) {
        rs[i] += __shfl_xor_sync(0xffffffffu, rs[i], 1);
        rs[i] += __shfl_xor_sync(0xffffffffu, rs[i], 2);
        rs[i] += __shfl_xor_sync(0xffffffffu, rs[i], 4);
        if (c8 == 0 && r0 + 64 * i < MO) a.rows[(int64_t)blockIdx.x * MO + r0 + 64 * i] = rs[i];
    }
    if (tid < 32) tc::tmem_free(d, 2 * COLS);
}

// a unit: 128 points while that leaves a block few units, else as many as a row has (fewer
// reads of the accumulators)
inline int wgrad_seg(int batch, int n) {
    if (n <= 128) return n;
    return (int64_t)batch * (n / 128) <= 16 * (int64_t)sm_count() ? 128 : n;
}

template <int MO, int W>
int run_wgrad(WgradArgs a, int* blocks, cudaStream_t st) {
    const size_t smem = sizeof(WgradSmem<MO, W>);
    static_assert(sizeof(WgradSmem<MO, W>) <= 227 * 1024, "shared memory");
    cudaFuncSetAttribute(k_fno_wgrad<MO, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    a.seg = wgrad_seg(a.batch, a.n);
    const int64_t units = (int64_t)a.batch * (a.n / a.seg);
    *blocks = units < sm_count() ? (int)units : sm_count();
    k_fno_wgrad<MO, W><<<*blocks, WG_WORKERS, smem, st>>>(a);
    return check_launch("fno weight gradient");
}

// ---- Fourier weight gradients -------------------------------------------------------------
// dW[c][o][k] = (c_k / n) sum_b conj(X[k][b][c]) G[k][b][o] (c_0 = 1, c_k = 2; torch's convention for
// complex gradients), all four layers: block = mode, layer, 16 of the o; thread: 4 c x 1 o, the
// factors Re X and Im X in separate packed accumulators (two packed operations per complex
// product), the next 32 trajectories loaded while these are multiplied.  67 MB are read (10.4 us
// at the copy rate for 256 trajectories of 64 channels and 16 modes); bound by the loads' and
// barriers' latency: 23.2 us with four warps a scheduler, 27.4 with two (32 of the o per
// block, 16 trajectories a time).
struct ModesGradArgs {
    const float2* x;  // [4][modes][batch][W]
    const float2* g;  // [4][modes][batch][W]
    float2* out[4];   // [W][W][modes] (NULL: not wanted)
    int batch, modes, n;
};
template <int W>
__global__ void __launch_bounds__(W * 4) k_fno_modes_grad(ModesGradArgs a) {
    constexpr int TB = 32, T = W * 4, LX = TB * W / T, LG = TB * 16 / T;
    __shared__ float2 X[TB][W], G[TB][16];
    const int k = blockIdx.x, l = blockIdx.y, o0 = blockIdx.z * 16;
    if (!a.out[l]) return;
    const int64_t base = ((int64_t)l * a.modes + k) * a.batch * W;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // o: tx; c: ty + i W / 4
    float2 rx[LX], rg[LG];
    auto load = [&](int b0) {
#pragma unroll
        for (int i = 0; i < LX; ++i) {
            const int e = threadIdx.x + i * T, b = b0 + e / W;
            rx[i] = b < a.batch ? __ldg(a.x + base + (int64_t)b * W + e % W) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < LG; ++i) {
            const int e = threadIdx.x + i * T, b = b0 + e / 16;
            rg[i] = b < a.batch ? __ldg(a.g + base + (int64_t)b * W + o0 + e % 16) : make_float2(0.f, 0.f);
        }
    };
    float2 tre[4], tim[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        tre[i] = tim[i] = make_float2(0.f, 0.f);
    load(0);
    for (int b0 = 0; b0 < a.batch; b0 += TB) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < LX; ++i) (&X[0][0])[threadIdx.x + i * T] = rx[i];
#pragma unroll
        for (int i = 0; i < LG; ++i) (&G[0][0])[threadIdx.x + i * T] = rg[i];
        __syncthreads();
        if (b0 + TB < a.batch) load(b0 + TB);
        float2 re[4], im[4];  // (a chunk's sum first: shorter chains)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            re[i] = im[i] = make_float2(0.f, 0.f);
#pragma unroll
        for (int b = 0; b < TB; ++b) {
            const float2 g = G[b][tx];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 x = X[b][ty + i * (W / 4)];
                re[i] = __ffma2_rn(make_float2(x.x, x.x), g, re[i]);
                im[i] = __ffma2_rn(make_float2(x.y, x.y), g, im[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            tre[i] = __fadd2_rn(tre[i], re[i]);
            tim[i] = __fadd2_rn(tim[i], im[i]);
        }
    }
    const float s = (k == 0 ? 1.f : 2.f) / (float)a.n;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        // conj(x) g = (x.x g.x + x.y g.y, x.x g.y - x.y g.x)
        a.out[l][((int64_t)(ty + i * (W / 4)) * W + o0 + tx) * a.modes + k] =
            make_float2((tre[i].x + tim[i].y) * s, (tre[i].y - tim[i].x) * s);
}

// ---- the blocks' partial sums, added in a fixed order ---------------------------------------
// job j: dst[i] = sum over p < count of src[p * stride + i], i < n.  Block: 32 outputs, 32 slices.
constexpr int MAX_JOBS = 11;
struct ReduceArgs {
    const float* src[MAX_JOBS];
    float* dst[MAX_JOBS];
    int stride[MAX_JOBS], count[MAX_JOBS], n[MAX_JOBS], first[MAX_JOBS + 1];
    int jobs;
};
__global__ void __launch_bounds__(1024) k_fno_reduce(ReduceArgs a) {
    __shared__ float s[32][33];
    int j = 0;
    while (j + 1 < a.jobs && (int)blockIdx.x >= a.first[j + 1]) ++j;
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const int i = (blockIdx.x - a.first[j]) * 32 + lane;
    float v = 0.f;
    if (i < a.n[j]) {
        const float* src = a.src[j] + i;
#pragma unroll 5
        for (int p = slice; p < a.count[j]; p += 32) v += __ldg(src + (int64_t)p * a.stride[j]);
    }
    s[slice][lane] = v;
    __syncthreads();
    if (threadIdx.x < 32 && i < a.n[j]) {
        float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 32; ++q) t[q & 3] += s[q][lane];
        a.dst[j][i] = (t[0] + t[1]) + (t[2] + t[3]);
    }
}

// Layer 0 and the lift from the six sums per channel: s[0..2][o] = sum dL/dz {u, grid, 1},
// s[3..5][c] = sum dL/dh {u, grid, 1}, with h[c] = w[c][0] u + w[c][1] grid + b[c].  Outputs
// that are NULL are not wanted.
template <int W>
__global__ void __launch_bounds__(256) k_fno_lift_grad(const float* __restrict__ s, const float* __restrict__ w,
                                                       const float* __restrict__ bias, float* __restrict__ g_w0,
                                                       float* __restrict__ g_b0, float* __restrict__ g_fc0_w,
                                                       float* __restrict__ g_fc0_b) {
    for (int i = blockIdx.x * 256 + threadIdx.x; i < W * W; i += gridDim.x * 256) {
        const int o = i / W, c = i % W;
        if (g_w0) g_w0[i] = fmaf(w[2 * c], s[o], fmaf(w[2 * c + 1], s[W + o], bias[c] * s[2 * W + o]));
        if (c == 0) {
            if (g_b0) g_b0[o] = s[2 * W + o];
            if (g_fc0_w) {
                g_fc0_w[2 * o] = s[3 * W + o];
                g_fc0_w[2 * o + 1] = s[4 * W + o];
            }
            if (g_fc0_b) g_fc0_b[o] = s[5 * W + o];
        }
    }
}

// scratch of the backward, in floats
template <int W>
struct BwdWork {
    int64_t prep, wt, mixed, gm, mmax, g1, gz, gzmax, g1max, sums, part, rows, six, total;
    BwdWork(int64_t B, int64_t n, int64_t M) {
        const int64_t nq = n < 128 ? 1 : n / 128, blocks = 2 * (int64_t)sm_count();
        int64_t at = 0;
        auto take = [&](int64_t floats) {
            const int64_t r = at;
            at += (floats + 3) / 4 * 4;  // (every array 16-byte aligned)
            return r;
        };
        prep = take((int64_t)sizeof(Prep<W>) / 4);
        wt = take(2 * 4 * M * W * W);
        mixed = take(2 * M * B * W);
        gm = take(2 * 4 * M * B * W);       // modes of dL/dz of every layer
        mmax = take(4 * B);
        g1 = take(B * 128 * n);
        gz = take(2 * B * W * n);           // dL/dz of two layers in turn
        gzmax = take(2 * nq * B);
        g1max = take(nq * B);
        sums = take(blocks * 132);
        part = take(blocks * (128 * W + 3 * W * W));
        rows = take(blocks * (128 + 3 * W));
        six = take(blocks * 6 * W + 6 * W);
        total = at;
    }
};

template <int W>
int run_backward(const inc_fno_desc* d, const float* u, const float* g_y, const float* z, const float* xm,
                 const float* tmax, const inc_fno_grads* gr, float* work, cudaStream_t st) {
    const int B = d->rows, n = d->n, M = d->modes, nq = n < 128 ? 1 : n / 128;
    const int64_t state = (int64_t)B * W * n, modes = (int64_t)M * B * W;
    const BwdWork<W> o(B, n, M);
    Prep<W>* prep = reinterpret_cast<Prep<W>*>(work + o.prep);
    float2* wt = reinterpret_cast<float2*>(work + o.wt);
    float2* mixed = reinterpret_cast<float2*>(work + o.mixed);
    float2* gm = reinterpret_cast<float2*>(work + o.gm);
    float* gz = work + o.gz;
    float* gzmax = work + o.gzmax;
    const int64_t most = 2 * (int64_t)sm_count();
    PrepArgs pa{};
    for (int l = 0; l < 4; ++l) {
        pa.modes_w[l] = reinterpret_cast<const float2*>(d->modes_w[l]);
        pa.w[l] = d->w[l];
    }
    pa.fc1 = d->fc1_w;
    pa.wt = wt;
    pa.zero = work + o.mmax;
    pa.batch = B;
    pa.n = n;
    pa.modes = M;
    int rc = run_prep<W, true>(pa, prep, st);
    if (rc) return rc;
    ReduceArgs ra{};
    auto job = [&](const float* src, float* dst, int stride, int count, int len) {
        if (!dst) return;
        const int j = ra.jobs++;
        ra.src[j] = src;
        ra.dst[j] = dst;
        ra.stride[j] = stride;
        ra.count[j] = count;
        ra.n[j] = len;
        ra.first[j + 1] = ra.first[j] + (len + 31) / 32;
    };
    int blocks = 0;
    {  // the projection: dL/dz of layer 3 into gz[1] (layer l's in gz[l & 1])
        const ProjBwdArgs p{z + 3 * state, tmax + 3 * nq * B, prep->fc1, prep->scale + 4, d->fc1_b, d->fc2_w, g_y,
                            work + o.g1, work + o.g1max, gz + state, gzmax + nq * B, work + o.sums, B};
        switch (n) {
            case 64: rc = launch_proj_bwd<W, 64>(p, &blocks, st); break;
            case 128: rc = launch_proj_bwd<W, 128>(p, &blocks, st); break;
            case 256: rc = launch_proj_bwd<W, 256>(p, &blocks, st); break;
            default: rc = launch_proj_bwd<W, 512>(p, &blocks, st); break;
        }
        if (rc) return rc;
        job(work + o.sums, gr->fc2_w, 132, blocks, 128);
        job(work + o.sums + 128, gr->fc2_b, 132, blocks, 1);
        float* part = work + o.part;
        float* rows = work + o.rows;
        if (gr->fc1_w || gr->fc1_b) {
            rc = run_wgrad<128, W>(WgradArgs{work + o.g1, work + o.g1max, z + 3 * state, tmax + 3 * nq * B, part, rows, B, n, 0}, &blocks, st);
            if (rc) return rc;
            job(part, gr->fc1_w, 128 * W, blocks, 128 * W);
            job(rows, gr->fc1_b, 128, blocks, 128);
        }
    }
    // only what is asked for: the lift's gradients and layer 0's come from its adjoint's sums; the
    // chain of adjoints ends at the lowest layer that something asks of
    const bool lift = gr->u || gr->w[0] || gr->b[0] || gr->fc0_w || gr->fc0_b;
    int lowest = 0;
    while (lowest < 4 && !(lowest == 0 && lift) && !gr->modes_w[lowest] && !gr->w[lowest] && !gr->b[lowest]) ++lowest;
    bool modes_wanted = false;
    for (int l = 0; l < 4; ++l) modes_wanted = modes_wanted || gr->modes_w[l];
    for (int l = 3; l >= lowest; --l) {
        const bool on = l > lowest || (l == 0 && lift);  // the adjoint goes on below this layer
        const float* g = gz + (l & 1) * state;
        const float* gmx = gzmax + (l & 1) * nq * B;
        if (on || gr->modes_w[l]) {
            rc = run_modes<W, false>(ModesArgs{g, gmx, prep->transform, gm + l * modes, B * W, B, M}, n, st);
            if (rc) return rc;
        }
        if (on) {
            rc = run_mix<W>(gm + l * modes, wt + (int64_t)l * M * W * W, mixed, work + o.mmax + l * B, B, n, M, st);
            if (rc) return rc;
        }
        if (l > 0 && (gr->w[l] || gr->b[l])) {
            float* part = work + o.part + most * (128 * W + (l - 1) * W * W);
            float* rows = work + o.rows + most * (128 + (l - 1) * W);
            rc = run_wgrad<W, W>(WgradArgs{g, gmx, z + (l - 1) * state, tmax + (int64_t)(l - 1) * nq * B, part, rows, B, n,
                                           0}, &blocks, st);
            if (rc) return rc;
            job(part, gr->w[l], W * W, blocks, W * W);
            job(rows, gr->b[l], W, blocks, W);
        }
        if (!on) break;
        LayerArgs a{};
        a.x = g;
        a.xmax = gmx;
        a.w = prep->w[l];
        a.inverse = prep->inverse[0];
        a.wscale = prep->scale + l;
        a.mixed = mixed;
        a.mixed_max = work + o.mmax + l * B;
        a.batch = B;
        a.modes = M;
        if (l > 0) {
            a.zprev = z + (l - 1) * state;
            a.out = gz + ((l - 1) & 1) * state;
            a.tmax = gzmax + ((l - 1) & 1) * nq * B;
            rc = run_layer<W, false, BWD, true>(a, n, st);
        } else {
            a.u = u;
            a.grid = d->grid;
            a.grid_stride = d->grid_stride;
            a.fc0_w = d->fc0_w;
            a.fc0_b = d->fc0_b;
            a.g_u = gr->u;
            a.sums = work + o.six + 6 * W;
            rc = run_layer<W, false, BWD0, true>(a, n, st);
        }
        if (rc) return rc;
    }
    const bool six = gr->w[0] || gr->b[0] || gr->fc0_w || gr->fc0_b;
    if (six) job(work + o.six + 6 * W, work + o.six, 6 * W, tile_grid(B, nq), 6 * W);
    if (ra.jobs) k_fno_reduce<<<ra.first[ra.jobs], 1024, 0, st>>>(ra);
    if (six)
        k_fno_lift_grad<W><<<W * W / 256, 256, 0, st>>>(work + o.six, d->fc0_w, d->fc0_b, gr->w[0], gr->b[0], gr->fc0_w,
                                                       gr->fc0_b);
    ModesGradArgs mg{};
    mg.x = reinterpret_cast<const float2*>(xm);
    mg.g = gm;
    for (int l = 0; l < 4; ++l) mg.out[l] = reinterpret_cast<float2*>(gr->modes_w[l]);
    mg.batch = B;
    mg.modes = M;
    mg.n = n;
    if (modes_wanted) k_fno_modes_grad<W><<<dim3(M, 4, W / 16), W * 4, 0, st>>>(mg);
    return check_launch("fno gradients");
}

}  // namespace fno
}  // namespace inc

using namespace inc;

extern "C" int64_t inc_fno_backward_work_size(const inc_fno_desc* d) {
    if (!d || d->rows <= 0 || !fno::supported(d->width, d->n, d->modes)) return -1;
    return d->width == 64 ? fno::BwdWork<64>(d->rows, d->n, d->modes).total
                          : fno::BwdWork<32>(d->rows, d->n, d->modes).total;
}

extern "C" int inc_fno_backward(const inc_fno_desc* d, const float* u, const float* g_y, const float* z,
                                const float* x_modes, const float* tmax, const inc_fno_grads* g, float* work,
                                void* stream) {
    const int rc = fno::check_fno(d);
    if (rc) return rc;
    bool ok = u && g_y && z && x_modes && tmax && g && work && (reinterpret_cast<uintptr_t>(work) & 15u) == 0 &&
              (reinterpret_cast<uintptr_t>(z) & 15u) == 0 && (reinterpret_cast<uintptr_t>(x_modes) & 7u) == 0;
    for (int l = 0; ok && l < 4; ++l) ok = (reinterpret_cast<uintptr_t>(g->modes_w[l]) & 7u) == 0;
    if (!ok) {
        set_error("fno_backward: bad arguments");
        return INC_E_INVALID;
    }
    cudaStream_t st = as_stream(stream);
    return d->width == 64 ? fno::run_backward<64>(d, u, g_y, z, x_modes, tmax, g, work, st)
                          : fno::run_backward<32>(d, u, g_y, z, x_modes, tmax, g, work, st);
}
