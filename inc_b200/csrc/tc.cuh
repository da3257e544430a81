// Fifth-generation tensor-core (tcgen05) helpers for FP32-accurate contractions.
//
// An FP32 operand is split into three fp16 pieces.  With a power of two s >= max|x| of the
// operand's scale group (the elements that share one scale along the contraction),
//   x / s * 256 = hi + 2^-14 mid + 2^-28 lo:
// hi is an integer of magnitude <= 256, mid the remainder (<= 1/2) rounded to fp16's 11 bits,
// lo what mid leaves, rounded to 11 bits; the powers of two keep the lower pieces in fp16's
// range.  An element x is represented to 2^-24 |x| (half a unit in the last place of FP32), whatever
// its size beside the group's maximum, down to 2^-36 of it; below that to 2^-61 of the
// maximum.  (Three bf16 pieces on the same grid, as these once were, keep 2^-27 of the maximum
// above 1/512 of it and 16 bits below: an output whose terms are all small, such as one
// fed by a channel of small activations, then lost up to 8 of FP32's 24 bits.)
//
// Eight of the nine piece products are accumulated, by order (the number of 2^-14): order 0 is
// hi.hi alone, whose partial sums are integers below 2^24 for up to 256 full-scale terms, so
// the accumulator's truncation never acts on it; order 1 hi.mid and mid.hi; order 2 hi.lo,
// mid.mid and lo.hi; order 3 mid.lo and lo.mid.  The one left out, lo.lo, is below 2^-24 |a b|.
// Truncation acts on the orders from 1 up, 2^-9 below order 0 for operands near their maxima
// (2^-33 of the sum), and at FP32's level for operands so small that their hi is 0.  Orders
// are kept in columns of their own, or gathered in one accumulator from the highest down
// with its input scaled by 2^-14 at each step (mma_scaled).  Against an FP32 fused multiply-add
// chain of the same length, which rounds at every term, the result is no further off.
//
// Operand tiles live in shared memory as [rows][K] fp16 in 8-row x 16-byte core
// matrices without swizzle: element (r, k) at (k / 8) * plane + r * 16 + (k % 8) * 2
// bytes, plane = rows * 16.  A row is 16 bytes from the next, so a tile shifted by
// one row (a convolution tap) is the same tile with the start address moved by 16.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace inc {
namespace tc {

INC_DEV uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// generic-proxy writes to shared memory visible to the tensor core's reads
INC_DEV void fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
INC_DEV void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
INC_DEV void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- tensor memory -------------------------------------------------------------
// One warp allocates ncols (a power of two >= 32) columns; the base goes to *dst (shared).
INC_DEV void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
INC_DEV void tmem_free(uint32_t base, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols) : "memory");
}
// 16 consecutive columns of this warp's 32 lanes (lane = accumulator row)
INC_DEV void tmem_ld16(uint32_t addr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
INC_DEV void tmem_ld8(uint32_t addr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
INC_DEV void tmem_ld(uint32_t addr, float (&v)[16]) { tmem_ld16(addr, v); }
INC_DEV void tmem_ld(uint32_t addr, float (&v)[8]) { tmem_ld8(addr, v); }
INC_DEV void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---- mbarrier --------------------------------------------------------------------
INC_DEV void mbar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
INC_DEV void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// Waits for the phase of this parity; false when it did not complete within the limit
// (try_wait suspends for a while by itself, so the limit is seconds).
INC_DEV bool mbar_wait(uint64_t* b, uint32_t parity) {
    const uint32_t a = smem_u32(b);
    for (int i = 0; i < (1 << 20); ++i) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Bulk copy of a contiguous global array (16-byte aligned, bytes a multiple of 16) into this
// CTA's shared memory; `b` expects its bytes (mbar_expect) and completes when they are there.
INC_DEV void mbar_expect(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
INC_DEV void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(b))
                 : "memory");
}

// ---- matrix instructions -----------------------------------------------------------
// Shared-memory descriptor of a tile in core matrices without swizzle: `lead` and
// `stride` are the byte distances of neighbouring core matrices along K and along the
// rows (K-major), or along the rows' 8-groups of K and along the columns (MN-major).
INC_DEV uint64_t smem_desc(uint32_t addr, uint32_t lead, uint32_t stride) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lead >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((stride >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// FP32 accumulator, fp16 operands, M x N tile; a_mn / b_mn: operand stored MN-major
__host__ __device__ constexpr uint32_t instr_desc(int M, int N, bool a_mn = false, bool b_mn = false) {
    return (1u << 4) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}
// the same tile `bytes` further on (a multiple of 16; within shared memory)
INC_DEV uint64_t desc_at(uint64_t d, uint32_t bytes) { return d + (bytes >> 4); }
// True for one lane of a full warp, the same at every call.  Matrix instructions stand
// under this and not under a comparison of the thread's index: their operands are
// per-warp registers, and only under an election does the compiler know that one
// thread is active; otherwise each instruction becomes a loop over the active lanes.
// Measured with 16 warps of dense FP32 work on the SM (M = 128, N = 96): 95 clocks an
// instruction against 540 to 890 (56 with an idle SM, either way).
INC_DEV bool elect() {
    uint32_t r;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(r));
    return r != 0;
}
// D[tmem] (+)= A B^T over K = 16; one thread issues (elect)
INC_DEV void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
// D[tmem] = 2^-14 D + A B^T: the step from one order of the pieces' products to the one below it
INC_DEV void mma_scaled(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.eq.b32 p, 0, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%4, %4, %4, %4}, p, 14;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(0)
        : "memory");
}
// arrives on `b` when every matrix instruction this thread issued has finished
INC_DEV void commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(b))
                 : "memory");
}

// ---- the three-piece split -----------------------------------------------------------
// A power of two >= m (m >= 0): the scale s of a group with max|x| = m.  Groups below
// 2^-100 use that (a product of two such groups is below FP32's smallest normal number);
// above 2^127, and for an infinite m or NaN, 2^127, so that 256 / s stays a normal number.
INC_DEV float pow2_above(float m) {
    const uint32_t e = (__float_as_uint(fminf(m, 1.7014118346046923e38f)) + 0x007FFFFFu) & 0x7F800000u;
    return fmaxf(__uint_as_float(e), 7.888609052210118e-31f);
}

// two values packed as fp16, rounded to nearest (a in the low half)
INC_DEV uint32_t cvt_f16x2(float a, float b) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
// The step between two orders of the pieces, 2^14 up and down
constexpr float UP = 16384.f, DOWN = 1.f / 16384.f;
// x * inv (a power of two, |x * inv| <= 256) of two values -> their pieces, packed.
// The products inside the fused operations are exact.
INC_DEV void split2(float2 x, float2 inv, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    constexpr float M = 12582912.f;  // 1.5 * 2^23: to integers
    const float2 y = __fmul2_rn(x, make_float2(inv.x * UP, inv.y * UP));
    const float2 t = __ffma2_rn(y, make_float2(DOWN, DOWN), make_float2(M, M));
    const float2 h = make_float2(t.x - M, t.y - M);
    hi = cvt_f16x2(h.x, h.y);  // integers <= 256: exact
    const float2 r = __ffma2_rn(h, make_float2(-UP, -UP), y);
    mid = cvt_f16x2(r.x, r.y);
    const float2 m = __half22float2(*reinterpret_cast<const __half2*>(&mid));
    const float2 q = __ffma2_rn(m, make_float2(-UP, -UP), make_float2(r.x * UP, r.y * UP));
    lo = cvt_f16x2(q.x, q.y);
}
// eight values -> 16 bytes of each piece
INC_DEV void split8(const float (&x)[8], float inv, uint4& hi, uint4& mid, uint4& lo) {
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        split2(make_float2(x[2 * i], x[2 * i + 1]), make_float2(inv, inv), h[i], m[i], l[i]);
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    mid = make_uint4(m[0], m[1], m[2], m[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

}  // namespace tc
}  // namespace inc
