// Tensor-core additions to the prelude, for the chunked kernels: tf32 matrix products (tcgen05) of an operand in
// Tensor Memory or shared memory with one in shared memory, accumulated in Tensor Memory.
//
// Shared-memory operands are K-major without swizzle: 8 x 4-element (128-byte) core matrices, element (row, k) at
// (k / 4) * lbo + (row / 8) * 128 + (row % 8) * 16 + (k % 4) * 4 bytes; lbo is free, and padding it by 16 bytes makes
// the producers' stores free of bank conflicts.  A product covers 8 values of k; M is 128 rows (the lanes of Tensor
// Memory), N a multiple of 16.  Measured on a B200, cycles per product in a row: first operand in Tensor Memory N / 2
// (N = 16: 10), in shared memory 40 up to N = 32, 48 at 64, 64 at 128 (its 4 KB and the other's 32 N bytes at 128 bytes a
// cycle); operands are truncated to tf32 (their low 13 bits are ignored), which the two-term splits below rely on.
#ifndef FRNN_EMU
FRNN_DEV u32 frnn_f32_bits(float x) { return __float_as_uint(x); }
FRNN_DEV float frnn_bits_f32(u32 x) { return __uint_as_float(x); }
FRNN_DEV float frnn_tf32_trunc(float x) { return __uint_as_float(__float_as_uint(x) & 0xffffe000u); }
FRNN_DEV u64 frnn_mma_desc(const void* smem, u32 lbo) {
    return (u64)((frnn_smem_addr(smem) & 0x3ffffu) >> 4) | ((u64)(lbo >> 4) << 16) | ((u64)(128u >> 4) << 32) | (1ull << 46);
}
// f32 accumulators, tf32 operands, both K-major, M = 128
#define FRNN_MMA_IDESC(n) ((1u << 4) | (2u << 7) | (2u << 10) | (((u32)(n) >> 3) << 17) | ((128u >> 4) << 24))
// d[128 x n] (+)= a[128 x 8] b[n x 8]^T, a in Tensor Memory (ts) or in shared memory (ss), shared-memory operands given by
// their descriptors: consecutive k steps of an operand are 2 * lbo bytes apart, so that a loop adds a constant instead of
// building each descriptor (one thread issues all products of a CTA).
FRNN_DEV u64 frnn_mma_next(u64 desc, u32 lbo, int k) { return desc + (u64)((u32)k * (2u * lbo >> 4)); }
FRNN_DEV void frnn_mma_ts_d(u32 d, u32 a, u64 b, u32 idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"((u32)accumulate) : "memory");
}
FRNN_DEV void frnn_mma_ss_d(u32 d, u64 a, u64 b, u32 idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"((u32)accumulate) : "memory");
}
// arrive on `bar` once every product this thread has issued so far is complete
FRNN_DEV void frnn_mma_commit(u64* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(frnn_smem_addr(bar)) : "memory");
}
// One thread of a whole warp, the same in every call.  The products are issued inside `if (frnn_elect())`: measured, a product
// takes the cycles given at the top there, and 45, whatever its width, inside `if (lane == 0)` (why was not established).
FRNN_DEV bool frnn_elect() {
    u32 r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
FRNN_DEV void frnn_half_warp_sync() { __syncwarp(0xffffu); }      // the first 16 lanes of a warp
#endif
// What tf32 truncation leaves out of x (13 bits), rounded to the 11 that tf32 holds: hi + rest is x to 2^-22, unbiased.
FRNN_DEV float frnn_tf32_rest(float x) {
    const float r = x - frnn_tf32_trunc(x);
    return frnn_bits_f32(frnn_f32_bits(r) + 0x1000u);       // the products ignore the bits below
}
// reciprocal by the fast division and one Newton step (relative error below 2e-7 for normal x)
FRNN_DEV float frnn_rcp1(float x) {
    const float r = frnn_divf(1.0f, x);
    return fmaf(r, fmaf(-x, r, 1.0f), r);
}
