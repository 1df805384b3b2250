// Issue of tcgen05 products by one lane of a converged warp.
//
// A product's operands (descriptors, tensor-memory addresses, instruction descriptor) are warp-wide registers.  In a branch on the lane number the
// compiler has to assume that they differ between lanes, and moving them there costs more than the product: 120 to 180 cycles each where a
// 128 x 128 x 16 bf16 product takes 64.  Here the whole warp runs the issuer's loop, and four products at a time are issued under
// the elected lane's predicate, their descriptors a constant's distance from the first ones'.  Branch / this, us per launch: paired prompt attention 435 / 320,
// FP8 products of a 2,048-row latent prompt 202 / 168, NVFP4 gate + up of 4,096 tokens 330 / 286, of one token 23.5 / 19.8, latent decode attention
// of 16 sequences at 8k 137 / 114.
#pragma once
#include "common.cuh"

// K of a product: 16 (bf16), 64 (NVFP4, an E4M3 scale per 16; MXFP4, a UE8M0 scale per 32), 32 (E4M3; E2M1 x E4M3 with a UE8M0 scale per 32)
enum { TI_F16 = 0, TI_NVF4 = 1, TI_MXF4 = 2, TI_F8 = 3, TI_W4A8 = 4 };

#define TI_DESC_HI "0x40004040"        // upper word of an operand's descriptor: 1,024 bytes between groups of eight rows, 128-byte swizzle
#define TI_SF_HI "0x4008"              // of a chunk of scales: 128 bytes between groups of eight rows, no swizzle
__device__ __forceinline__ uint32_t ti_desc(uint32_t saddr) { return (uint32_t)umma_desc_sw128(saddr); }        // lower words
__device__ __forceinline__ uint32_t ti_desc_sf(uint32_t saddr) { return (uint32_t)umma_desc_sf(saddr); }

#define TI_BEGIN "{\n\t.reg .pred e, z, t;\n\t.reg .b32 al, bl, sa, sb, id;\n\t.reg .b64 a, b;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 z, %3, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
#define TI_AB(K_) "add.u32 al, %1, 2 * " #K_ ";\n\tadd.u32 bl, %2, 2 * " #K_ ";\n\tmov.b64 a, {al, " TI_DESC_HI "};\n\tmov.b64 b, {bl, " TI_DESC_HI "};\n\t"
#define TI_MMA(K_, KIND_, P_) TI_AB(K_) "@e tcgen05.mma.cta_group::1.kind::" KIND_ " [%0], a, b, %4, " P_ ";\n\t"
// scale columns S_ steps behind the first, scale byte I_ of the columns (0x20000010: one up in both of the instruction descriptor's fields)
#define TI_MMA_SF(K_, KIND_, S_, I_, P_) TI_AB(K_) "add.u32 sa, %5, %7 * " #S_ ";\n\tadd.u32 sb, %6, %8 * " #S_ ";\n\tadd.u32 id, %4, 0x20000010 * " #I_ ";\n\t" \
  "@e tcgen05.mma.cta_group::1.kind::" KIND_ " [%0], a, b, id, [sa], [sb], " P_ ";\n\t"
// d (+)= a b over the 128 bytes of every row of a stage, operands in shared memory (K-major); accumulate 0: the first product replaces what is there.  Scales (FP4,
// W4A8) from column sa / sb on, SA / SB columns from one 4-byte column of scales to the next.
template <int KIND, int SA = 0, int SB = 0>
__device__ __forceinline__ void ti_mma4(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate, uint32_t sa = 0, uint32_t sb = 0) {
#define TI_ARGS ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(accumulate), "r"(idesc)
  if (KIND == TI_F16) asm volatile(TI_BEGIN TI_MMA(0, "f16", "z") TI_MMA(1, "f16", "t") TI_MMA(2, "f16", "t") TI_MMA(3, "f16", "t") "}" TI_ARGS : "memory");
  else if (KIND == TI_F8) asm volatile(TI_BEGIN TI_MMA(0, "f8f6f4", "z") TI_MMA(1, "f8f6f4", "t") TI_MMA(2, "f8f6f4", "t") TI_MMA(3, "f8f6f4", "t") "}" TI_ARGS : "memory");
  else if (KIND == TI_NVF4)
    asm volatile(TI_BEGIN TI_MMA_SF(0, "mxf4nvf4.block_scale.scale_vec::4X", 0, 0, "z") TI_MMA_SF(1, "mxf4nvf4.block_scale.scale_vec::4X", 1, 0, "t")
                 TI_MMA_SF(2, "mxf4nvf4.block_scale.scale_vec::4X", 2, 0, "t") TI_MMA_SF(3, "mxf4nvf4.block_scale.scale_vec::4X", 3, 0, "t") "}"
                 TI_ARGS, "r"(sa), "r"(sb), "n"(SA), "n"(SB) : "memory");
  else if (KIND == TI_MXF4)         // a column holds the scales of two products
    asm volatile(TI_BEGIN TI_MMA_SF(0, "mxf4.block_scale.scale_vec::2X", 0, 0, "z") TI_MMA_SF(1, "mxf4.block_scale.scale_vec::2X", 0, 2, "t")
                 TI_MMA_SF(2, "mxf4.block_scale.scale_vec::2X", 1, 0, "t") TI_MMA_SF(3, "mxf4.block_scale.scale_vec::2X", 1, 2, "t") "}"
                 TI_ARGS, "r"(sa), "r"(sb), "n"(SA), "n"(SB) : "memory");
  else                              // one column holds those of all four
    asm volatile(TI_BEGIN TI_MMA_SF(0, "mxf8f6f4.block_scale.scale_vec::1X", 0, 0, "z") TI_MMA_SF(1, "mxf8f6f4.block_scale.scale_vec::1X", 0, 1, "t")
                 TI_MMA_SF(2, "mxf8f6f4.block_scale.scale_vec::1X", 0, 2, "t") TI_MMA_SF(3, "mxf8f6f4.block_scale.scale_vec::1X", 0, 3, "t") "}"
                 TI_ARGS, "r"(sa), "r"(sb), "n"(SA), "n"(SB) : "memory");
#undef TI_ARGS
}
// bf16, 64 of K in four products with the operands' own steps (16-byte units of a descriptor, or tensor-memory columns) and a's own upper word
#define TI_STEP_SS(K_, P_) "add.u32 al, %1, %5 * " #K_ ";\n\tadd.u32 bl, %2, %6 * " #K_ ";\n\tmov.b64 a, {al, %7};\n\tmov.b64 b, {bl, " TI_DESC_HI "};\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, " P_ ";\n\t"
#define TI_STEP_TS(K_, P_) "add.u32 al, %1, 8 * " #K_ ";\n\tadd.u32 bl, %2, %5 * " #K_ ";\n\tmov.b64 b, {bl, " TI_DESC_HI "};\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], b, %4, " P_ ";\n\t"
template <int A_STEP, int B_STEP, int A_HI = 0x40004040>
__device__ __forceinline__ void ti_f16x4_ss(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(TI_BEGIN TI_STEP_SS(0, "z") TI_STEP_SS(1, "t") TI_STEP_SS(2, "t") TI_STEP_SS(3, "t") "}"
               ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(accumulate), "r"(idesc), "n"(A_STEP), "n"(B_STEP), "n"(A_HI) : "memory");
}
template <int B_STEP>
__device__ __forceinline__ void ti_f16x4_ts(uint32_t d, uint32_t a_col, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(TI_BEGIN TI_STEP_TS(0, "z") TI_STEP_TS(1, "t") TI_STEP_TS(2, "t") TI_STEP_TS(3, "t") "}"
               ::"r"(d), "r"(a_col), "r"(b_lo), "r"(accumulate), "r"(idesc), "n"(B_STEP) : "memory");
}
// 512 bytes of scales, 32 rows x 128 bits, to four tensor-memory columns, the same in all four lane quarters
__device__ __forceinline__ void ti_cp_sf(uint32_t col, uint32_t s_lo) {
  asm volatile("{\n\t.reg .pred e;\n\t.reg .b64 s;\n\telect.sync _|e, 0xffffffff;\n\tmov.b64 s, {%1, " TI_SF_HI "};\n\t@e tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], s;\n\t}"
               ::"r"(col), "r"(s_lo) : "memory");
}
__device__ __forceinline__ void ti_commit(uint64_t* bar) {
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
