// tk_umma.cuh -- pieces shared by the tcgen05 kernels: shared-memory and
// instruction descriptors, shared-memory accesses, and the tensor maps of
// their 128-polynomial tiles (host side, tk_tc5.cu).
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace tk {

// Shared-memory matrix descriptor (sm_100 format: start, leading and stride
// byte offsets in 16-byte units, version 1 at bit 46, layout at bits 61-63).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo,
                                              uint32_t layout) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | ((uint64_t)layout << 61);
}
constexpr uint32_t kLayoutNone = 0, kLayoutSw128 = 2;

// Instruction descriptor of kind::i8: D format s32 (bits 4-5 = 2), A / B
// format (bits 7-9 / 10-12: 0 unsigned, 1 signed), K-major A and B, N >> 3
// (bits 17-22), M >> 4 (bits 24-28) = 8: M = 128, K = 32 bytes.
__host__ __device__ constexpr uint32_t idesc_i8(uint32_t n, bool a_signed, bool b_signed) {
  return (2u << 4) | (a_signed ? 1u << 7 : 0u) | (b_signed ? 1u << 10 : 0u) | ((n >> 3) << 17) |
         (8u << 24);
}

__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t a) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(a) : "memory");
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c,
                                             uint32_t d) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c),
               "r"(d)
               : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

// The batch as a [npoly][256] uint16 tensor: boxes of 64 coefficients x 128
// polynomials with the 128-byte swizzle (16 KiB each, four per tile).
bool encode_swizzled_map(CUtensorMap* map, const int16_t* base, int npoly);
// A packed batch as a [npoly][row_bytes / 4] uint32 tensor, boxes of 128 whole
// rows (64 or 128 bytes) with the swizzle of the row size.
bool encode_packed_tile_map(CUtensorMap* map, const void* base, int npoly, int row_bytes);

}  // namespace tk
