// tk_pack.cu -- forward NTT of packed small polynomials (2- or 3-bit fields,
// the reference's TC-PACK input, ntt_bench/ntt_bench.cu:284-391) as one dense
// product on the 5th-generation tensor cores, sm_100a.
//
// The transform never mixes even and odd coefficients, and both halves meet
// the same 128 x 128 matrix F: out[2t + p] = sum_j F[t][j] x[2j + p].  For
// coefficients of 2 or 3 bits that product needs no second stage, no second
// constant limb and no int32 intermediates:
//
//   * A constant c, centred in [-(q-1)/2, (q-1)/2], is c0 + 2^s c1 (s = 8 -
//     bits) with both parts int8.  The data side carries the coefficient
//     twice, as x and as 2^s x -- the packed field moved to the top of a byte
//     -- so one signed K run holds both and the accumulator is the sum itself:
//     128 outputs per parity, K = 256 bytes, |S| <= 128 * 4 * 1664 < 2^20.
//   * The operand goes from the packed words straight to tensor memory: two
//     table look-ups (__byte_perm) per four 2-bit fields, or a mask and a
//     multiply-add per four 3-bit ones.  Nothing is staged in shared memory.
//   * One exact reduction per output, in the pair: the quotients are the high
//     words of S * ceil(2^32 / q) + 2^31 / q (exact floors for either sign in
//     this range), and S0 + 2^16 S1 - q (q0 + 2^16 q1) is the packed pair, 2.5
//     instructions per coefficient.
//
// What bounds it: the memory, mostly its writes.  2^20 polynomials of 2-bit
// fields take 104.7 us, 5.8 TB/s (0.88 of a measured copy); the mma.sync form
// took 187.1 us, issuing 103 warp-instructions per polynomial for two matrix
// stages with fragments through shared memory, however small its input.
//
// Tile: 128 polynomials, the M dimension of every MMA (one per tensor-memory
// lane).  Roles (640 threads, one CTA per SM by shared memory):
//   warps 0-15   four groups of four (warp w reaches lanes 32 (w % 4) ..):
//                unpack quarter g of every row of tile k + 1, then read, reduce
//                and write quarter g of tile k's outputs (pairs 32 g .. + 31)
//   warps 16, 17 lane 0 issues the MMAs of output half 0 / 1 (64 outputs of
//                each parity: one issuing thread cannot keep the pipe fed)
//   warp 18      lane 0 loads packed tiles (and the constants, once)
//   warp 19      lane 0 stores the output boxes; the first issuer's warp owns
//                the tensor-memory allocation
// Tensor memory (512 columns): two operand buffers of 128 columns (even,
// odd: 64 each) at 128 b, and an accumulator buffer of 128 columns per output
// half (even, odd: 64 each) at 256 + 128 c.  So tile k + 1 is unpacked and
// multiplied while tile k is reduced, and the stores of tiles k and k - 1
// drain from two 64 KiB output slots (TMA's 128-byte swizzle layout, boxes of
// 64 coefficients).
// Every mbarrier wait gives up after 2 s (status bit 0); the issuers then
// drain their MMAs and the copy warps their copies before the CTA ends.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "tk_internal.h"
#include "tk_ptx.cuh"
#include "tk_tables.h"
#include "tk_umma.cuh"

namespace tk {
namespace {

constexpr int kPkTile = 128;                       // polynomials per tile (MMA M)
constexpr int kPkOutBox = kPkTile * 128;           // 64 coefficients x 128 rows
constexpr int kPkOutSlot = 4 * kPkOutBox;          // 64 KiB
constexpr int kPkEpiWarps = 16;
constexpr int kPkMmaWarp = 16, kPkLoadWarp = 18, kPkStoreWarp = 19;
constexpr int kPkThreads = 640;
constexpr uint32_t kPkTmemCols = 512;
constexpr uint64_t kPkWaitNs = 2000000000ull;

template <int kBits>
struct PkLayout {
  static constexpr int kRow = kBits == 2 ? 64 : 128;  // packed bytes per polynomial
  static constexpr int kInSlots = kBits == 2 ? 4 : 3;
  static constexpr int kInBytes = kPkTile * kRow;
  static constexpr int kOffOut = kPackTableBytes;     // 1024-byte aligned
  static constexpr int kOffIn = kOffOut + 2 * kPkOutSlot;
  static constexpr int kOffBars = kOffIn + kInSlots * kInBytes;
  // in_full, in_empty [kInSlots]; x_ready, op_free [2]; d_full, d_empty [2];
  // out_ready [2][4]; out_free [2]; consts; drain
  static constexpr int kBars = 2 * kInSlots + 4 + 4 + 8 + 2 + 2;
  static constexpr int kOffTmemSlot = kOffBars + 8 * kBars;
  static constexpr int kSmemBytes = kOffTmemSlot + 8;
  static_assert(2 * kSmemBytes > 228 * 1024, "one CTA per SM: it owns all tensor memory");
  static_assert(kSmemBytes <= 227 * 1024, "shared memory per CTA");
};

__device__ __align__(128) uint8_t g_pack_tables[2][kPackTableBytes];

struct PkParams {
  CUtensorMap in;   // [npoly][row bytes] as uint32, boxes of 128 rows, swizzled by the row size
  CUtensorMap out;  // [npoly][256] uint16, boxes 64 x 128 rows, 128-byte swizzle
  const uint8_t* tables;
  unsigned* status;
  int ntiles;
};

// Quarter g (64 coefficients) of one packed row -> this thread's 16 even and
// 16 odd operand columns.  Column order per packed word as
// build_pack_tables' K order.
template <int kBits>
__device__ __forceinline__ void unpack_quarter(const uint4* v, uint32_t (&ev)[16],
                                               uint32_t (&od)[16]) {
  if constexpr (kBits == 2) {
    // byte_perm tables indexed by the field: x in {0, 1, -2, -1} and 64 x
    constexpr uint32_t kX = 0xfffe0100u, kTop = 0xc0804000u;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t w = i == 0 ? v[0].x : i == 1 ? v[0].y : i == 2 ? v[0].z : v[0].w;
      const uint32_t e = w & 0x33333333u, o = (w >> 2) & 0x33333333u;
      ev[4 * i + 0] = __byte_perm(kX, 0, e);
      ev[4 * i + 1] = __byte_perm(kX, 0, e >> 16);
      ev[4 * i + 2] = __byte_perm(kTop, 0, e);
      ev[4 * i + 3] = __byte_perm(kTop, 0, e >> 16);
      od[4 * i + 0] = __byte_perm(kX, 0, o);
      od[4 * i + 1] = __byte_perm(kX, 0, o >> 16);
      od[4 * i + 2] = __byte_perm(kTop, 0, o);
      od[4 * i + 3] = __byte_perm(kTop, 0, o >> 16);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint4& q = v[i >> 2];
      const uint32_t w = (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w;
      const uint32_t e = w & 0x07070707u, o = (w >> 3) & 0x07070707u;
      // sign-extend each byte: + 0xf8 where bit 2 is set (4 * 62 = 0xf8)
      ev[2 * i] = e + (e & 0x04040404u) * 62u;
      ev[2 * i + 1] = e << 5;  // 32 x: the field at the top of the byte
      od[2 * i] = o + (o & 0x04040404u) * 62u;
      od[2 * i + 1] = o << 5;
    }
  }
}

// S0, S1 (|S| < 2^20) -> the packed pair of their residues in [0, q).  With m
// = ceil(2^32 / q), S m = S 2^32 / q + S e / q, e = 1976, |S e / q| < 506 k;
// adding 2^31 / q = 645 k keeps the high word at floor(S / q) for S = j q
// (error from below) and S = j q + q - 1 (2^32 / q = 1290 k from above).
__device__ __forceinline__ uint32_t reduce_pair(uint32_t s0, uint32_t s1) {
  constexpr long long kM = 1290168, kHalf = 645083;
  const uint32_t q0 = (uint32_t)((unsigned long long)((long long)(int32_t)s0 * kM + kHalf) >> 32);
  const uint32_t q1 = (uint32_t)((unsigned long long)((long long)(int32_t)s1 * kM + kHalf) >> 32);
  return (s0 + (s1 << 16)) - (q0 + (q1 << 16)) * (uint32_t)kQ;
}

template <int kBits>
__global__ void __launch_bounds__(kPkThreads, 1) k_ntt_packed(const __grid_constant__ PkParams P) {
  using L = PkLayout<kBits>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  if (base & 1023u) {  // the swizzled slots need the 1024-byte atom alignment
    if (threadIdx.x == 0) atomicOr(P.status, 1u);
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = (int)gridDim.x;
  const int t_begin = (int)((long long)blockIdx.x * P.ntiles / G);
  const int t_end = (int)((long long)(blockIdx.x + 1) * P.ntiles / G);
  const int nmine = t_end - t_begin;

  const uint32_t bars = base + L::kOffBars;
  constexpr int S = L::kInSlots;
  auto in_full = [&](int s) { return bars + 8u * s; };
  auto in_empty = [&](int s) { return bars + 8u * (S + s); };
  constexpr uint32_t kB = 8u * (2 * S);
  auto x_ready = [&](int b) { return bars + kB + 8u * b; };
  auto op_free = [&](int b) { return bars + kB + 16u + 8u * b; };
  auto d_full = [&](int c) { return bars + kB + 32u + 8u * c; };
  auto d_empty = [&](int c) { return bars + kB + 48u + 8u * c; };
  auto out_ready = [&](int b, int g) { return bars + kB + 64u + 8u * (4 * b + g); };
  auto out_free = [&](int b) { return bars + kB + 128u + 8u * b; };
  const uint32_t consts = bars + kB + 144u, drain = bars + kB + 152u;

  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(in_full(s), 1);
      mbar_init(in_empty(s), kPkEpiWarps);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(x_ready(b), kPkEpiWarps);
      mbar_init(op_free(b), 2);
      mbar_init(d_full(b), 1);
      mbar_init(d_empty(b), 8);
      for (int g = 0; g < 4; g++) mbar_init(out_ready(b, g), 4);
      mbar_init(out_free(b), 1);
    }
    mbar_init(consts, 1);
    mbar_init(drain, 2);
    fence_mbar_init();
  }
  if (warp == kPkMmaWarp) {
    tmem_alloc(base + L::kOffTmemSlot, kPkTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();  // the mbarriers are initialised (and fenced) before any use
  tc_fence_after();
  const uint32_t tmem = *(volatile uint32_t*)(smem_raw + L::kOffTmemSlot);
  if (warp == kPkLoadWarp && lane == 0) {  // constants (written once by the host)
    mbar_expect_tx(consts, kPackTableBytes);
    bulk_g2s(base, P.tables, kPackTableBytes, consts);
  }
  // the input may have been written, the output read, by the previous kernel
  grid_dependency_wait();
  grid_launch_dependents();

  bool ok = true;
  if (warp == kPkLoadWarp) {
    if (lane == 0) {
      int k = 0;
      for (; k < nmine; k++) {
        const int s = k % S;
        if (k >= S && !(ok = mbar_wait_bounded(in_empty(s), (uint32_t)(k / S - 1) & 1u, kPkWaitNs)))
          break;
        mbar_expect_tx(in_full(s), L::kInBytes);
        tma_load_2d(base + L::kOffIn + s * L::kInBytes, &P.in, 0, kPkTile * (t_begin + k),
                    in_full(s));
      }
      // every load has landed before the CTA's memory goes
      for (int j = k > S ? k - S : 0; j < k; j++)
        ok &= mbar_wait_bounded(in_full(j % S), (uint32_t)(j / S) & 1u, kPkWaitNs);
      ok &= mbar_wait_bounded(consts, 0, kPkWaitNs);
    }
  } else if (warp == kPkStoreWarp) {
    if (lane == 0) {
      for (int k = 0; k < nmine && ok; k++) {
        const int b = k & 1;
        for (int g = 0; g < 4; g++) {
          if (!(ok = mbar_wait_bounded(out_ready(b, g), (uint32_t)(k >> 1) & 1u, kPkWaitNs))) break;
          tma_store_2d(&P.out, 64 * g, kPkTile * (t_begin + k),
                       base + L::kOffOut + b * kPkOutSlot + g * kPkOutBox);
          bulk_commit();
        }
        if (!ok) break;
        if (k >= 1) {  // tile k - 1's four boxes have been read out
          bulk_wait_read<4>();
          mbar_arrive(out_free(b ^ 1));
        }
      }
      bulk_wait_all();
    }
  } else if (warp >= kPkMmaWarp) {
    if (lane == 0) {
      // ---- MMA issuer c: outputs 64 c .. + 63 of both parities ----
      const int c = warp - kPkMmaWarp;
      // a K step's B tile: 64 rows x 32 bytes, K-major without swizzle, 2 KiB
      const uint64_t bd = smem_desc(base + (uint32_t)c * (kPackTableBytes / 2), 128, 256,
                                    kLayoutNone);
      const uint32_t d = tmem + 256u + 128u * (uint32_t)c;
      ok = mbar_wait_bounded(consts, 0, kPkWaitNs);
      for (int k = 0; k < nmine && ok; k++) {
        const int b = k & 1;
        if (!(ok = mbar_wait_bounded(x_ready(b), (uint32_t)(k >> 1) & 1u, kPkWaitNs))) break;
        if (k >= 1 && !(ok = mbar_wait_bounded(d_empty(c), (uint32_t)(k - 1) & 1u, kPkWaitNs)))
          break;
        tc_fence_after();
        const uint32_t a = tmem + 128u * (uint32_t)b;
#pragma unroll
        for (int par = 0; par < 2; par++)
#pragma unroll
          for (int j = 0; j < 8; j++)
            tc_mma_ts(d + 64u * par, a + 64u * par + 8u * j, bd + (uint64_t)(j * (2048 >> 4)),
                      idesc_i8(64, true, true), j != 0);
        tc_commit(d_full(c));
        tc_commit(op_free(b));
      }
      // every MMA issued above has completed before tensor memory is freed
      tc_commit(drain);
      ok &= mbar_wait_bounded(drain, 0, kPkWaitNs);
    }
  } else {
    // ---- warps 0-15: packed words -> tensor memory -> output rows ----
    const int g = warp >> 2, lq = warp & 3, c = g >> 1;
    const uint32_t lanes = (uint32_t)(32 * lq) << 16;
    const uint32_t p = (uint32_t)(32 * lq + lane);  // polynomial (row) of the tile
    auto unpack = [&](int t) {
      const int s = t % S, b = t & 1;
      bool r = mbar_wait_bounded(in_full(s), (uint32_t)(t / S) & 1u, kPkWaitNs);
      const uint32_t row = base + L::kOffIn + s * L::kInBytes + p * L::kRow;
      uint4 v[kBits == 2 ? 1 : 2];
      if constexpr (kBits == 2) {  // 64-byte swizzle: chunk xor (row / 2) % 4
        v[0] = ld_shared_v4(row + (((uint32_t)g ^ ((p >> 1) & 3u)) << 4));
      } else {  // 128-byte swizzle: chunk xor row % 8
        v[0] = ld_shared_v4(row + (((2u * g) ^ (p & 7u)) << 4));
        v[1] = ld_shared_v4(row + (((2u * g + 1u) ^ (p & 7u)) << 4));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(in_empty(s));
      uint32_t ev[16], od[16];
      unpack_quarter<kBits>(v, ev, od);
      // the MMAs of tile t - 2 have read this operand buffer
      if (t >= 2) r &= mbar_wait_bounded(op_free(b), (uint32_t)((t >> 1) - 1) & 1u, kPkWaitNs);
      if (!__all_sync(0xffffffffu, r)) return false;
      tc_fence_after();
      const uint32_t a = tmem + lanes + 128u * (uint32_t)b + 16u * (uint32_t)g;
      tc_st16(a, ev);
      tc_st16(a + 64u, od);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(x_ready(b));
      return true;
    };
    if (nmine > 0) ok = unpack(0);
    for (int k = 0; k < nmine && ok; k++) {
      if (k + 1 < nmine && !(ok = unpack(k + 1))) break;
      const int b = k & 1;
      bool r = mbar_wait_bounded(d_full(c), (uint32_t)k & 1u, kPkWaitNs);
      if (!(ok = __all_sync(0xffffffffu, r))) break;
      tc_fence_after();
      uint32_t s[64];  // outputs 32 g .. + 31 of each parity
      const uint32_t d = tmem + lanes + 256u + 128u * (uint32_t)c + 32u * (uint32_t)(g & 1);
      tc_ld32x2_sync(d, d + 64u, s);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(d_empty(c));
      // tile k - 2's output has been read out of this slot
      r = k < 2 || mbar_wait_bounded(out_free(b), (uint32_t)((k >> 1) - 1) & 1u, kPkWaitNs);
      if (!(ok = __all_sync(0xffffffffu, r))) break;
      const uint32_t row = base + L::kOffOut + b * kPkOutSlot + g * kPkOutBox + p * 128u;
#pragma unroll
      for (int j = 0; j < 8; j++)
        st_shared_v4(row + (((uint32_t)j ^ (p & 7u)) << 4),
                     reduce_pair(s[4 * j], s[32 + 4 * j]),
                     reduce_pair(s[4 * j + 1], s[32 + 4 * j + 1]),
                     reduce_pair(s[4 * j + 2], s[32 + 4 * j + 2]),
                     reduce_pair(s[4 * j + 3], s[32 + 4 * j + 3]));
      fence_proxy_async_smem();  // generic-proxy writes -> the TMA store
      __syncwarp();
      if (lane == 0) mbar_arrive(out_ready(b, g));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kPkMmaWarp) {
    __syncwarp();  // lane 0 issued MMAs alone; dealloc is warp-wide
    tc_fence_after();
    tmem_dealloc(tmem, kPkTmemCols);
  }
  if (!ok) atomicOr(P.status, 1u);
}

const uint8_t* g_pack_ptr[64];

const void* packed_fn(int bits) {
  return bits == 2 ? (const void*)k_ntt_packed<2> : (const void*)k_ntt_packed<3>;
}
int packed_smem(int bits) { return bits == 2 ? PkLayout<2>::kSmemBytes : PkLayout<3>::kSmemBytes; }

}  // namespace

bool pack_init_device(DeviceInfo* info) {
  static uint8_t image[2][kPackTableBytes];
  static std::once_flag once;
  std::call_once(once, [] {
    build_pack_tables(2, image[0]);
    build_pack_tables(3, image[1]);
  });
  if (info->device < 0 || info->device >= 64) return false;
  if (cudaMemcpyToSymbol(g_pack_tables, image, sizeof(image)) != cudaSuccess) return false;
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_pack_tables) != cudaSuccess || !p) return false;
  g_pack_ptr[info->device] = (const uint8_t*)p;
  for (int bits = 2; bits <= 3; bits++)
    if (cudaFuncSetAttribute(packed_fn(bits), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             packed_smem(bits)) != cudaSuccess)
      return false;
  return true;
}

cudaError_t launch_packed(int bits, const void* src, int16_t* dst, int npoly,
                          const DeviceInfo& info, cudaStream_t stream) {
  const uint8_t* tables = g_pack_ptr[info.device];
  if (!tables || !info.status) return cudaErrorInitializationError;
  PkParams m = {};
  if (!encode_packed_tile_map(&m.in, src, npoly, bits == 2 ? 64 : 128) ||
      !encode_swizzled_map(&m.out, dst, npoly))
    return cudaErrorInvalidResourceHandle;
  m.tables = tables + (bits - 2) * kPackTableBytes;
  m.status = info.status;
  m.ntiles = (npoly + kPkTile - 1) / kPkTile;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(m.ntiles < info.num_sms ? m.ntiles : info.num_sms));
  cfg.blockDim = dim3((unsigned)kPkThreads);
  cfg.dynamicSmemBytes = (size_t)packed_smem(bits);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[1] = {(void*)&m};
  return cudaLaunchKernelExC(&cfg, packed_fn(bits), args);
}

}  // namespace tk
