// tk_pack.cu -- forward NTT of packed small polynomials (2- or 3-bit fields,
// the reference's TC-PACK input, ntt_bench/ntt_bench.cu:284-391) as one dense
// product on the 5th-generation tensor cores, sm_100a.
//
// The transform never mixes even and odd coefficients, and both halves meet
// the same 128 x 128 matrix F: out[2t + p] = sum_j F[t][j] x[2j + p].  Rows 2m and
// 2m + 1 of F belong to roots z and -z, so F is 64 rows over even j (P) and 64
// over odd j (M) with outputs P + M and P - M.  For coefficients of 2 or 3 bits
// that needs no second stage, no second constant limb and no int32
// intermediates:
//
//   * A constant c is, mod q, c0 + 2^s c1 (s = 8 - bits) with both parts int8.
//     The data side carries the coefficient twice, as x + 2^(bits-1) -- the field
//     with its sign bit flipped -- and as 2^s x, the field moved to the top of a
//     byte, so one signed K run holds both and the accumulator is the sum itself:
//     64 sums per part and parity, K = 128 bytes.  Every row's c0 sum to zero, so
//     the offset of the first form adds nothing; its small bytes toggle less
//     of the multipliers than sign-extended ones.  |P +- M| < 2^20.
//   * The operand goes from the packed words straight to tensor memory, a mask, an
//     exclusive or and a shift per two operand words: only the packed rows pass
//     through shared memory.
//   * One exact reduction per output, in the pair: the quotients are the high
//     words of S * ceil(2^32 / q) + 2^31 / q (exact floors for either sign in
//     this range), and S0 + 2^16 S1 - q (q0 + 2^16 q1) is the packed pair, 2.5
//     instructions per coefficient.
//
// What bounds it: the memory, mostly its writes, and in a long loop the 1 kW
// limit.  2^20 polynomials of 2-bit fields take 105-113 us (0.82-0.88 of a
// measured copy; 123 in a long loop), of 3-bit ones 114; the mma.sync form took
// 187 and 191, issuing 103 warp-instructions per polynomial for two matrix stages
// with fragments through shared memory, however small its input.  Energy decides
// the long loop: issuing every MMA twice cost 20 us there, hence P and M instead
// of the full matrix (half the products for one addition per output) and the small
// operand bytes; 3-bit 134 -> 127 us, 262,144 polynomials 36.5 -> 34.6.
//
// Tile: 128 polynomials, the M dimension of every MMA (one per tensor-memory
// lane).  Roles (768 threads, one CTA per SM by shared memory):
//   warps 0-15   four groups of four (warp w reaches lanes 32 (w % 4) ..): read,
//                reduce and write quarter g of a tile's outputs (pairs 32 g .. +
//                31, from P and M rows 16 g .. + 15), eight rows at a time
//   warps 16-19  unpack, a row per thread, up to two tiles ahead: as part of the
//                other warps' loop it held the stores back
//   warps 20, 21 lane 0 issues the MMAs of the even / odd coefficients (one
//                issuing thread cannot keep the pipe fed)
//   warp 22      lane 0 loads packed tiles (and the constants, once)
//   warp 23      lane 0 stores the output boxes; the first issuer's warp owns
//                the tensor-memory allocation
// Tensor memory (512 columns): two operand buffers of 128 columns (even, odd:
// P and M parts of 32 each) at 128 b, and 128 accumulator columns per parity (P,
// M: 64 each) at 256 + 128 p.  So the next tiles are unpacked and multiplied while
// a tile is reduced, and stores drain from two or three 64 KiB output slots (TMA's
// 128-byte swizzle layout, boxes of 64 coefficients).
// Every mbarrier wait gives up after 2 s (status bit 0); the issuers then
// drain their MMAs and the copy warps their copies before the CTA ends.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "tk_internal.h"
#include "tk_ptx.cuh"
#include "tk_split.h"
#include "tk_tables.h"
#include "tk_umma.cuh"

namespace tk {
namespace {

constexpr int kPkTile = 128;                       // polynomials per tile (MMA M)
constexpr int kPkOutBox = kPkTile * 128;           // 64 coefficients x 128 rows
constexpr int kPkOutSlot = 4 * kPkOutBox;          // 64 KiB
constexpr int kPkEpiWarps = 16;
constexpr int kPkUnpackWarp = 16, kPkUnpackWarps = 4;
constexpr int kPkMmaWarp = 20, kPkLoadWarp = 22, kPkStoreWarp = 23;
constexpr int kPkThreads = 768;
constexpr uint32_t kPkTmemCols = 512;
constexpr uint64_t kPkWaitNs = 2000000000ull;

template <int kBits>
struct PkLayout {
  static constexpr int kRow = kBits == 2 ? 64 : 128;  // packed bytes per polynomial
  static constexpr int kInSlots = kBits == 2 ? 2 : 3;
  static constexpr int kOutSlots = kBits == 2 ? 3 : 2;  // what fits beside the input
  static constexpr int kInBytes = kPkTile * kRow;
  static constexpr int kOffOut = kPackTableBytes;     // 1024-byte aligned
  static constexpr int kOffIn = kOffOut + kOutSlots * kPkOutSlot;
  static constexpr int kOffBars = kOffIn + kInSlots * kInBytes;
  // in_full, in_empty [kInSlots]; x_ready, op_free [2]; d_full; d_empty;
  // out_ready [kOutSlots][4]; out_free [kOutSlots]; consts; drain
  static constexpr int kBars = 2 * kInSlots + 4 + 2 + 5 * kOutSlots + 2;
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

// Quarter g (64 coefficients) of one packed row -> this thread's operand columns:
// op[2 p + h], parity p, part h, eight words (two per 16 coefficients: x +
// 2^(bits-1) and 2^s x of four).
template <int kBits>
__device__ __forceinline__ void unpack_quarter(const uint4* v, uint32_t (&op)[4][8]) {
  constexpr uint32_t kMask = kBits == 2 ? 0x03030303u : 0x07070707u;
  constexpr uint32_t kSign = kBits == 2 ? 0x02020202u : 0x04040404u;
  auto put = [&](int p, int h, int i, uint32_t w) {
    const uint32_t f = w & kMask;
    op[2 * p + h][2 * i] = f ^ kSign;
    op[2 * p + h][2 * i + 1] = f << (8 - kBits);
  };
  auto word = [&](int i) {
    const uint4& q = v[i >> 2];
    return (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w;
  };
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if constexpr (kBits == 2) {  // fields 0, 4, 8, 12 of a word are even j = 0, 2, 4, 6, ...
      const uint32_t w = word(i);
      put(0, 0, i, w);
      put(1, 0, i, w >> 2);
      put(0, 1, i, w >> 4);
      put(1, 1, i, w >> 6);
    } else {  // byte b of a word: coefficients 2 b (low field) and 2 b + 1
      const uint32_t w0 = __byte_perm(word(2 * i), word(2 * i + 1), 0x6420);
      const uint32_t w1 = __byte_perm(word(2 * i), word(2 * i + 1), 0x7531);
      put(0, 0, i, w0);
      put(1, 0, i, w0 >> 3);
      put(0, 1, i, w1);
      put(1, 1, i, w1 >> 3);
    }
  }
}

// S0, S1 (|S| < 2^20) -> the packed pair of their residues in [0, q).  With m
// = ceil(2^32 / q), S m = S 2^32 / q + S e / q, e = 1976, |S e / q| < 623 k;
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
  // tiles round robin: the launch moves through the batch as one front
  const int nmine = front_tile_count(P.ntiles, G, (int)blockIdx.x);
  auto tile_row = [&](int k) {
    return kPkTile * front_tile(P.ntiles, G, (int)blockIdx.x, k, false);
  };

  // the first tile into L2 ahead of the wait for the previous kernel (only a prefetch):
  // 100,003 polynomials 2-bit 15.5 -> 14.9 us, 3-bit 16.6 -> 15.4
  if (warp == kPkLoadWarp && lane == 0) tma_prefetch_2d(&P.in, 0, tile_row(0));
  const uint32_t bars = base + L::kOffBars;
  constexpr int S = L::kInSlots;
  auto in_full = [&](int s) { return bars + 8u * s; };
  auto in_empty = [&](int s) { return bars + 8u * (S + s); };
  constexpr uint32_t kB = 8u * (2 * S);
  auto x_ready = [&](int b) { return bars + kB + 8u * b; };
  auto op_free = [&](int b) { return bars + kB + 16u + 8u * b; };
  const uint32_t d_full = bars + kB + 32u, d_empty = bars + kB + 40u;
  auto out_ready = [&](int b, int g) { return bars + kB + 48u + 8u * (4 * b + g); };
  constexpr int NO = L::kOutSlots;
  auto out_free = [&](int b) { return bars + kB + 48u + 32u * NO + 8u * b; };
  const uint32_t consts = bars + kB + 48u + 40u * NO, drain = consts + 8u;

  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(in_full(s), 1);
      mbar_init(in_empty(s), kPkUnpackWarps);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(x_ready(b), kPkUnpackWarps);
      mbar_init(op_free(b), 2);
    }
    for (int b = 0; b < NO; b++) {
      for (int g = 0; g < 4; g++) mbar_init(out_ready(b, g), 4);
      mbar_init(out_free(b), 1);
    }
    mbar_init(d_full, 2);
    mbar_init(d_empty, kPkEpiWarps);
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
        tma_load_2d(base + L::kOffIn + s * L::kInBytes, &P.in, 0, tile_row(k),
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
        const int b = k % NO;
        for (int g = 0; g < 4; g++) {
          if (!(ok = mbar_wait_bounded(out_ready(b, g), (uint32_t)(k / NO) & 1u, kPkWaitNs))) break;
          tma_store_2d(&P.out, 64 * g, tile_row(k),
                       base + L::kOffOut + b * kPkOutSlot + g * kPkOutBox);
          bulk_commit();
        }
        if (!ok) break;
        if (k >= NO - 1) {  // tile k - (NO - 1)'s four boxes have been read out
          bulk_wait_read<4 * (NO - 1)>();
          mbar_arrive(out_free((k + 1) % NO));
        }
      }
      bulk_wait_all();
    }
  } else if (warp >= kPkMmaWarp) {
    if (lane == 0) {
      // ---- MMA issuer p: the coefficients of parity p ----
      const int p = warp - kPkMmaWarp;
      // a K step's B tile: 64 rows x 32 bytes, K-major without swizzle, 2 KiB
      const uint64_t bd = smem_desc(base, 128, 256, kLayoutNone);
      const uint32_t d = tmem + 256u + 128u * (uint32_t)p;
      ok = mbar_wait_bounded(consts, 0, kPkWaitNs);
      for (int k = 0; k < nmine && ok; k++) {
        const int b = k & 1;
        if (!(ok = mbar_wait_bounded(x_ready(b), (uint32_t)(k >> 1) & 1u, kPkWaitNs))) break;
        if (k >= 1 && !(ok = mbar_wait_bounded(d_empty, (uint32_t)(k - 1) & 1u, kPkWaitNs))) break;
        tc_fence_after();
        const uint32_t a = tmem + 128u * (uint32_t)b + 64u * (uint32_t)p;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int j = 0; j < 4; j++)
            tc_mma_ts(d + 64u * h, a + 32u * h + 8u * j, bd + (uint64_t)((4 * h + j) * (2048 >> 4)),
                      idesc_i8(64, true, true), j != 0);
        tc_commit(d_full);
        tc_commit(op_free(b));
      }
      // every MMA issued above has completed before tensor memory is freed
      tc_commit(drain);
      ok &= mbar_wait_bounded(drain, 0, kPkWaitNs);
    }
  } else if (warp >= kPkUnpackWarp) {
    // ---- unpack: packed words -> tensor memory, one row per thread ----
    const int lq = warp & 3;
    const uint32_t p = (uint32_t)(32 * lq + lane);  // polynomial (row) of the tile
    constexpr int kChunks = L::kRow / 16;
    for (int t = 0; t < nmine; t++) {
      const int s = t % S, b = t & 1;
      bool r = mbar_wait_bounded(in_full(s), (uint32_t)(t / S) & 1u, kPkWaitNs);
      const uint32_t row = base + L::kOffIn + s * L::kInBytes + p * L::kRow;
      // 64-byte rows: chunk xor (row / 2) % 4; 128-byte rows: chunk xor row % 8
      const uint32_t x = kBits == 2 ? (p >> 1) & 3u : p & 7u;
      uint4 v[kChunks];
#pragma unroll
      for (int c = 0; c < kChunks; c++) v[c] = ld_shared_v4(row + (((uint32_t)c ^ x) << 4));
      __syncwarp();
      if (lane == 0) mbar_arrive(in_empty(s));
      // the MMAs of tile t - 2 have read this operand buffer
      if (t >= 2) r &= mbar_wait_bounded(op_free(b), (uint32_t)((t >> 1) - 1) & 1u, kPkWaitNs);
      if (!(ok = __all_sync(0xffffffffu, r))) break;
      tc_fence_after();
      const uint32_t a = tmem + ((uint32_t)(32 * lq) << 16) + 128u * (uint32_t)b;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        uint32_t op[4][8];
        unpack_quarter<kBits>(v + q * (kChunks / 4), op);
#pragma unroll
        for (int i = 0; i < 4; i++) tc_st8(a + 32u * i + 8u * q, op[i]);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(x_ready(b));
    }
  } else {
    // ---- warps 0-15: sums -> output rows ----
    const int g = warp >> 2, lq = warp & 3;
    const uint32_t p = (uint32_t)(32 * lq + lane);  // polynomial (row) of the tile
    const uint32_t d0 = tmem + ((uint32_t)(32 * lq) << 16) + 256u + 16u * (uint32_t)g;
    for (int k = 0; k < nmine; k++) {
      const int b = k % NO;
      // the tile's sums are complete; tile k - NO's output has been read out of the slot
      bool r = k < NO || mbar_wait_bounded(out_free(b), (uint32_t)(k / NO - 1) & 1u, kPkWaitNs);
      r &= mbar_wait_bounded(d_full, (uint32_t)k & 1u, kPkWaitNs);
      if (!(ok = __all_sync(0xffffffffu, r))) break;
      tc_fence_after();
      const uint32_t row = base + L::kOffOut + b * kPkOutSlot + g * kPkOutBox + p * 128u;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint32_t s[32];  // rows 16 g + 8 h .. + 7: even P, even M, odd P, odd M
        const uint32_t d = d0 + 8u * h;
        tc_ld8x4_sync(d, d + 64u, d + 128u, d + 192u, s);
        if (h == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(d_empty);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
          uint32_t w[4];  // rows 2 j and 2 j + 1: two output pairs each
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const int m = 2 * j + i;
            w[2 * i] = reduce_pair(s[m] + s[8 + m], s[16 + m] + s[24 + m]);
            w[2 * i + 1] = reduce_pair(s[m] - s[8 + m], s[16 + m] - s[24 + m]);
          }
          st_shared_v4(row + (((uint32_t)(4 * h + j) ^ (p & 7u)) << 4), w[0], w[1], w[2], w[3]);
        }
      }
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
