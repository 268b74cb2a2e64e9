// Rules of the host-buffer calls.  Host-only.
//
// Chunk schedule of the transforms (tk_ntt_host / tk_invntt_host).
// Chunks of at most `chunk` polynomials: the first ones grow from
// kHostRampPolys (doubling) and the last ones shrink towards it (at most half
// of what remains), because the first upload and the last download run with
// nothing beside them; a remainder below kHostRampPolys is never left behind
// when the rest fits one chunk.
#pragma once

#include <stddef.h>

namespace tk {

constexpr size_t kHostRampPolys = 4096;

// Size of chunk c (0-based) when `remaining` polynomials are left.
inline size_t host_chunk_size(int c, size_t remaining, size_t chunk) {
  size_t n = chunk;
  if (c < 16 && (kHostRampPolys << c) < n) n = kHostRampPolys << c;
  const size_t half = (remaining + 1) / 2;
  const size_t tail = half > kHostRampPolys ? half : kHostRampPolys;
  if (tail < n) n = tail;
  if (remaining - n < kHostRampPolys && remaining <= chunk) n = remaining;  // no sliver
  return n < remaining ? n : remaining;
}

// tk_matvec_host uses page-locked buffers in place up to this many bytes of A, s,
// e and out together (20 us of the link).  In place, the kernel's CTAs stay on their
// SMs for as long as the link takes, and a kernel on another stream that needs
// those SMs waits; staged, the copy engines do the waiting.  Another stream's
// forward of 16,411 polynomials / inverse of 262,144 beside back-to-back calls of k
// = 4, median us a call, in place / staged: 73 jobs (1 MB) 32 / 23 and 66 / 65, 290
// (4 MB) 70 / 31 and 117 / 73, 8,000 (110 MB) 180-640 / 36-41 and 174 (a tenth above
// 1,500) / 80.  Fewer CTAs do not help: with 18 of them the inverse, which needs
// whole SMs, still takes 110.  What a call itself gains in place is 9-12 us and, above
// the limit, 5-13 %: 0.5 MB 38 -> 28, 1 MB 47 -> 36, 4 MB 103 -> 90 (staged copies of
// 2-16 MB took twice as long on one of three boxes), 64 MB 1,244 -> 1,190.
constexpr size_t kMatvecInPlaceBytes = (size_t)1 << 20;

}  // namespace tk
