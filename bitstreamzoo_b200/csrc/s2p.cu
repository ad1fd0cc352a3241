// Byte -> basis-bit transposition ("serial to parallel") on the device.
//
// Replaces payload_to_basis_bits / payload_to_basis_bits_fast
// (benchmark/apps/regex/src/run.py:164-187): basis stream i holds, at bit j,
// bit i of byte j.  With streams stored as little-endian uint64 words, word w
// of stream i is built from the 64 bytes [64w, 64w+64), which one thread per
// output word transposes in registers:
//
//   1. each 8-byte group x_q (bytes 8q..8q+7) is an 8x8 bit matrix (row =
//      byte, column = bit); three masked delta swaps (block sizes 1, 2, 4)
//      transpose it, so byte i of the result holds bit i of the 8 bytes;
//   2. the eight results form an 8x8 byte matrix (row q, column i); three
//      block swaps (32-, 16-, 8-bit halves) transpose it, so word i holds
//      byte i of every group, i.e. bits 64w..64w+63 of basis stream i.
//
// HBM-bound: n bytes in, n bytes out (eight streams of n bits), each warp
// storing 8 coalesced 256-byte rows.  Bytes past n read as zero, so every
// stream's bits at and above n are clean.
#include "device.h"
#include "pdl.cuh"
#include "s2p.h"

#include <algorithm>
#include <stdexcept>
#include <string>

namespace bsz {

namespace {

constexpr int kS2PThreads = 128;
// Words below which one step per warp spreads better over the SMs.
constexpr int64_t kS2PLongWords = int64_t(1) << 18;

struct BasisOut {
  uint64_t* p[8];
};

// A warp owns STEPS x 32 words.  VEC: the byte source is 16-byte aligned, so
// the warp's bytes load as coalesced 16-byte loads, all STEPS x 4 of a lane in
// flight, and change lanes in shared memory (each lane needs 64 consecutive
// bytes).  Steps past the whole 64-byte groups, and any unaligned source, load
// byte by byte.  512 MiB on a B200: 199 us with one strided group per thread
// and a persistent grid (0.83 of the copy rate), 179 us coalesced at 4 steps
// and 256 threads, 169 us at 128 threads (0.97).
//
// Shared memory: 16-byte piece c of a step's bytes lies at c ^ ((c >> 3) & 3),
// which keeps both the rows written and the columns read free of conflicts.
template <bool VEC, int STEPS>
__global__ void __launch_bounds__(kS2PThreads)
k_s2p(const uint8_t* __restrict__ bytes, int64_t n_bytes, int64_t nw, BasisOut out) {
  after_previous(bytes);
  __shared__ uint4 s_bytes[VEC ? kS2PThreads / 32 : 1][128];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (kS2PThreads / 32);
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * (kS2PThreads / 32) + warp; t * 32 * STEPS < nw; t += warps) {
    uint4 v[STEPS][4];
    if (VEC) {
#pragma unroll
      for (int s = 0; s < STEPS; ++s) {
        const int64_t w0 = (t * STEPS + s) * 32;
        if ((w0 + 32) * 64 <= n_bytes) {
          const uint4* src = reinterpret_cast<const uint4*>(bytes + w0 * 64);
#pragma unroll
          for (int k = 0; k < 4; ++k) v[s][k] = __ldg(src + k * 32 + lane);
        }
      }
    }
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
      const int64_t w0 = (t * STEPS + s) * 32, w = w0 + lane;
      uint64_t x[8];
      if (VEC && (w0 + 32) * 64 <= n_bytes) {
        __syncwarp();   // the step before has been read
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int c = k * 32 + lane;
          s_bytes[warp][c ^ ((c >> 3) & 3)] = v[s][k];
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int c = lane * 4 + k;
          const uint4 q = s_bytes[warp][c ^ ((c >> 3) & 3)];
          x[2 * k] = static_cast<uint64_t>(q.x) | (static_cast<uint64_t>(q.y) << 32);
          x[2 * k + 1] = static_cast<uint64_t>(q.z) | (static_cast<uint64_t>(q.w) << 32);
        }
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          uint64_t u = 0;
          for (int k = 0; k < 8; ++k) {
            const int64_t j = w * 64 + q * 8 + k;
            if (j < n_bytes) u |= static_cast<uint64_t>(bytes[j]) << (8 * k);
          }
          x[q] = u;
        }
      }
      s2p_transpose64(x);
      if (w < nw) {
#pragma unroll
        for (int i = 0; i < 8; ++i) out.p[i][w] = x[i];
      }
    }
  }
}

}  // namespace

void launch_s2p(Device& dev, const uint8_t* bytes, int64_t n_bytes, uint64_t* const* out) {
  if (n_bytes <= 0) return;
  const int64_t nw = (n_bytes + 63) / 64;
  BasisOut o;
  for (int i = 0; i < 8; ++i) {
    if (!out[i]) throw std::invalid_argument("s2p: output stream " + std::to_string(i) + " is null");
    o.p[i] = out[i];
  }
  const bool vec = (reinterpret_cast<uintptr_t>(bytes) & 15) == 0;
  const int steps = vec && nw >= kS2PLongWords ? 4 : 1;
  const int64_t per_block = static_cast<int64_t>(kS2PThreads) * steps;
  const unsigned blocks = static_cast<unsigned>(std::min<int64_t>((nw + per_block - 1) / per_block, 0x7fffffff));
  ProfScope prof(dev, "k_s2p");
  if (steps == 4) launch_after(dev.stream(), blocks, kS2PThreads, 0, k_s2p<true, 4>, bytes, n_bytes, nw, o);
  else if (vec) launch_after(dev.stream(), blocks, kS2PThreads, 0, k_s2p<true, 1>, bytes, n_bytes, nw, o);
  else launch_after(dev.stream(), blocks, kS2PThreads, 0, k_s2p<false, 1>, bytes, n_bytes, nw, o);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw CudaError(std::string("s2p launch failed: ") + cudaGetErrorString(e));
  ++dev.n_launches;
}

}  // namespace bsz
