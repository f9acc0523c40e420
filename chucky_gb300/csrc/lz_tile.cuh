// What the LZ4 and zstd decoders share: sequences (literals, then a match)
// executed a tile of output at a time by a whole CTA, in shared memory.
//
// Every byte of the tile starts as a literal's value, a byte of the output
// before the tile, or a reference to an earlier byte of the tile; references
// are followed by doubling (a byte takes its source's value or its source's
// reference), so a chain of d matches takes log2(d) rounds instead of d
// steps.  The tile leaves with aligned 16-byte stores.
#pragma once

#include "copy.cuh"

#include <stdint.h>

// Threads of the decoders' CTAs (the CPU emulation of the kernels, where every
// thread costs, has fewer): the small form, the large one, the zstd execution, and
// warps where a warp works alone.
#ifndef CHUCKY_DECODE_THREADS
#define CHUCKY_DECODE_THREADS 256
#define CHUCKY_LZ4_THREADS 1024
#define CHUCKY_ZSTD_EXEC_THREADS 512
#define CHUCKY_DECODE_WARPS 2
#endif

namespace chucky {

// copy_bytes for a source with nothing readable past its end
__device__ __forceinline__ void copy_exact(uint8_t* dst,
                                           const uint8_t* src,
                                           uint64_t n,
                                           unsigned lane,
                                           unsigned lanes)
{
  const uint64_t body = n > 64 ? n - 32 : 0; // (copy_bytes reads < 24 bytes on)
  if (body)
    copy_bytes(dst, src, body, lane, lanes);
  for (uint64_t j = body + lane; j < n; j += lanes)
    dst[j] = src[j];
}

// Exclusive prefix sum over the CTA (one value per thread); `total` for all.
template<int NT, typename T>
__device__ __forceinline__ T cta_scan(T v, T* warp_sum, T& total)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o)
      x += y;
  }
  __syncthreads(); // the sums' last readers
  if (lane == 31)
    warp_sum[warp] = x;
  __syncthreads();
  T t = lane < NT / 32 ? warp_sum[lane] : T(0);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, t, o);
    if (lane >= o)
      t += y;
  }
  total = __shfl_sync(0xffffffffu, t, 31);
  const T before = __shfl_sync(0xffffffffu, t, warp ? warp - 1 : 0);
  return (warp ? before : T(0)) + x - v;
}

// A match of any length by the whole CTA: `ml` bytes at `to` from `off`
// bytes back (both final before it; a barrier before the call).  The first
// 64 periods, or 16 bytes per thread, byte by byte, then copies of doubling
// length from the bytes already written, which lie a multiple of the offset
// behind.
template<int NT>
__device__ void cta_match(uint8_t* to, uint64_t off, uint64_t ml)
{
  const uint64_t first = off * 64 < NT * 16 ? NT * 16 / off * off : off * 64;
  uint64_t done = first < ml ? first : ml; // (below 2^32: ml or 64 offsets are)
  const uint32_t period = uint32_t(off);
  for (uint32_t j = threadIdx.x; j < uint32_t(done); j += NT)
    to[j] = (to - off)[j < period ? j : j % period];
  while (done < ml) {
    __syncthreads();
    const uint64_t k = done < ml - done ? done : ml - done;
    copy_exact(to + done, to, k, threadIdx.x, NT);
    done += k;
  }
}

template<int NT>
struct LzTile
{
  static constexpr uint32_t kBytes = NT * 16;
  alignas(16) uint16_t ref[kBytes + 16]; // value | 0x8000, or a tile index
  uint32_t start[NT / 2 + 1];            // sequences starting among 32 bytes each
  uint16_t start_at[NT / 2 + 1];         // sequences before them
};

template<int NT>
__device__ __forceinline__ void tile_clear(LzTile<NT>& S)
{
  for (uint32_t i = threadIdx.x; i < NT / 2 + 1; i += NT)
    S.start[i] = 0;
}

// A sequence whose first byte is byte `out` of the tile (`shd`: the tile's
// first byte modulo 16 in memory); sequences of no bytes are not marked.
template<int NT>
__device__ __forceinline__ void tile_mark(LzTile<NT>& S, uint32_t shd, uint32_t out)
{
  atomicOr(&S.start[(out + shd) >> 5], 1u << ((out + shd) & 31));
}

// The tile's `nout` bytes at `to`, from its marked sequences in order:
// sequence k is tok[k + 1] (tok[0] is not used, only read), with
//   .bound  the tile index (from the 16-byte boundary below `to`: + shd) past
//           its literals;
//   .dlit   what leads from a literal's tile index to its place at `lits`;
//   .off    the match offset.
// A barrier separates the marks and sequences from the call; nothing of the
// tile is stored before every literal is read.  kGroup: bytes whose loads a
// thread has in flight.
//
// Bound by the integer instructions per byte (about 25: with the places
// worked out per byte it took 50 and a tile of 8 KiB 9,400 cycles), then by
// the latency of its loads: a warp's 32 bytes share their word of start
// bits, and there is no branch, so the loads of several bytes are in flight
// together (a branch per kind of source waited for each on its own: 13,300
// cycles).  A match refers `off` back also where it overlaps itself: such a
// chain is ml / off deep, and doubling shortens it like any other.
template<int NT, uint32_t kGroup, typename Tok>
__device__ __forceinline__ void tile_run(LzTile<NT>& S,
                                         uint32_t* warp_sum,
                                         const Tok* tok,
                                         const uint8_t* lits,
                                         uint8_t* to,
                                         uint32_t nout)
{
  const uint32_t tid = threadIdx.x;
  const uint32_t shd = uint32_t(reinterpret_cast<uintptr_t>(to) & 15);
  const uint32_t lim = shd + nout;
  uint32_t total;
  const uint32_t c = tid < NT / 2 ? uint32_t(__popc(S.start[tid])) : 0;
  const uint32_t before = cta_scan<NT>(c, warp_sum, total);
  if (tid <= NT / 2) // (the tile's phase makes it spill by < 16 bytes)
    S.start_at[tid] = uint16_t(before);
  __syncthreads();
  uint8_t* const o16 = to - shd;
  const uint32_t upto = 0xFFFFFFFFu >> (31 - (tid & 31));
  uint32_t open = 0; // this thread's unresolved bytes
#pragma unroll 1
  for (uint32_t i0 = 0; i0 * NT < lim; i0 += kGroup) {
    uint32_t v[kGroup];
    const uint8_t* a[kGroup];
#pragma unroll
    for (uint32_t u = 0; u < kGroup; ++u) {
      const uint32_t j = (i0 + u) * NT + tid;
      uint32_t w = (i0 + u) * (NT / 32) + (tid >> 5);
      w = w < NT / 2 ? w : NT / 2; // (bytes past the tile: not used)
      const Tok t = tok[S.start_at[w] + uint32_t(__popc(S.start[w] & upto))];
      const bool in = j - shd < nout, lit = j < t.bound;
      const int32_t s = int32_t(j) - int32_t(t.off);
      const bool ref = !lit && s >= int32_t(shd);
      a[u] = in && !ref ? (lit ? lits + (int32_t(j) + t.dlit) : o16 + s) : nullptr;
      v[u] = uint32_t(s);
      open |= uint32_t(in && ref) << (i0 + u);
    }
#pragma unroll
    for (uint32_t u = 0; u < kGroup; ++u)
      if (a[u])
        v[u] = 0x8000u | *a[u];
#pragma unroll
    for (uint32_t u = 0; u < kGroup; ++u) {
      const uint32_t j = (i0 + u) * NT + tid;
      if (j < lim)
        S.ref[j] = uint16_t(v[u]);
    }
  }
  // follow the references
  while (__syncthreads_or(open != 0)) {
    for (uint32_t m = open; m; m &= m - 1) {
      const uint32_t i = uint32_t(__ffs(int(m)) - 1), j = i * NT + tid;
      const uint16_t v = S.ref[S.ref[j]];
      S.ref[j] = v;
      if (v & 0x8000u)
        open &= ~(1u << i);
    }
  }
  for (uint32_t v = tid; v * 16 < lim; v += NT) {
    const uint32_t lo = v * 16;
    if (lo >= shd && lo + 16 <= lim) {
      const uint4 x = reinterpret_cast<const uint4*>(S.ref)[2 * v];
      const uint4 y = reinterpret_cast<const uint4*>(S.ref)[2 * v + 1];
      auto four = [](uint32_t a, uint32_t b) { // four 16-bit values -> their bytes
        return (a & 0xFFu) | ((a >> 8) & 0xFF00u) | ((b & 0xFFu) << 16) |
               ((b & 0xFF0000u) << 8);
      };
      *reinterpret_cast<uint4*>(o16 + lo) =
        make_uint4(four(x.x, x.y), four(x.z, x.w), four(y.x, y.y), four(y.z, y.w));
    } else {
      for (uint32_t k = lo < shd ? shd : lo; k < lo + 16 && k < lim; ++k)
        to[k - shd] = uint8_t(S.ref[k]);
    }
  }
}

} // namespace chucky
