// LZ4 block decoder: raw LZ4 blocks (the CODEC_LZ4_NON_STANDARD chunk
// format) back to chunk bytes on the device, for on-device verification and
// readback of stores.  The reference decodes its chunks on the host with
// LZ4_decompress_safe and the known chunk size (src/cpu/compress.c:85,
// tests/test_compress_cpu.c:75-190); this is the same contract on the GPU.
//
// A CTA per block, a tile of the block at a time.  The format is a chain of
// tokens, each known only once the one before it is, and every match reads
// bytes that earlier sequences wrote; decoded token by token a warp spends
// about 500 cycles of memory latency on each.  Here both chains are
// followed by all threads at once, in shared memory:
//   parse  : for every byte of a window of the compressed block, where the
//            next token would start if a token started there; exits of
//            32-byte pieces by doubling within a warp (shuffles), of
//            512-byte pieces by hops over those, so that the true chain
//            crosses the window in one hop per warp; the tokens on it are
//            then listed in order;
//   place  : prefix sums of the sequences' lengths give each its place in
//            an output tile;
//   execute: every byte of the tile finds its value by following references
//            to earlier bytes (lz_tile.cuh).
// A long sequence (literal run or match) is copied by the whole CTA.
//
// With few blocks two CTAs work on each, one parsing and placing ahead of the
// other's execution (lz4_decode_pair_k).  With more blocks than the chip holds
// CTAs, those of few sequences are decoded by a warp each, token by token:
// there are enough of them to hide each other's latency (launch_lz4_decode).
//
// Bound by the integer instructions of the parse and of the tiles (about 20
// us for a 16 KiB tile: 12 of parse and placement, of them 5 chain steps, 2
// chain, 5 sequences, and 8 tile), not by memory: 64 sensor chunks of 1 MiB take
// 1.00 ms with two CTAs each, 1.39 with one (a warp per block, sequence by
// sequence: 62.3 ms), 912 of 16 KiB 0.15 ms.
//
// Every read is checked against the block's size and every write against
// the chunk size.  A block the fast path cannot finish is decoded once more
// by one warp, sequence by sequence, which sets its status; nothing is read
// or written out of bounds.
#include "chucky_gb300.h"
#include "kernels_codec.hpp"
#include "launch.cuh"
#include "lz_tile.cuh"

#include <cuda_runtime.h>

namespace chucky {

namespace {

// CTAs of the small form that an SM holds (64 registers a thread), and that
// the chip does
constexpr int kSmallCtas = 4;
#ifndef CHUCKY_LZ4_SLOTS
#define CHUCKY_LZ4_SLOTS(sms) (kSmallCtas * (sms))
#endif

enum : uint32_t
{
  kDecodeOk = 0,
  kDecodeTruncated = 1, // the block ends inside a token, length or literals
  kDecodeBadOffset = 2, // a match offset of 0 or before the chunk start
  kDecodeOverrun = 3,   // the output would exceed the chunk size
  kDecodeShort = 4,     // the block ends before the chunk is complete
  kDecodeLeft = 99,     // (not a status: left to the whole CTA)
};

// Copies by one warp.
__device__ __forceinline__ void warp_copy(uint8_t* dst, const uint8_t* src, uint64_t n)
{
  copy_exact(dst, src, n, threadIdx.x & 31, 32);
}

// A match by one warp (the bytes before `to` final and seen by all lanes): whole
// periods of the offset first, then copies of doubling length.
__device__ __forceinline__ void warp_match(uint8_t* to, uint32_t off, uint64_t ml)
{
  const uint8_t* const from = to - off;
  const uint64_t first = off < 128 ? 128 / off * off : off;
  uint64_t done = first < ml ? first : ml;
  for (uint32_t j = threadIdx.x & 31; j < uint32_t(done); j += 32)
    to[j] = from[j < off ? j : j % off];
  while (done < ml) {
    __syncwarp();
    const uint64_t k = done < ml - done ? done : ml - done;
    warp_copy(to + done, to, k);
    done += k;
  }
}

// A warp that may leave its block counts sequences by their bytes above
// `worth`: once they fall kWorthLag sequences' worth behind (they get kWorthLead
// ahead at most), or one has kLongSequence literals or match bytes, the rest is
// left to the whole CTA.
constexpr int kWorthLag = 3, kWorthLead = 32;
constexpr uint32_t kLongSequence = 16 << 10;

// One block by one warp, from ip and op on; `worth` 0: to its end, otherwise it
// may be left at the sequence that ip and op then name.  Every lane parses the
// same tokens (the byte loads broadcast within the warp); a match reads only
// bytes already final before op.  kVec: copies by vectors where they are long
// (the code for it costs a short kernel more than it gives).
template<bool kVec>
__device__ __forceinline__ uint32_t lz4_decode_warp(const uint8_t* src,
                                                    uint64_t n,
                                                    uint8_t* dst,
                                                    uint64_t chunk_bytes,
                                                    int worth,
                                                    uint64_t& ip,
                                                    uint64_t& op)
{
  const uint32_t lane = threadIdx.x & 31;
  int lead = 0;
  for (;;) {
    uint64_t at = ip, to = op; // (the sequence is taken once it is done)
    if (at >= n)
      return kDecodeTruncated;
    const uint32_t token = src[at++];
    uint64_t lit = token >> 4;
    if (lit == 15)
      for (uint32_t b = 255; b == 255; lit += b) {
        if (at >= n)
          return kDecodeTruncated;
        b = src[at++];
      }
    if (worth && lit >= kLongSequence)
      return kDecodeLeft;
    if (lit > n - at)
      return kDecodeTruncated;
    if (lit > chunk_bytes - to)
      return kDecodeOverrun;
    if (!kVec) {
      for (uint64_t j = lane; j < lit; j += 32)
        dst[to + j] = src[at + j];
    } else if (lit >= 256) {
      warp_copy(dst + to, src + at, lit);
    } else { // four loads in flight: one by one they took a tenth longer
      for (uint32_t j = lane; j < uint32_t(lit); j += 128) {
        uint8_t v[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
          if (j + 32 * u < lit)
            v[u] = src[at + j + 32 * u];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
          if (j + 32 * u < lit)
            dst[to + j + 32 * u] = v[u];
      }
    }
    at += lit;
    to += lit;
    if (at == n) // the last sequence has literals only
      return to == chunk_bytes ? kDecodeOk : kDecodeShort;
    if (n - at < 2)
      return kDecodeTruncated;
    const uint32_t off = src[at] | uint32_t(src[at + 1]) << 8;
    at += 2;
    if (off == 0 || off > to)
      return kDecodeBadOffset;
    uint64_t ml = (token & 15) + 4;
    if ((token & 15) == 15)
      for (uint32_t b = 255; b == 255; ml += b) {
        if (at >= n)
          return kDecodeTruncated;
        b = src[at++];
      }
    if (worth && ml >= kLongSequence)
      return kDecodeLeft; // (its literals are written once more)
    if (ml > chunk_bytes - to)
      return kDecodeOverrun;
    // the literals just written by other lanes are read below
    __syncwarp();
    if (kVec && ml >= 256) {
      warp_match(dst + to, off, ml);
    } else {
      const uint8_t* m = dst + to - off;
      for (uint64_t j = lane; j < ml; j += 32)
        dst[to + j] = m[j < off ? j : j % off];
    }
    __syncwarp();
    const uint64_t made = to + ml - op;
    ip = at;
    op = to + ml;
    if (worth) {
      lead = min(lead + int(min(made, uint64_t(65536))) - worth, kWorthLead * worth);
      if (lead < -kWorthLag * worth)
        return kDecodeLeft;
    }
  }
}

// ... called, for the registers of the kernels of whole CTAs
__device__ CHUCKY_NOINLINE uint32_t lz4_decode_serial(const uint8_t* src,
                                                      uint64_t n,
                                                      uint8_t* dst,
                                                      uint64_t chunk_bytes,
                                                      int worth,
                                                      uint64_t& ip_out,
                                                      uint64_t& op_out)
{
  uint64_t ip = 0, op = 0;
  const uint32_t st = lz4_decode_warp<true>(src, n, dst, chunk_bytes, worth, ip, op);
  ip_out = ip;
  op_out = op;
  return st;
}

// ---- the tiled decoder -------------------------------------------------------

constexpr uint32_t kPer = 16;       // window positions / tile bytes per thread
constexpr uint32_t kWarpSpan = 512; // window positions per warp
static_assert(kWarpSpan == 32 * kPer, "a warp's threads share its span");
// length bytes of one field followed inside a window (each adds 255)
constexpr uint32_t kMaxExt = 32;
// ... and those of one that is copied without a window being parsed: a length
// of 525 in a small tile, 2,055 in a large one, which holds several such; in a
// block of half a small tile, whose window is parsed anyway, most of the block.
// 300 blocks of 16 KiB that are constant or random take 23 us in small tiles
// (62 with random ones of 8 KiB and up taken so).
template<int NT>
__device__ __forceinline__ uint32_t lz4_peek_bytes(uint64_t chunk_bytes)
{
  if (NT <= 256 && chunk_bytes <= 2048)
    return (uint32_t(chunk_bytes) * 3 / 4 + 239) / 255;
  return NT <= 256 ? 2 : 8;
}
// where the chain goes from a position: the next token's position, or
constexpr uint32_t kStop = 0x8000;  // | position: that token is not complete here
constexpr uint32_t kEnd = 0xFFFE;   // the block's last sequence

// One sequence of a tile, as tile_run wants it.
struct LzTok
{
  uint16_t bound; // (its bytes, until its place is known)
  uint16_t off;   // (0: none, the last sequence)
  int32_t dlit;   // (literals << 16 | the window position of the first)
};

template<int NT>
struct LzShared
{
  static constexpr uint32_t kWindow = NT * kPer;
  static constexpr uint32_t kWarps = NT / 32;
  alignas(16) uint8_t win[kWindow + 32]; // compressed bytes (16-byte phase kept)
  union
  {
    struct
    {
      uint16_t next[kWindow]; // chain step of every position
      uint16_t exit[kWindow]; // where it leaves the position's 32-byte piece
    } p;
    struct
    {
      LzTile<NT> tile;
      LzTok tok[kWindow / 3 + 3]; // (a sequence takes >= 3 bytes)
    } t;
  };
  uint32_t mask[NT / 2];      // tokens among 32 window positions each
  uint16_t exit2[kWarps][32]; // where a span's first 32 positions leave it
  uint16_t entry[kWarps];     // the chain's first position in each span
  uint32_t warp_sum[kWarps];
  uint32_t chain_end;         // where the chain left the window (as `next`)
  uint32_t cut, cut_pos, cut_out; // first sequence past the tile
  uint32_t found;             // (long sequences) first byte that is not 255
  uint32_t bad;
};

// The sequence at window position p: its literals and match, and the chain
// step (the return value).  Straight-line for the common lengths: the first
// length byte of either field is loaded whether it is needed or not (the
// window is padded), only a second one takes a loop.
__device__ __forceinline__ uint32_t lz4_step(const uint8_t* b,
                                             uint32_t p,
                                             uint32_t wlen,
                                             bool at_end,
                                             uint32_t& src,
                                             uint32_t& lit,
                                             uint32_t& ml,
                                             uint32_t& off)
{
  const uint32_t t = b[p], x = b[p + 1];
  lit = t >> 4;
  src = p + 1;
  if (lit == 15) {
    lit += x;
    ++src;
    if (x == 255) {
      uint32_t y = 255;
      for (uint32_t c = 1; y == 255; ++c) {
        if (src >= wlen || c == kMaxExt)
          return kStop | p;
        y = b[src++];
        lit += y;
      }
    }
  }
  const uint32_t e = src + lit; // past the literals
  off = ml = 0;
  if (e + 2 > wlen)
    return at_end && e == wlen ? kEnd : (kStop | p);
  off = uint32_t(b[e]) | uint32_t(b[e + 1]) << 8;
  ml = (t & 15) + 4;
  uint32_t q = e + 2;
  if (ml == 19) {
    uint32_t y = b[q++];
    ml += y;
    for (uint32_t c = 1; y == 255; ++c) {
      if (q >= wlen || c == kMaxExt)
        return kStop | p;
      y = b[q++];
      ml += y;
    }
    if (q > wlen)
      return kStop | p;
  }
  return q;
}

// The length bytes at ip of a field that is already at its nibble's limit,
// by the whole CTA; false when the block ends inside them.
template<int NT>
__device__ bool lz4_long_length(LzShared<NT>& S,
                                const uint8_t* src,
                                uint64_t n,
                                uint64_t& ip,
                                uint64_t& len)
{
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0)
      S.found = NT;
    __syncthreads();
    const uint64_t at = ip + threadIdx.x;
    if (at >= n || src[at] != 255)
      atomicMin(&S.found, threadIdx.x);
    __syncthreads();
    const uint32_t f = S.found;
    len += uint64_t(f) * 255;
    ip += f;
    if (f < uint32_t(NT))
      break;
  }
  if (ip >= n)
    return false;
  len += src[ip++];
  return true;
}

// What the parse hands to the execution: a tile whose sequences are listed
// (lit: its bytes), or one sequence of any length.
struct LzWork
{
  enum : uint32_t
  {
    kDone,
    kTile,
    kLong,
  };
  uint32_t kind;
  const uint8_t* lits; // (a tile: the window's first byte)
  uint8_t* to;
  uint64_t lit, off, ml;
};

// One sequence of any length at ip, read by the whole CTA; false: malformed.
template<int NT>
__device__ bool lz4_long_sequence(LzShared<NT>& S,
                                  const uint8_t* src,
                                  uint64_t n,
                                  uint8_t* dst,
                                  uint64_t chunk_bytes,
                                  uint64_t& ip,
                                  uint64_t& op,
                                  bool& last,
                                  LzWork& q)
{
  if (ip >= n)
    return false;
  const uint32_t token = src[ip++];
  uint64_t lit = token >> 4;
  if (lit == 15 && !lz4_long_length(S, src, n, ip, lit))
    return false;
  if (lit > n - ip || lit > chunk_bytes - op)
    return false;
  q = LzWork{ LzWork::kLong, src + ip, dst + op, lit, 0, 0 };
  ip += lit;
  op += lit;
  last = ip == n;
  if (last)
    return true;
  if (n - ip < 2)
    return false;
  q.off = uint64_t(src[ip]) | uint64_t(src[ip + 1]) << 8;
  ip += 2;
  q.ml = (token & 15) + 4;
  if (q.ml == 19 && !lz4_long_length(S, src, n, ip, q.ml))
    return false;
  if (q.off == 0 || q.off > op || q.ml > chunk_bytes - op)
    return false;
  op += q.ml;
  return true;
}

// ... and copied by the whole CTA
template<int NT>
__device__ void lz4_copy_long(const LzWork& q)
{
  copy_exact(q.to, q.lits, q.lit, threadIdx.x, NT);
  __syncthreads(); // the literals
  if (q.ml)
    cta_match<NT>(q.to + q.lit, q.off, q.ml);
  __syncthreads();
}

// A CTA executes what it has parsed: the list is in its shared memory.
template<int NT>
struct LzOwn
{
  LzShared<NT>& S;
  __device__ LzTok* tok() { return S.t.tok; }
  __device__ void tile(const uint8_t*, const uint8_t* b, uint8_t* to, uint32_t nout)
  {
    // (a last sequence of no bytes follows all marked ones)
    tile_run<NT, 6>(S.t.tile, S.warp_sum, S.t.tok, b, to, nout);
  }
  __device__ void run_long(const LzWork& q) { lz4_copy_long<NT>(q); }
};

// `n` bytes of a block at src by all NT threads, from ip and op on; false when
// it is malformed.  X: who executes the tiles.
template<int NT, typename X>
__device__ bool lz4_decode_tiles(LzShared<NT>& S,
                                 X& exec,
                                 const uint8_t* src,
                                 const uint64_t n,
                                 uint8_t* dst,
                                 const uint64_t chunk_bytes,
                                 uint64_t ip = 0,
                                 uint64_t op = 0)
{
  using Sh = LzShared<NT>;
  constexpr unsigned kAll = 0xffffffffu;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t want = Sh::kWindow; // window bytes worth parsing
  bool peek = true;            // a long sequence may follow
  auto run_long = [&](bool& last) {
    LzWork q;
    if (!lz4_long_sequence(S, src, n, dst, chunk_bytes, ip, op, last, q))
      return false;
    exec.run_long(q);
    want = Sh::kWindow;
    peek = true;
    return true;
  };
  for (;;) {
    if (ip >= n)
      return false;
    if (peek) {
      // a long literal run (an incompressible block is one) and a long match
      // behind a few literals (constant data is one after another) are known
      // by their length bytes: no window is parsed for them
      peek = false;
      const uint32_t bytes = lz4_peek_bytes<NT>(chunk_bytes);
      auto full = [&](uint64_t at) { return lane >= bytes || (at + lane < n && src[at + lane] == 255); };
      bool is_long = full(ip + 1); // (loaded beside the token, not behind it)
      const uint32_t t = src[ip];
      if (t >> 4 != 15)
        is_long = (t & 15) == 15 && full(ip + 3 + (t >> 4));
      if (__all_sync(kAll, is_long)) {
        bool last = false;
        if (!run_long(last))
          return false;
        if (last)
          return op == chunk_bytes;
        continue;
      }
    }
    const uint32_t wlen = uint32_t(n - ip < want ? n - ip : want);
    const bool at_end = ip + wlen == n;
    // ---- the window, in the 16-byte phase of the block
    const uint32_t sh = uint32_t(reinterpret_cast<uintptr_t>(src + ip) & 15);
    const uint8_t* b = S.win + sh;
    for (uint32_t v = tid; v * 16 < sh + wlen; v += NT) {
      const uint32_t lo = v * 16, hi = lo + 16;
      const uint8_t* g = src + ip + lo - sh; // (formed for the inner vectors)
      if (lo >= sh && hi <= sh + wlen) {
        *reinterpret_cast<uint4*>(S.win + lo) = *reinterpret_cast<const uint4*>(g);
      } else {
        for (uint32_t k = lo < sh ? sh : lo; k < hi && k < sh + wlen; ++k)
          S.win[k] = src[ip + k - sh];
      }
    }
    if (lane == 0)
      S.entry[warp] = 0xFFFFu;
    if (tid == 0) {
      S.cut = ~0u;
      S.bad = 0;
    }
    __syncthreads();
    // ---- chain steps and the exits of 32-byte pieces
    const uint32_t w0 = warp * kWarpSpan;
    if (w0 < wlen) {
#pragma unroll 4
      for (uint32_t i = 0; i < kPer; ++i) {
        const uint32_t base = w0 + 32 * i, p = base + lane;
        uint32_t a, l, m, o;
        uint32_t j = p < wlen ? lz4_step(b, p, wlen, at_end, a, l, m, o) : (kStop | p);
        S.p.next[p] = uint16_t(j);
        // a piece holds at most 11 tokens: four doublings
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t r = __shfl_sync(kAll, j, int((j - base) & 31));
          if (j - base < 32)
            j = r;
        }
        S.p.exit[p] = uint16_t(j);
      }
      __syncwarp();
      uint32_t e = w0 + lane;
      do // (leaves the first piece, then hops over the others)
        e = S.p.exit[e];
      while (e < w0 + kWarpSpan && e < wlen);
      S.exit2[warp][lane] = uint16_t(e);
    }
    __syncthreads();
    // ---- the chain through the spans
    if (tid == 0) {
      uint32_t e = 0;
      do {
        const uint32_t w = e / kWarpSpan, r = e % kWarpSpan;
        S.entry[w] = uint16_t(e);
        if (r < 32) {
          e = S.exit2[w][r];
        } else {
          const uint32_t hi = (w + 1) * kWarpSpan;
          do
            e = S.p.exit[e];
          while (e < hi && e < wlen);
        }
      } while (e < wlen);
      S.chain_end = e;
    }
    __syncthreads();
    // ---- the tokens: each span's chain over its pieces, then each piece's
    uint32_t mine = 0xFFFFu;
    {
      uint32_t e = S.entry[warp];
      while (e < w0 + kWarpSpan && e < wlen) {
        if (lane == ((e - w0) >> 5))
          mine = e;
        e = S.p.exit[e];
      }
    }
    if (lane < kPer) {
      uint32_t m = 0;
      const uint32_t hi = w0 + 32 * (lane + 1);
      for (uint32_t p = mine; p < hi && p < wlen;) {
        const uint32_t x = S.p.next[p];
        if (x >= kStop && x != kEnd)
          break;
        m |= 1u << (p & 31);
        p = x;
      }
      S.mask[warp * kPer + lane] = m;
    }
    __syncthreads();
    uint32_t ntok;
    {
      // two threads per piece: 16 positions each
      const uint32_t half = (S.mask[tid >> 1] >> (16 * (tid & 1))) & 0xFFFFu;
      const uint32_t at = cta_scan<NT>(uint32_t(__popc(half)), S.warp_sum, ntok);
      // parse them once more, now that they are tokens (the chain arrays'
      // room is reused: everybody is past them)
      uint32_t sum = 0, k = at, bits = half;
      while (bits) {
        const uint32_t p = (tid >> 1) * 32 + 16 * (tid & 1) + uint32_t(__ffs(int(bits)) - 1);
        bits &= bits - 1;
        uint32_t a = 0, l = 0, m = 0, o = 0;
        const uint32_t x = lz4_step(b, p, wlen, at_end, a, l, m, o);
        if (o == 0 && x != kEnd)
          S.bad = 1; // (an offset of 0)
        S.t.tok[++k] = LzTok{ uint16_t(l + m), uint16_t(o), int32_t(l << 16 | a) };
        sum += l + m;
      }
      tile_clear(S.t.tile);
      uint32_t total;
      uint32_t out = cta_scan<NT>(sum, S.warp_sum, total);
      const uint32_t shd = uint32_t(reinterpret_cast<uintptr_t>(dst + op) & 15);
      bits = half;
      for (k = at; bits; ++k, bits &= bits - 1) {
        const LzTok t = S.t.tok[k + 1];
        const uint32_t len = t.bound, l = uint32_t(t.dlit) >> 16, a = uint32_t(t.dlit) & 0xFFFFu;
        if (out <= LzTile<NT>::kBytes && out + len > LzTile<NT>::kBytes) { // first past the tile
          S.cut = k;
          S.cut_pos = (tid >> 1) * 32 + 16 * (tid & 1) + uint32_t(__ffs(int(bits)) - 1);
          S.cut_out = out;
        }
        if (out + len <= LzTile<NT>::kBytes) {
          exec.tok()[k + 1] =
            LzTok{ uint16_t(shd + out + l), t.off, int32_t(a) - int32_t(shd + out) };
          if (t.off > op + out + l)
            S.bad = 1;
          if (len)
            tile_mark(S.t.tile, shd, out);
        }
        out += len;
      }
      __syncthreads();
      const bool cut = S.cut != ~0u;
      const uint32_t chain_end = S.chain_end;
      if (S.bad)
        return false;
      const uint32_t nout = cut ? S.cut_out : total;
      const uint32_t used =
        cut ? S.cut_pos
            : (chain_end == kEnd ? wlen : (chain_end >= kStop ? chain_end - kStop : chain_end));
      if (nout > chunk_bytes - op)
        return false;
      if (used == 0) { // a sequence that fits neither window nor tile
        bool last = false;
        __syncthreads(); // (S.bad and S.cut have been read)
        if (!run_long(last))
          return false;
        if (last)
          return op == chunk_bytes;
        continue;
      }
      exec.tile(src + ip, b, dst + op, nout);
      ip += used;
      op += nout;
      if (!cut && chain_end == kEnd)
        return op == chunk_bytes;
      // a well compressed block fills the tile from part of the window:
      // parse about as much next time
      const uint32_t next = cut ? used + used / 4 + kWarpSpan : 2 * wlen;
      want = next < Sh::kWindow ? next : Sh::kWindow;
    }
    __syncthreads(); // the tile is final and the shared arrays free
  }
}

// Whether a block has few sequences, by its size: it saved less than a 64th of
// its bytes (matches are rare), or takes less than an eighth (a sequence is
// three bytes or more).
__device__ __forceinline__ bool lz4_few_by_size(uint64_t n, uint64_t chunk_bytes)
{
  return n < chunk_bytes / 8 || n >= chunk_bytes - chunk_bytes / 64;
}

// Whether it starts with kLongSequence literals, which a CTA copies sooner
// (every lane of a warp).
__device__ __forceinline__ bool lz4_long_start(const uint8_t* src, uint64_t n)
{
  constexpr uint32_t kBytes = kLongSequence / 255 + 1;
  static_assert(kBytes > 32 && kBytes <= 96, "two or three length bytes per lane");
  bool full = n > kBytes && src[0] >> 4 == 15;
  for (uint32_t k = threadIdx.x & 31; k < kBytes && full; k += 32)
    full = src[1 + k] == 255;
  return __all_sync(0xffffffffu, full);
}

// kMany: CTAs below `groups` take `per` blocks each (a warp a block at most): the
// warps decode those of few sequences alone, as far as that is worth it, and the
// CTA then goes over what they left.  The others take one of the remaining
// blocks each.  A warp needs no barriers, and the chip holds 32 of them per SM,
// but it waits 0.3 to 0.65 us for every sequence.
template<int NT, bool kMany>
__global__ void __launch_bounds__(NT, NT <= 256 ? kSmallCtas : 1)
lz4_decode_k(const uint8_t* in,
             const uint64_t* in_off,
             const uint64_t* in_size,
             uint64_t n_chunks,
             uint8_t* out,
             uint64_t out_stride,
             uint64_t chunk_bytes,
             uint32_t* status,
             uint32_t groups,
             uint32_t per,
             int worth)
{
  CHUCKY_DYN_SHARED(uint4, sm);
  LzShared<NT>& S = *reinterpret_cast<LzShared<NT>*>(sm);
  auto block = [&](uint64_t c, uint64_t ip, uint64_t op) {
    const uint8_t* src = in + in_off[c];
    const uint64_t n = in_size[c];
    uint8_t* dst = out + c * out_stride;
    LzOwn<NT> own{ S };
    const bool ok = lz4_decode_tiles<NT>(S, own, src, n, dst, chunk_bytes, ip, op);
    __syncthreads();
    if (threadIdx.x < 32) {
      uint64_t ip0 = 0, op0 = 0;
      const uint32_t st =
        ok      ? uint32_t(kDecodeOk)
        : kMany ? lz4_decode_serial(src, n, dst, chunk_bytes, 0, ip0, op0)
                : lz4_decode_warp<false>(src, n, dst, chunk_bytes, 0, ip0, op0);
      if (threadIdx.x == 0)
        status[c] = st;
    }
    __syncthreads();
  };
  if constexpr (kMany) {
    __shared__ uint64_t left_ip[NT / 32], left_op[NT / 32];
    __shared__ uint32_t left[NT / 32];
    const uint32_t warp = threadIdx.x >> 5;
    const bool group = blockIdx.x < groups;
    uint64_t c0 = blockIdx.x - groups;
    uint32_t m = 1;
    if (group) {
      c0 = uint64_t(blockIdx.x) * per;
      m = uint32_t(n_chunks - c0 < per ? n_chunks - c0 : per);
      if (warp < m) {
        const uint64_t c = c0 + warp, n = in_size[c];
        const uint8_t* src = in + in_off[c];
        uint64_t ip = 0, op = 0;
        uint32_t st = kDecodeOk; // (another CTA's block)
        if (lz4_few_by_size(n, chunk_bytes) && !lz4_long_start(src, n)) {
          st = lz4_decode_serial(src, n, out + c * out_stride, chunk_bytes, worth, ip, op);
          if (st != kDecodeLeft && (threadIdx.x & 31) == 0)
            status[c] = st;
        }
        if ((threadIdx.x & 31) == 0) {
          left_ip[warp] = ip;
          left_op[warp] = op;
          left[warp] = st;
        }
      }
      __syncthreads();
    } else if (const uint64_t n = in_size[c0]; lz4_few_by_size(n, chunk_bytes)) {
      const bool keep = warp == 0 && lz4_long_start(in + in_off[c0], n);
      if (!__syncthreads_or(keep))
        return; // (a warp's block)
    }
    for (uint32_t k = 0; k < m; ++k)
      if (!group || left[k] == kDecodeLeft) // (the whole CTA)
        block(c0 + k, group ? left_ip[k] : 0, group ? left_op[k] : 0);
  } else {
    for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x)
      block(c, 0, 0);
  }
}

// A warp per block, for chunks too small for more.
constexpr int kAloneThreads = 128;
__global__ void __launch_bounds__(kAloneThreads) lz4_decode_alone_k(const uint8_t* in,
                                                                    const uint64_t* in_off,
                                                                    const uint64_t* in_size,
                                                                    uint64_t n_chunks,
                                                                    uint8_t* out,
                                                                    uint64_t out_stride,
                                                                    uint64_t chunk_bytes,
                                                                    uint32_t* status)
{
  constexpr uint32_t kWarps = kAloneThreads / 32;
  for (uint64_t c = uint64_t(blockIdx.x) * kWarps + (threadIdx.x >> 5); c < n_chunks;
       c += uint64_t(gridDim.x) * kWarps) {
    uint64_t ip = 0, op = 0;
    const uint32_t st = lz4_decode_warp<false>(in + in_off[c], in_size[c], out + c * out_stride,
                                               chunk_bytes, 0, ip, op);
    if ((threadIdx.x & 31) == 0)
      status[c] = st;
  }
}

#ifndef CHUCKY_LZ4_UNPAIRED // (the CPU emulation of the kernels has no clusters)
// Two CTAs per block, a cluster: the first parses the block and lists the
// sequences of one tile after another in the second's shared memory, the
// second executes a tile while the first parses the next.  A cluster barrier
// per tile; both CTAs pass the same ones: the first ends its block with a
// kDone of its own, the second leaves its loop only there.  Bound by the parse
// and placement (12 of 20 us per tile), the longer half; over both CTAs 43 % of
// the issue slots are taken, and a third of the stalls are at the CTA's own
// barriers.
template<int NT>
struct LzPairShared // the second CTA's
{
  LzTile<NT> tile;
  struct
  {
    LzWork work;
    uint32_t start[NT / 2 + 1];
    LzTok tok[LzShared<NT>::kWindow / 3 + 3];
  } slot[2];
  uint32_t warp_sum[NT / 32];
};

__device__ __forceinline__ void pair_barrier()
{
  asm volatile("barrier.cluster.arrive.release;\n\t"
               "barrier.cluster.wait.acquire;" ::
                 : "memory");
}

template<int NT>
struct LzOther
{
  LzShared<NT>& S;
  LzPairShared<NT>& P; // (in the second CTA's shared memory)
  uint32_t turn;       // the slot being filled
  __device__ LzTok* tok() { return P.slot[turn].tok; }
  __device__ void post(const LzWork& q)
  {
    if (threadIdx.x == 0)
      P.slot[turn].work = q;
    pair_barrier();
    turn ^= 1;
  }
  __device__ void tile(const uint8_t* lits, const uint8_t*, uint8_t* to, uint32_t nout)
  {
    for (uint32_t i = threadIdx.x; i < NT / 2 + 1; i += NT)
      P.slot[turn].start[i] = S.t.tile.start[i];
    post(LzWork{ LzWork::kTile, lits, to, nout, 0, 0 });
  }
  __device__ void run_long(const LzWork& q) { post(q); }
};

template<int NT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NT)
lz4_decode_pair_k(const uint8_t* in,
                  const uint64_t* in_off,
                  const uint64_t* in_size,
                  uint64_t n_chunks,
                  uint8_t* out,
                  uint64_t out_stride,
                  uint64_t chunk_bytes,
                  uint32_t* status)
{
  CHUCKY_DYN_SHARED(uint4, sm);
  const bool first = (blockIdx.x & 1) == 0;
  pair_barrier(); // the second CTA's shared memory exists
  uint32_t turn = 0;
  for (uint64_t c = blockIdx.x >> 1; c < n_chunks; c += gridDim.x >> 1) {
    if (first) {
      LzShared<NT>& S = *reinterpret_cast<LzShared<NT>*>(sm);
      uint64_t p = 0;
      asm("mapa.u64 %0, %1, 1;" : "=l"(p) : "l"(reinterpret_cast<uint64_t>(sm)));
      LzOther<NT> other{ S, *reinterpret_cast<LzPairShared<NT>*>(p), turn };
      const uint8_t* src = in + in_off[c];
      const uint64_t n = in_size[c];
      uint8_t* dst = out + c * out_stride;
      const bool ok = lz4_decode_tiles<NT>(S, other, src, n, dst, chunk_bytes);
      __syncthreads(); // (a malformed block leaves from anywhere)
      other.post(LzWork{ LzWork::kDone, nullptr, nullptr, 0, 0, 0 });
      turn = other.turn;
      // every tile is executed
      if (threadIdx.x < 32) {
        uint64_t ip = 0, op = 0;
        const uint32_t st =
          ok ? uint32_t(kDecodeOk)
             : lz4_decode_warp<false>(src, n, dst, chunk_bytes, 0, ip, op);
        if (threadIdx.x == 0)
          status[c] = st;
      }
      __syncthreads();
    } else {
      LzPairShared<NT>& P = *reinterpret_cast<LzPairShared<NT>*>(sm);
      for (;;) {
        pair_barrier();
        const auto& slot = P.slot[turn];
        turn ^= 1;
        const LzWork q = slot.work;
        if (q.kind == LzWork::kDone)
          break;
        if (q.kind == LzWork::kLong) {
          lz4_copy_long<NT>(q);
          continue;
        }
        for (uint32_t i = threadIdx.x; i < NT / 2 + 1; i += NT)
          P.tile.start[i] = slot.start[i]; // (tile_run reads them behind a barrier)
        tile_run<NT, 6>(P.tile, P.warp_sum, slot.tok, q.lits, q.to, uint32_t(q.lit));
      }
    }
  }
}

template<int NT>
cudaError_t launch_lz4_decode_pair(const uint8_t* in,
                                   const uint64_t* in_off,
                                   const uint64_t* in_size,
                                   uint64_t n_chunks,
                                   uint8_t* out,
                                   uint64_t out_stride,
                                   uint64_t chunk_bytes,
                                   uint32_t* status,
                                   cudaStream_t st)
{
  constexpr size_t smem = sizeof(LzShared<NT>) > sizeof(LzPairShared<NT>)
                            ? sizeof(LzShared<NT>)
                            : sizeof(LzPairShared<NT>);
  const cudaError_t e = cudaFuncSetAttribute(
    lz4_decode_pair_k<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess)
    return e;
  lz4_decode_pair_k<NT><<<unsigned(2 * n_chunks), NT, smem, st>>>(
    in, in_off, in_size, n_chunks, out, out_stride, chunk_bytes, status);
  note_launches(1);
  return cudaGetLastError();
}
#endif

template<int NT, bool kMany>
cudaError_t launch_lz4_decode_nt(const uint8_t* in,
                                 const uint64_t* in_off,
                                 const uint64_t* in_size,
                                 uint64_t n_chunks,
                                 uint8_t* out,
                                 uint64_t out_stride,
                                 uint64_t chunk_bytes,
                                 uint32_t* status,
                                 uint32_t per,
                                 int worth,
                                 cudaStream_t st)
{
  constexpr size_t smem = sizeof(LzShared<NT>);
  const cudaError_t e = cudaFuncSetAttribute(
    lz4_decode_k<NT, kMany>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess)
    return e;
  const uint64_t groups = kMany ? (n_chunks + per - 1) / per : 0, ctas = groups + n_chunks;
  const uint64_t grid = ctas < 0x7FFFFFFFull ? ctas : 0x7FFFFFFFull;
  CHUCKY_LAUNCH((lz4_decode_k<NT, kMany>), unsigned(grid), NT, smem, st, in, in_off, in_size,
                n_chunks, out, out_stride, chunk_bytes, status, uint32_t(groups), per, worth);
  note_launches(1);
  return cudaGetLastError();
}

} // namespace

cudaError_t launch_lz4_decode(const uint8_t* in,
                              const uint64_t* in_off,
                              const uint64_t* in_size,
                              uint64_t n_chunks,
                              uint8_t* out,
                              uint64_t out_stride,
                              uint64_t chunk_bytes,
                              uint32_t* status,
                              cudaStream_t st)
{
  // CTAs of 1,024 threads (one per SM) take the least time per chunk, CTAs of
  // 256 (tiles of 4 KiB) keep more chunks on the chip.  us, for sensor counts, a
  // textured volume (rare matches), noise, and chunks that are constant or
  // random:
  //   chunks x bytes   256                1,024              two CTAs
  //      64 x 4,096     19  24  10  14     18  18  10  15
  //      64 x 16,384    64  65  10  21     27  33  10  24
  //      64 x 65,536   222 205  11  55     97  90  11  52     79  70  11  44
  //     300 x 16,384    69  69  10  24     48  59  35  40
  //     300 x 65,536   243 222  13  60    190 174  16  97
  //     456 x 65,536   276 249  16  68    281 257  23 141
  // So: the small ones for chunks of one of their tiles, for chunks of one large
  // tile when there are more than SMs (each form is the better one for half of
  // the data there), and for more than two waves of larger ones; two CTAs per
  // chunk where they fit the chip side by side and there is a second tile to
  // parse ahead.
  //
  // From two waves of small CTAs on (four per SM; from one for chunks up to 1
  // KiB) warps decode the blocks of few sequences first; with fewer blocks a
  // wave of CTAs is as quick.  A sequence must be worth its 0.65 us, with 32
  // warps on an SM, against the CTA's 4.7 us per KiB of each of its chunks.
  // us, every chunk to a CTA / so / every chunk to a warp:
  //   chunks x bytes     sensor counts   volume           constant or random
  //   1,467 x 4,440       80  81  260     72  32  38      76  16  30
  //   4,096 x 4,096      126 130  325    149  38  40     141  20  34
  //   4,096 x 8,192      280 287  719    251  82  81     204  26  62
  //   2,048 x 16,384     288 293 1111    247 129 143     199  36  93
  // Chunks of up to 512 bytes are all left to single warps (608 of 256 bytes: 3.3
  // us on the device, 9.2 with CTAs; 64 sensor ones of 500 bytes 13.5 and 10.6),
  // and so are many of up to 1 KiB (4,096 of sensor counts: 54 and 82 us).
  const uint64_t sms = uint64_t(device_sm_count()), slots = CHUCKY_LZ4_SLOTS(sms);
  constexpr int kSmallNT = CHUCKY_DECODE_THREADS, kNT = CHUCKY_LZ4_THREADS;
  constexpr uint64_t kSmallTile = kSmallNT * 16, kTile = kNT * 16;
  if (chunk_bytes <= 512 || (chunk_bytes <= 1024 && n_chunks > 3 * slots)) {
    constexpr uint32_t kWarps = kAloneThreads / 32;
    const uint64_t ctas = (n_chunks + kWarps - 1) / kWarps;
    CHUCKY_LAUNCH(lz4_decode_alone_k, unsigned(ctas < 0x7FFFFFFFull ? ctas : 0x7FFFFFFFull),
                  kAloneThreads, 0, st, in, in_off, in_size, n_chunks, out, out_stride,
                  chunk_bytes, status);
    note_launches(1);
    return cudaGetLastError();
  }
#ifndef CHUCKY_LZ4_UNPAIRED
  if (chunk_bytes > kTile && n_chunks <= sms / 2)
    return launch_lz4_decode_pair<kNT>(in, in_off, in_size, n_chunks, out, out_stride,
                                       chunk_bytes, status, st);
#endif
  if (chunk_bytes > kSmallTile && n_chunks <= (chunk_bytes <= kTile ? sms : 2 * sms))
    return launch_lz4_decode_nt<kNT, false>(in, in_off, in_size, n_chunks, out, out_stride,
                                            chunk_bytes, status, 1, 0, st);
  if (n_chunks <= (chunk_bytes <= 1024 ? 1 : 2) * slots || n_chunks >= (1ull << 30))
    return launch_lz4_decode_nt<kSmallNT, false>(in, in_off, in_size, n_chunks, out, out_stride,
                                                 chunk_bytes, status, 1, 0, st);
  const uint64_t share = (n_chunks + slots - 1) / slots;
  const uint32_t per = uint32_t(share < kSmallNT / 32 ? share : kSmallNT / 32);
  return launch_lz4_decode_nt<kSmallNT, true>(in, in_off, in_size, n_chunks, out, out_stride,
                                              chunk_bytes, status, per,
                                              160 / int(per > 2 ? per - 1 : 1), st);
}

} // namespace chucky

extern "C" int chucky_lz4_decode_chunks(const void* d_in,
                                        const uint64_t* d_in_offsets,
                                        const uint64_t* d_in_sizes,
                                        size_t n_chunks,
                                        void* d_out,
                                        size_t out_stride,
                                        size_t chunk_bytes,
                                        uint32_t* d_status,
                                        void* cuda_stream)
{
  if (n_chunks == 0)
    return 0;
  if (!d_in || !d_in_offsets || !d_in_sizes || !d_out || !d_status ||
      out_stride < chunk_bytes)
    return 1;
  const cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  if (n_chunks > (uint64_t(1) << 32))
    return 1;
  return chucky::launch_lz4_decode(static_cast<const uint8_t*>(d_in), d_in_offsets,
                                   d_in_sizes, n_chunks, static_cast<uint8_t*>(d_out),
                                   out_stride, chunk_bytes, d_status, st) == cudaSuccess
           ? 0
           : 3;
}
