// zstd frames decoded block-parallel (RFC 8878).  Included by zstd_decode.cu.
//
// Within a frame only three things are sequential: where a block lies in the
// input (block sizes), which tables a block repeats, and the output bytes a
// match copies.  The rest of a block -- its Huffman streams and its FSE
// sequence stream, where the time goes -- depends on its own bytes and those
// tables alone.  So:
//   zd_parse_k    a warp per frame walks the block headers and notes for
//                 every block where its sections lie and which blocks
//                 describe the tables it uses;
//   zd_seq_k      a warp per run of blocks decodes their sequences (tables
//                 built by the whole warp, the state chain on one lane) to a
//                 list, with repeat offsets left symbolic (they name the
//                 block's starting offsets), and sums up the block's output;
//   zd_place_k    a warp per frame: output offset and starting repeat offsets
//                 of every block, and whether the frame fills the chunk;
//   zd_lit_k      a warp per eight blocks: Huffman streams, a lane each (32 in
//                 flight when the blocks share a table), into the end of the
//                 block's own output range.  A block's literals there never
//                 lie before the bytes still to be written: no literal
//                 buffer, and a block without sequences is finished;
//   zd_exec_k     a CTA per frame executes the sequences tile by tile
//                 (lz_tile.cuh).
// A frame that is anything but one conforming frame that fills its chunk
// (malformed, several frames, skippable ones, a dictionary, more blocks or
// sequences than the lists hold) is flagged on the way and decoded by the
// sequential kernel afterwards, which sets its status.
//
// Bound by latency: a Huffman symbol takes 45 ns on its lane, a sequence 220
// ns, a tile of 8 KiB 5 us.  64 chunks of the u16 cube (512 KiB each, level 3:
// 1,370 sequences per 8 KiB block) take 0.99 ms -- 0.04 parse, 0.37 sequences,
// 0.13 literals, 0.4 execution -- against 167 ms for the sequential decoder;
// 64 sensor chunks (4 MiB, level 1) 3.3 ms.
#pragma once

#include "lz_tile.cuh"

namespace chucky {

namespace {

constexpr int32_t kPredef = -2;

struct ZBlk
{
  uint64_t src;      // the block's content, from the chunk's first byte
  uint64_t out;      // its output, from the chunk's first byte
  uint32_t size;     // content bytes
  uint32_t type;     // 0 raw, 1 RLE, 2 compressed
  uint32_t ltype;    // literals: 0 raw, 1 RLE, 2 Huffman, 3 Huffman with an earlier tree
  uint32_t streams;  // Huffman streams (1 or 4)
  uint32_t tree_at;  // places within the content: the tree,
  uint32_t lit_at;   // the literals or Huffman streams,
  uint32_t lit_len;  // (bytes of the streams)
  uint32_t seq_at;   // the first sequence table description
  uint32_t nlit, nseq;
  uint32_t modes;    // sequence table modes byte
  uint32_t seq0;     // its first sequence in the frame's list
  int32_t huf;       // block that describes its Huffman tree
  int32_t def[3];    // ... its LL, OF and ML tables; kPredef: the predefined ones
  uint32_t regen;    // output bytes
  uint32_t rep[3];   // repeat offsets: after the block (symbolic), then before it
};

struct ZFrame
{
  uint64_t content; // declared content size, ~0: not declared
  uint32_t nblk;
  uint32_t slow;    // left to the sequential decoder
};

struct ZWave // one launch set's chunks and lists
{
  const uint8_t* in;
  const uint64_t* in_off;
  const uint64_t* in_size;
  uint8_t* out;
  uint64_t out_stride, chunk_bytes;
  uint32_t* status;
  uint64_t n;
  ZFrame* frames;  // [n]
  ZBlk* blocks;    // [n][max_blk]
  uint64_t* seqs;  // [n][max_seq]
  uint32_t max_blk, max_seq;
};

// lists of one launch set
#ifndef CHUCKY_ZSTD_SCRATCH
#define CHUCKY_ZSTD_SCRATCH (256ull << 20)
#endif
constexpr uint64_t kZdScratch = CHUCKY_ZSTD_SCRATCH;
// chunks up to this size are decoded sequentially
constexpr uint64_t kZdSequential = 64;
// chunks whose frames' records are kept for one pass of the sequential decoder
#ifndef CHUCKY_ZSTD_FRAMES
#define CHUCKY_ZSTD_FRAMES (1ull << 20)
#endif
constexpr uint64_t kZdFrames = CHUCKY_ZSTD_FRAMES;

// Lists of a frame: blocks of 4 KiB on average or more (the format allows
// less), sequences of 4 bytes on average or more.
inline uint32_t zd_max_blk(uint64_t chunk_bytes) { return uint32_t(chunk_bytes >> 12) + 16; }
inline uint32_t zd_max_seq(uint64_t chunk_bytes) { return uint32_t(chunk_bytes >> 2) + 64; }
inline uint64_t zd_list_bytes(uint64_t chunk_bytes)
{
  return zd_max_blk(chunk_bytes) * sizeof(ZBlk) + zd_max_seq(chunk_bytes) * 8ull;
}

// A sequence in the list: literals (17 bits), match length (18), offset
// (29: the distance, or kSymOff, the index of a starting repeat offset in
// bits 26-27 and what is taken off it below).
constexpr uint32_t kSymOff = 1u << 28;
constexpr uint32_t kSym = 1u << 31; // the same in a 32-bit offset, index in bits 29-30

__device__ __forceinline__ uint32_t zd_rep(uint32_t v, uint32_t r0, uint32_t r1, uint32_t r2)
{
  if (!(v & kSym))
    return v;
  const uint32_t k = (v >> 29) & 3;
  return (k == 0 ? r0 : k == 1 ? r1 : r2) - (v & 0x1FFFFFFFu);
}

// ---- headers -----------------------------------------------------------------

// Sections of a compressed block (RFC 8878 3.1.1.3.1.1, 3.1.1.3.2.1).
__device__ bool zd_block_sections(const uint8_t* p, uint32_t n, ZBlk& B)
{
  if (n < 1)
    return false;
  const uint32_t b0 = p[0], fmt = (b0 >> 2) & 3;
  uint32_t at;
  B.ltype = b0 & 3;
  B.streams = 0;
  if (B.ltype <= 1) {
    at = fmt == 1 ? 2 : fmt == 3 ? 3 : 1;
    if (at > n)
      return false;
    B.nlit = at == 1 ? b0 >> 3
                     : (b0 >> 4) + (uint32_t(p[1]) << 4) + (at == 3 ? uint32_t(p[2]) << 12 : 0u);
    B.lit_at = at;
    const uint32_t len = B.ltype == 0 ? B.nlit : 1;
    if (B.nlit > kBlockMax || len > n - at)
      return false;
    at += len;
  } else {
    at = fmt <= 1 ? 3 : fmt + 2;
    if (at > n)
      return false;
    uint64_t v = 0;
    for (uint32_t k = at; k-- > 0;)
      v = (v << 8) | p[k];
    const int field = at == 3 ? 10 : at == 4 ? 14 : 18;
    B.nlit = uint32_t((v >> 4) & ((1ull << field) - 1));
    const uint32_t comp = uint32_t((v >> (4 + field)) & ((1ull << field) - 1));
    B.streams = fmt == 0 ? 1 : 4;
    if (B.nlit > kBlockMax || comp > n - at)
      return false;
    uint32_t tree = 0;
    if (B.ltype == 2) {
      if (comp < 1)
        return false;
      const uint32_t h = p[at];
      tree = h >= 128 ? 1 + (h - 126) / 2 : 1 + h;
      if (h == 0 || tree > comp)
        return false;
    }
    B.tree_at = at;
    B.lit_at = at + tree;
    B.lit_len = comp - tree;
    at += comp;
  }
  if (at >= n)
    return false;
  B.nseq = p[at++];
  if (B.nseq == 0) {
    B.regen = B.nlit;
    return at == n;
  }
  if (B.nseq >= 128) {
    const uint32_t more = B.nseq == 255 ? 2 : 1;
    if (more > n - at)
      return false;
    B.nseq = more == 2 ? p[at] + (uint32_t(p[at + 1]) << 8) + 0x7F00
                       : ((B.nseq - 128) << 8) + p[at];
    at += more;
    if (B.nseq == 0) // (two bytes that say none: left to the sequential decoder)
      return false;
  }
  if (at >= n)
    return false;
  B.modes = p[at++];
  B.seq_at = at;
  return (B.modes & 3) == 0;
}

__device__ __forceinline__ int warp_last(int v) // inclusive running maximum over lanes
{
  const int lane = threadIdx.x & 31;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o && y > v)
      v = y;
  }
  return v;
}

constexpr int kParseWarps = CHUCKY_DECODE_WARPS;

__global__ void __launch_bounds__(32 * kParseWarps) zd_parse_k(ZWave W)
{
  __shared__ uint64_t s_src[kParseWarps][32];
  __shared__ uint32_t s_head[kParseWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t f = uint64_t(blockIdx.x) * kParseWarps + w;
  if (f >= W.n)
    return; // the whole warp
  const uint8_t* p = W.in + W.in_off[f];
  const uint64_t n = W.in_size[f];
  ZFrame F{ ~uint64_t(0), 0, 1 };
  // frame header (every lane reads the same bytes)
  uint64_t at = 5;
  bool ok = n >= 5 && p[0] == 0x28 && p[1] == 0xB5 && p[2] == 0x2F && p[3] == 0xFD;
  int checksum = 0;
  if (ok) {
    const uint32_t d = p[4];
    const int fcs_flag = int(d >> 6), single = int((d >> 5) & 1);
    checksum = int((d >> 2) & 1);
    const int fcs_bytes = fcs_flag == 0 ? (single ? 1 : 0) : (1 << fcs_flag);
    const uint64_t hdr = uint64_t(single ? 0 : 1) + uint64_t(fcs_bytes);
    ok = !(d & 8) && !(d & 3) && at + hdr <= n;
    if (ok) {
      at += hdr;
      if (fcs_bytes) {
        uint64_t v = 0;
        for (int i = 1; i <= fcs_bytes; ++i)
          v = (v << 8) | p[at - i];
        F.content = v + (fcs_bytes == 2 ? 256 : 0);
      }
    }
  }
  ZBlk* const blk = W.blocks + f * W.max_blk;
  uint32_t nblk = 0;
  uint64_t nseq = 0;
  int huf = -1, def[3] = { -1, -1, -1 };
  bool last = false;
  while (ok && !last) {
    // up to 32 block headers, one after another
    uint32_t got = 0;
    for (; got < 32 && !last && ok; ++got) {
      if (at + 3 > n) {
        ok = false;
        break;
      }
      const uint32_t h = p[at] | (uint32_t(p[at + 1]) << 8) | (uint32_t(p[at + 2]) << 16);
      at += 3;
      const uint32_t type = (h >> 1) & 3, size = h >> 3;
      const uint32_t body = type == 1 ? 1 : size;
      last = h & 1;
      ok = type != 3 && size <= kBlockMax && at + body <= n;
      if (lane == 0) {
        s_src[w][got] = at;
        s_head[w][got] = h;
      }
      at += body;
    }
    if (!ok || nblk + got > W.max_blk) {
      ok = false;
      break;
    }
    __syncwarp();
    // a lane per block
    ZBlk B{};
    const bool mine = uint32_t(lane) < got;
    bool good = true;
    if (mine) {
      const uint32_t h = s_head[w][lane];
      B.src = s_src[w][lane];
      B.type = (h >> 1) & 3;
      B.size = h >> 3;
      if (B.type == 2)
        good = zd_block_sections(p + B.src, B.size, B);
      else
        B.regen = B.nlit = B.size;
    }
    const int b = int(nblk) + lane;
    const bool comp = mine && B.type == 2;
    const int h0 = max(huf, warp_last(comp && B.ltype == 2 ? b : -1));
    B.huf = h0;
    good &= !(comp && B.ltype == 3 && h0 < 0);
    for (int k = 0; k < 3; ++k) { // LL, OF, ML
      // 2 b + 1 where block b takes the predefined table, 2 b where it
      // describes one
      const int mode = int(B.modes >> (6 - 2 * k)) & 3;
      const int d =
        max(def[k], warp_last(comp && B.nseq && mode != 3 ? 2 * b + (mode == 0 ? 1 : 0) : -1));
      B.def[k] = (d & 1) ? kPredef : d >> 1;
      good &= !(comp && B.nseq && d < 0);
      def[k] = __shfl_sync(0xffffffffu, d, 31);
    }
    huf = __shfl_sync(0xffffffffu, h0, 31);
    uint32_t x = comp ? B.nseq : 0;
    const uint32_t own = x;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o)
        x += y;
    }
    B.seq0 = uint32_t(nseq) + x - own;
    for (int k = 0; k < 3; ++k)
      B.rep[k] = kSym | (uint32_t(k) << 29); // unchanged
    if (mine)
      blk[b] = B;
    nseq += __shfl_sync(0xffffffffu, x, 31);
    ok = __all_sync(0xffffffffu, good) && nseq <= W.max_seq;
    nblk += got;
    __syncwarp();
  }
  if (ok && checksum) {
    ok = at + 4 <= n;
    at += 4;
  }
  if (lane == 0) {
    F.nblk = nblk;
    F.slow = !(ok && at == n); // (more than one frame, too)
    W.frames[f] = F;
  }
}

// ---- bits --------------------------------------------------------------------

// A lane's share of the input, staged in shared memory: kWords words from its
// stream's next bit downwards, word k of lane l at [k][l].  All lanes stage
// at the same steps and all loads of a stage are in flight together, so a
// warp waits for memory once per stage; loaded word by word as they were
// needed, one of 32 streams had always left its cache line and the warp
// waited on nearly every symbol.
template<int kWords>
struct ZStage
{
  uint32_t w[kWords][32];
};

// A backward bitstream of n bytes at p, the next bit on top of hi:lo; at least
// 32 bits are there after fill(), and at most 31 are taken before the next.
// left() counts the stream's bits not yet taken: 0 when it is consumed
// exactly, negative past its start (what is read there is never used: the
// caller checks).
struct ZBits
{
  const uint8_t* p;
  uint32_t hi, lo;
  int have;
  uint32_t slot;  // next staged word
  int32_t staged; // left() when everything up to `slot` is taken, + 32 slot

  __device__ __forceinline__ bool init(const uint8_t* q, uint32_t n)
  {
    p = q;
    if (n == 0 || q[n - 1] == 0)
      return false;
    have = 0;
    slot = 0;
    staged = int32_t(n - 1) * 8 + dec_highbit(q[n - 1]);
    return true;
  }
  __device__ __forceinline__ int32_t left() const { return staged - 32 * int32_t(slot) + have; }
  // Stage the words from the next bit on; [in0, in1) may be read.  At least
  // kWords - 4 of them follow the one that holds the next bit.
  template<int kWords>
  __device__ __forceinline__ void stage(ZStage<kWords>& S, const uint8_t* in0, const uint8_t* in1)
  {
    constexpr int kQuads = kWords / 4;
    const int lane = threadIdx.x & 31;
    const int32_t bits = left();
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const int32_t top = int32_t(a & 15) * 8 + (bits > 0 ? bits : 0); // from 16 B below p
    const int32_t quad = (top - 1) >> 7;
    const uint8_t* const s = p - (a & 15) + 16 * int64_t(quad); // the first vector
    uint4 v[kQuads];
    if (s + 16 <= in1 && s - 16 * (kQuads - 1) >= in0) {
      // (vectors below the stream are the input before it: not used)
#pragma unroll
      for (int k = 0; k < kQuads; ++k)
        v[k] = *reinterpret_cast<const uint4*>(s - 16 * k);
#pragma unroll
      for (int k = 0; k < kQuads; ++k) {
        S.w[4 * k][lane] = v[k].w;
        S.w[4 * k + 1][lane] = v[k].z;
        S.w[4 * k + 2][lane] = v[k].y;
        S.w[4 * k + 3][lane] = v[k].x;
      }
    } else { // at the input's first and last bytes
#pragma unroll 1
      for (int k = 0; k < kWords; ++k) {
        const uint8_t* g = s + 12 - 4 * k;
        uint32_t x = 0;
        for (int i = 0; i < 4; ++i)
          if (g + i >= in0 && g + i < in1)
            x |= uint32_t(g[i]) << (8 * i);
        S.w[k][lane] = x;
      }
    }
    const int32_t word = (top - 1) >> 5;
    slot = uint32_t(4 * quad + 3 - word);
    have = top - 32 * word; // 1 .. 32
    hi = S.w[slot][lane] << (32 - have);
    lo = 0;
    ++slot;
    staged = bits - have + 32 * int32_t(slot);
    fill(S);
  }
  // (without a branch: lanes refill at different steps)
  template<int kWords>
  __device__ __forceinline__ void fill(const ZStage<kWords>& S)
  {
    const bool need = have < 32;
    const uint32_t w = S.w[slot < kWords ? slot : kWords - 1][threadIdx.x & 31];
    hi |= need ? w >> (have & 31) : 0u;
    lo = need ? w << ((32 - have) & 31) : lo;
    have += need ? 32 : 0;
    slot += need ? 1 : 0;
  }
  __device__ __forceinline__ void drop(uint32_t nb) // nb <= 31
  {
    hi = __funnelshift_l(lo, hi, nb);
    lo <<= nb;
    have -= int(nb);
  }
  __device__ __forceinline__ uint32_t take(uint32_t nb)
  {
    const uint32_t v = hi >> 1 >> (31 - nb); // (nb 0: 0)
    drop(nb);
    return v;
  }
};

// ---- tables, by a warp --------------------------------------------------------

// Decoding table entry: next state's base (10 bits), bits to read for it
// (from bit 10) and extra bits of the symbol's value (from bit 16) below, the
// symbol's base value (Huffman weights: the symbol) above.
__device__ __forceinline__ uint64_t zd_entry(uint32_t base, int nb, uint32_t sym, int kind)
{
  const uint32_t xb = kind == 0 ? kLLBits[sym] : kind == 1 ? sym : kind == 2 ? kMLBits[sym] : 0;
  const uint32_t v = kind == 0   ? kLLBase[sym]
                     : kind == 1 ? 1u << sym
                     : kind == 2 ? kMLBase[sym]
                                 : sym;
  return uint64_t(base | uint32_t(nb) << 10 | xb << 16) | uint64_t(v) << 32;
}

struct ZFseWork
{
  int16_t norm[64];
  uint16_t next[64]; // states given out per symbol
  uint16_t cum[64];  // regular states before a symbol
  uint32_t text[34]; // a staged description
};

// Decoding table from normalized counts (RFC 8878 4.1.1), as build_fse, by
// the whole warp: walk position i is (i * step) mod size, the r-th position
// at or below `high` goes to the symbol whose counts cover r; states are
// numbered per symbol in position order.  `kind` (0 LL, 1 OF, 2 ML, 3
// Huffman weights) gives the extra bits.  False: the counts do not fill it.
__device__ bool zd_build_fse(uint64_t* t, ZFseWork& S, int nsym, int al, int kind)
{
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, size = 1 << al;
  if (nsym < 1 || nsym > 64)
    return false;
  // regular states and "less than one" symbols (<< 16) before each symbol
  int before[2], sum = 0;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int s = 32 * k + lane;
    const int v = s < nsym ? S.norm[s] : 0;
    const int own = v == -1 ? 1 << 16 : v > 0 ? v : 0;
    int x = own;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kAll, x, o);
      if (lane >= o)
        x += y;
    }
    before[k] = sum + x - own;
    sum += __shfl_sync(kAll, x, 31);
    S.next[s] = uint16_t(v == -1 ? 1 : own);
    S.cum[s] = uint16_t(before[k] & 0xFFFF);
  }
  const int less = sum >> 16;
  if ((sum & 0xFFFF) + less != size)
    return false;
#pragma unroll
  for (int k = 0; k < 2; ++k) { // the latter from the top, in symbol order
    const int s = 32 * k + lane;
    if (s < nsym && S.norm[s] == -1)
      t[size - 1 - (before[k] >> 16)] = uint64_t(s);
  }
  __syncwarp();
  const int high = size - 1 - less;
  const int step = (size >> 1) + (size >> 3) + 3, mask = size - 1;
  int rank0 = 0;
  for (int i0 = 0; i0 < size; i0 += 32) {
    const int i = i0 + lane, pos = (i * step) & mask;
    const bool v = i < size && pos <= high;
    const unsigned m = __ballot_sync(kAll, v);
    if (v) {
      const int r = rank0 + __popc(m & ((1u << lane) - 1));
      int lo = 0; // the last symbol whose states start at or before r
      for (int d = 32; d; d >>= 1)
        if (lo + d < 64 && S.cum[lo + d] <= r)
          lo += d;
      t[pos] = uint64_t(lo);
    }
    rank0 += __popc(m);
  }
  __syncwarp();
  for (int u0 = 0; u0 < size; u0 += 32) {
    const int u = u0 + lane;
    const uint32_t s = u < size ? uint32_t(t[u]) : 64u + uint32_t(lane);
    const unsigned peers = __match_any_sync(kAll, s);
    uint32_t ns = 0;
    if (u < size)
      ns = S.next[s] + __popc(peers & ((1u << lane) - 1));
    __syncwarp();
    if (u < size) {
      if (lane == __ffs(int(peers)) - 1)
        S.next[s] = uint16_t(ns + __popc(peers));
      const int nb = al - dec_highbit(ns);
      t[u] = zd_entry((ns << nb) - uint32_t(size), nb, s, kind);
    }
    __syncwarp();
  }
  return true;
}

// Normalized counts at p, as read_ncount, for the warp: the description is
// staged by all lanes (valid ones are shorter than 128 bytes), lane 0 reads
// it there.
__device__ uint32_t zd_ncount(const uint8_t* p, uint32_t avail, int max_al, int max_sym,
                              ZFseWork& S, int& nsym, int& al)
{
  const uint32_t lane = threadIdx.x & 31;
  {
    uint32_t v = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
      if (4 * lane + k < avail)
        v |= uint32_t(p[4 * lane + k]) << (8 * k);
    S.text[lane] = v;
    if (lane < 2)
      S.text[32 + lane] = 0;
  }
  __syncwarp();
  uint32_t d = 0;
  int s = 0, a = 0;
  if (lane == 0) {
    const uint32_t bits = (avail < 128 ? avail : 128) * 8;
    auto peek = [&](uint32_t at) {
      return __funnelshift_r(S.text[at >> 5], S.text[(at >> 5) + 1], at & 31);
    };
    a = int(peek(0) & 15) + 5;
    uint32_t bit = 4;
    int remaining = (1 << a) + 1, threshold = 1 << a, nb = a + 1;
    bool prev0 = false, ok = a <= max_al && avail > 0;
    while (ok && remaining > 1 && s <= max_sym) {
      if (prev0) { // runs of zero counts: 2-bit repeat flags
        int n0 = 0;
        uint32_t r = 3;
        while (r == 3 && ok) {
          r = peek(bit) & 3;
          bit += 2;
          n0 += int(r);
          ok = bit <= bits;
        }
        if (!ok || s + n0 > max_sym) { // (a count must follow the zeros)
          ok = false;
          break;
        }
        for (int k = 0; k < n0; ++k)
          S.norm[s++] = 0;
      }
      const int mx = (2 * threshold - 1) - remaining;
      const uint32_t v = peek(bit);
      int count = int(v & uint32_t(threshold - 1));
      if (count < mx) {
        bit += uint32_t(nb - 1);
      } else {
        count = int(v & uint32_t(2 * threshold - 1));
        if (count >= threshold)
          count -= mx;
        bit += uint32_t(nb);
      }
      --count; // -1: a "less than one" probability
      remaining -= count < 0 ? -count : count;
      ok = remaining >= 1 && bit <= bits;
      S.norm[s++] = int16_t(count);
      prev0 = count == 0;
      while (remaining < threshold && nb > 0) {
        --nb;
        threshold >>= 1;
      }
    }
    d = ok && remaining == 1 ? (bit + 7) >> 3 : 0;
  }
  __syncwarp();
  nsym = __shfl_sync(0xffffffffu, s, 0);
  al = __shfl_sync(0xffffffffu, a, 0);
  return __shfl_sync(0xffffffffu, d, 0);
}

// ---- sequences ---------------------------------------------------------------

constexpr int kSeqWarps = CHUCKY_DECODE_WARPS; // (small CTAs spread over the SMs)
// sequences per stage and its words: a sequence takes at most 28 + 32 + 26
// bits (what takes more is left to the sequential decoder)
constexpr int kSeqStep = 16, kSeqStage = 52;
static_assert(kSeqStep * 86 + 64 <= 32 * (kSeqStage - 4), "a stage feeds its sequences");
struct ZSeqTables
{
  uint64_t t[3][512]; // LL, OF, ML
  ZFseWork w;
  ZStage<kSeqStage> stage;
  uint32_t al[3]; // accuracy logs
};

// The predefined tables of those in `want`.
__device__ void zd_predef_tables(unsigned want, ZSeqTables& S)
{
  const int lane = threadIdx.x & 31;
  for (int k = 0; k < 3; ++k) {
    if (!((want >> k) & 1))
      continue;
    const int n = k == 0 ? 36 : k == 1 ? 29 : 53;
    for (int s = lane; s < n; s += 32)
      S.w.norm[s] = k == 0 ? kLLNormD[s] : k == 1 ? kOFNormD[s] : kMLNormD[s];
    __syncwarp();
    const int al = k == 1 ? 5 : 6;
    if (lane == 0)
      S.al[k] = uint32_t(al);
    zd_build_fse(S.t[k], S.w, n, al, k);
    __syncwarp();
  }
}

// The tables that block D describes, of those in `want`, and the place after
// its descriptions (within its content); 0: malformed.
__device__ uint32_t zd_seq_tables(const uint8_t* base,
                                  const ZBlk& D,
                                  unsigned want,
                                  ZSeqTables& S)
{
  const uint8_t* p = base + D.src;
  const bool lane0 = (threadIdx.x & 31) == 0;
  uint32_t at = D.seq_at;
  for (int k = 0; k < 3; ++k) {
    const int mode = int(D.modes >> (6 - 2 * k)) & 3;
    const bool build = (want >> k) & 1;
    if (mode == 1) {
      const uint32_t top = k == 0 ? 35 : k == 1 ? 31 : 52;
      if (at >= D.size || p[at] > top)
        return 0;
      if (build) {
        const uint32_t s = p[at];
        if (lane0) {
          S.t[k][0] = zd_entry(0, 0, s, k);
          S.al[k] = 0;
        }
      }
      at += 1;
    } else if (mode == 2) {
      int nsym, a;
      const uint32_t d = zd_ncount(p + at, D.size - at, k == 1 ? 8 : 9,
                                   k == 0 ? 35 : k == 1 ? 31 : 52, S.w, nsym, a);
      if (!d)
        return 0;
      if (build) {
        if (lane0)
          S.al[k] = uint32_t(a);
        if (!zd_build_fse(S.t[k], S.w, nsym, a, k))
          return 0;
      }
      at += d;
    }
    __syncwarp();
  }
  return at;
}

// One block's sequences (its stream at p, n bytes) by one lane: the list, the
// match bytes (`out`) and the repeat offsets after it; false: malformed.
__device__ __forceinline__ bool zd_sequences(const uint8_t* p,
                             uint32_t n,
                             const uint8_t* lo,
                             const uint8_t* hi,
                             uint32_t nseq,
                             uint32_t nlit,
                             ZSeqTables& S,
                             uint64_t* list,
                             uint32_t& out,
                             uint32_t (&rep)[3])
{
  ZBits bi;
  if (!bi.init(p, n))
    return false;
  bi.stage(S.stage, lo, hi);
  uint32_t sl, so, sm;
  {
    // initial states: LL, OF, ML
    const uint32_t a1 = S.al[1], a2 = S.al[2], v = bi.take(S.al[0] + a1 + a2);
    sm = v & ((1u << a2) - 1);
    so = (v >> a2) & ((1u << a1) - 1);
    sl = v >> (a1 + a2);
  }
  // Errors are collected and looked at once per stage: whatever the bits say,
  // the states stay inside their tables and the list inside its room.
  uint32_t r0 = kSym, r1 = kSym | 1u << 29, r2 = kSym | 2u << 29;
  uint32_t sum_ll = 0, sum_ml = 0, bad = 0;
  for (uint32_t i = 0; i < nseq; ++i) {
    if (i % kSeqStep == 0 && i) {
      if (bad || bi.left() < 0 || sum_ll > nlit || sum_ml >= (1u << 30))
        return false;
      bi.stage(S.stage, lo, hi);
    }
    const uint64_t el = S.t[0][sl], eo = S.t[1][so], em = S.t[2][sm];
    const uint32_t fl = uint32_t(el), fo = uint32_t(eo), fm = uint32_t(em);
    const uint32_t oc = fo >> 16, mb = fm >> 16, lb = fl >> 16;
    const uint32_t xb = oc + mb + lb;
    uint32_t ofv = uint32_t(eo >> 32), ml = uint32_t(em >> 32), ll = uint32_t(el >> 32);
    bi.fill(S.stage);
    if (xb <= 31) { // offset's, match length's, literal length's extra bits
      const uint32_t x = bi.take(xb);
      ofv += x >> (mb + lb);
      ml += (x >> lb) & ((1u << mb) - 1);
      ll += x & ((1u << lb) - 1);
    } else {
      ofv += bi.take(oc);
      bi.fill(S.stage);
      ml += bi.take(mb);
      bi.fill(S.stage);
      ll += bi.take(lb);
    }
    bi.fill(S.stage);
    if (i + 1 < nseq) { // next states: LL, ML, OF
      const uint32_t bl = (fl >> 10) & 63, bm = (fm >> 10) & 63, bo = (fo >> 10) & 63;
      const uint32_t y = bi.take(bl + bm + bo);
      sl = (fl & 1023) + (y >> (bm + bo));
      sm = (fm & 1023) + ((y >> bo) & ((1u << bm) - 1));
      so = (fo & 1023) + (y & ((1u << bo) - 1));
    }
    // repeat codes (RFC 8878 3.1.2.5)
    uint32_t off = ofv - 3;
    if (ofv > 3) {
      r2 = r1;
      r1 = r0;
      bad |= off >> 28; // (longer than the list holds)
    } else {
      const uint32_t idx = ofv - 1 + (ll == 0 ? 1 : 0);
      off = idx == 0 ? r0 : idx == 1 ? r1 : idx == 2 ? r2 : (r0 & kSym) ? r0 + 1 : r0 - 1;
      if (idx > 1)
        r2 = r1;
      if (idx > 0)
        r1 = r0;
      const uint32_t low = off & 0x1FFFFFFFu;
      bad |= uint32_t(off == 0) | ((off & kSym) ? low >> 26 : 0u);
      if (off & kSym)
        off = kSymOff | ((off >> 29) & 3) << 26 | low;
    }
    r0 = (off & kSymOff) ? kSym | ((off >> 26) & 3) << 29 | (off & 0x3FFFFFFu) : off;
    sum_ll += ll;
    sum_ml += ml;
    list[i] = uint64_t(ll | ml << 17) | uint64_t(ml >> 15 | off << 3) << 32;
  }
  out = sum_ml;
  rep[0] = r0;
  rep[1] = r1;
  rep[2] = r2;
  return !bad && bi.left() == 0 && sum_ll <= nlit && sum_ml < (1u << 30);
}

// `per` blocks per warp, a lane each where they share their tables.
__global__ void __launch_bounds__(32 * kSeqWarps, 1) zd_seq_k(ZWave W, uint32_t runs, uint32_t per)
{
  CHUCKY_DYN_SHARED(uint4, sm);
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  ZSeqTables& S = reinterpret_cast<ZSeqTables*>(sm)[threadIdx.x >> 5];
  const uint64_t g = uint64_t(blockIdx.x) * kSeqWarps + (threadIdx.x >> 5);
  // run by run over all frames: the lists are longer than most frames, so
  // the busy warps come first and fill the chip evenly
  const uint64_t f = g % W.n;
  if (g / W.n >= runs)
    return; // the whole warp
  ZFrame& F = W.frames[f];
  const uint32_t nblk = F.nblk, b0 = uint32_t(g / W.n) * per;
  if (F.slow || b0 >= nblk)
    return;
  const uint8_t* const base = W.in + W.in_off[f];
  const uint8_t* const end = base + W.in_size[f];
  ZBlk* const blk = W.blocks + f * W.max_blk;
  const uint32_t b = b0 + uint32_t(lane);
  bool todo = uint32_t(lane) < per && b < nblk && blk[b].type == 2 && blk[b].nseq != 0;
  int def[3] = { kPredef, kPredef, kPredef };
  if (todo)
    for (int k = 0; k < 3; ++k)
      def[k] = blk[b].def[k];
  bool good = true;
  int have[3] = { -1, -1, -1 }; // the tables in S, by defining block
  for (;;) {
    const unsigned m = __ballot_sync(kAll, todo);
    if (!m)
      break;
    const int first = __ffs(int(m)) - 1;
    const int own = __shfl_sync(kAll, int(b), first);
    int want[3];
    unsigned need = 0; // tables to build; a block's own also tell where its stream starts
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      want[k] = __shfl_sync(kAll, def[k], first);
      need |= unsigned(have[k] != want[k] || want[k] == own) << k;
    }
    bool ok = true;
    uint32_t at = 0; // past the first lane's own descriptions
    while (need && ok) { // a definer's tables in one walk
      const int d = (need & 1) ? want[0] : (need & 2) ? want[1] : want[2];
      unsigned set = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k)
        set |= unsigned(((need >> k) & 1) && want[k] == d) << k;
      need &= ~set;
      if (d == kPredef) {
        zd_predef_tables(set, S);
      } else {
        const uint32_t e = zd_seq_tables(base, blk[d], set, S);
        ok = e != 0;
        at = d == own ? e : at;
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
      have[k] = ok ? want[k] : -1;
    __syncwarp();
    if (todo && def[0] == want[0] && def[1] == want[1] && def[2] == want[2]) {
      todo = false;
      const uint32_t size = blk[b].size;
      const uint32_t from = lane == first && at ? at : blk[b].seq_at;
      uint32_t ml = 0, rep[3];
      good = ok && from < size &&
             zd_sequences(base + blk[b].src + from, size - from, base, end, blk[b].nseq,
                          blk[b].nlit, S, W.seqs + f * W.max_seq + blk[b].seq0, ml, rep);
      if (good) {
        blk[b].regen = blk[b].nlit + ml;
        for (int k = 0; k < 3; ++k)
          blk[b].rep[k] = rep[k];
      }
    }
    __syncwarp();
  }
  if (!__all_sync(kAll, good) && lane == 0)
    F.slow = 1;
}

// ---- output offsets and starting repeat offsets ---------------------------------

__global__ void __launch_bounds__(32 * kParseWarps) zd_place_k(ZWave W)
{
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint64_t f = uint64_t(blockIdx.x) * kParseWarps + (threadIdx.x >> 5);
  if (f >= W.n)
    return; // the whole warp
  ZFrame& F = W.frames[f];
  if (F.slow)
    return;
  ZBlk* const blk = W.blocks + f * W.max_blk;
  uint64_t out = 0;
  uint32_t r0 = 1, r1 = 4, r2 = 8;
  for (uint32_t g = 0; g < F.nblk; g += 32) {
    const uint32_t b = g + uint32_t(lane);
    const bool v = b < F.nblk;
    const uint64_t own = v ? blk[b].regen : 0;
    uint64_t x = own;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(kAll, x, o);
      if (lane >= o)
        x += y;
    }
    // Blocks with sequences, in order: a block starts with the repeat
    // offsets that the one before leaves.  Most leave three distances and
    // are done; the others (`sym`) are filled in one after another.
    const bool has = v && blk[b].type == 2 && blk[b].nseq != 0;
    uint32_t a[3] = { 0, 0, 0 };
    if (has)
      for (int k = 0; k < 3; ++k)
        a[k] = blk[b].rep[k];
    const unsigned all = __ballot_sync(kAll, has);
    unsigned sym = __ballot_sync(kAll, has && ((a[0] | a[1] | a[2]) & kSym));
    const unsigned below = (1u << lane) - 1;
    for (; sym; sym &= sym - 1) {
      const int l = __ffs(int(sym)) - 1;
      const unsigned m = all & ((1u << l) - 1);
      const int prev = m ? 31 - __clz(int(m)) : 0;
      const uint32_t p0 = __shfl_sync(kAll, a[0], prev), p1 = __shfl_sync(kAll, a[1], prev),
                     p2 = __shfl_sync(kAll, a[2], prev);
      if (lane == l)
        for (int k = 0; k < 3; ++k)
          a[k] = m ? zd_rep(a[k], p0, p1, p2) : zd_rep(a[k], r0, r1, r2);
    }
    const unsigned mine = all & below;
    const int prev = mine ? 31 - __clz(int(mine)) : 0;
    const uint32_t p0 = __shfl_sync(kAll, a[0], prev), p1 = __shfl_sync(kAll, a[1], prev),
                   p2 = __shfl_sync(kAll, a[2], prev);
    if (v)
      blk[b].out = out + x - own;
    if (has) {
      blk[b].rep[0] = mine ? p0 : r0;
      blk[b].rep[1] = mine ? p1 : r1;
      blk[b].rep[2] = mine ? p2 : r2;
    }
    if (all) {
      const int last = 31 - __clz(int(all));
      r0 = __shfl_sync(kAll, a[0], last);
      r1 = __shfl_sync(kAll, a[1], last);
      r2 = __shfl_sync(kAll, a[2], last);
    }
    out += __shfl_sync(kAll, x, 31);
  }
  if (lane == 0 && (out != W.chunk_bytes || (F.content != ~uint64_t(0) && F.content != out)))
    F.slow = 1;
}

// ---- literals ----------------------------------------------------------------

constexpr int kLitWarps = CHUCKY_DECODE_WARPS;
constexpr uint32_t kLitBlocks = 8; // blocks per warp: four lanes each

// symbols per stage and its words
constexpr uint32_t kLitStep = 64;
constexpr int kLitStage = 28;
static_assert(kLitStep * kDecHufBits + 64 <= 32 * (kLitStage - 4), "a stage feeds its symbols");

struct ZLitTables
{
  uint16_t huf[1 << kDecHufBits]; // symbol | bits << 8
  uint16_t sorted[256];           // symbols by (weight, symbol)
  uint8_t weight[256];
  uint64_t fse[1 << 6];
  ZFseWork w;
  ZStage<kLitStage> stage;
  uint32_t first[kDecHufBits + 2]; // first table entry of a weight
  uint32_t nth[kDecHufBits + 2];   // first place in `sorted` of a weight
};

// Huffman table from the tree description at p (RFC 8878 4.2.1, as
// read_huffman; its size was checked), by a warp; its bits, 0 when malformed.
__device__ int zd_huffman(const uint8_t* p, const uint8_t* lo, const uint8_t* hi, ZLitTables& S)
{
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t hb = p[0];
  int nw = 0;
  if (hb >= 128) {
    nw = int(hb) - 127;
    for (int i = lane; i < nw; i += 32)
      S.weight[i] = (i & 1) ? (p[1 + i / 2] & 15) : (p[1 + i / 2] >> 4);
    __syncwarp();
  } else {
    int nsym, al;
    const uint32_t d = zd_ncount(p + 1, hb, 6, 15, S.w, nsym, al);
    if (!d || d >= hb || !zd_build_fse(S.fse, S.w, nsym, al, 3))
      return 0;
    if (lane == 0) { // two interleaved states
      ZBits bi;
      if (bi.init(p + 1 + d, hb - d)) {
        bi.stage(S.stage, lo, hi);
        uint32_t s = bi.take(uint32_t(al)), other = bi.take(uint32_t(al));
        bool good = bi.left() >= 0;
        while (good) {
          if (nw >= 255) {
            good = false;
            break;
          }
          const uint64_t e = S.fse[s];
          S.weight[nw++] = uint8_t(e >> 32);
          if (nw % 64 == 0) // (64 weights: at most 6 bits each)
            bi.stage(S.stage, lo, hi);
          bi.fill(S.stage);
          s = other; // the states take turns
          other = (uint32_t(e) & 1023) + bi.take((uint32_t(e) >> 10) & 63);
          if (bi.left() < 0) { // the other state gives the last weight
            if (nw >= 255)
              good = false;
            else
              S.weight[nw++] = uint8_t(S.fse[s] >> 32);
            break;
          }
        }
        nw = good ? nw : 0;
      }
    }
    nw = __shfl_sync(kAll, nw, 0);
    __syncwarp();
    if (nw == 0)
      return 0;
  }
  // the last weight completes the sum of 2^(w-1) to a power of two
  uint32_t total = 0;
  bool good = nw <= 255;
  for (int i = lane; i < nw; i += 32) {
    const uint32_t wt = S.weight[i];
    good &= wt <= uint32_t(kDecHufBits);
    if (wt && wt <= uint32_t(kDecHufBits))
      total += 1u << (wt - 1);
  }
  for (int o = 16; o; o >>= 1)
    total += __shfl_xor_sync(kAll, total, o);
  if (!__all_sync(kAll, good) || total == 0)
    return 0;
  const int bits = dec_highbit(total) + 1;
  if (bits > kDecHufBits)
    return 0;
  const uint32_t rest = (1u << bits) - total;
  if (rest & (rest - 1))
    return 0;
  if (lane == 0)
    S.weight[nw] = uint8_t(dec_highbit(rest) + 1);
  ++nw;
  __syncwarp();
  // symbols by (weight, symbol): each symbol's rank among its weight's, 32
  // symbols at a time
  if (lane < kDecHufBits + 2)
    S.nth[lane] = 0;
  __syncwarp();
  uint32_t rank[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    rank[i] = 0;
    if (32 * i >= nw)
      continue;
    const uint32_t wt = 32 * i + lane < nw ? S.weight[32 * i + lane] : 0u;
    const unsigned peers = __match_any_sync(kAll, wt);
    rank[i] = S.nth[wt] + uint32_t(__popc(peers & ((1u << lane) - 1)));
    __syncwarp();
    if (lane == __ffs(int(peers)) - 1)
      S.nth[wt] = rank[i] + uint32_t(__popc(peers));
    __syncwarp();
  }
  // counts -> the first table entry and the first symbol of every weight
  {
    const uint32_t c = lane >= 1 && lane <= kDecHufBits ? S.nth[lane] : 0;
    uint32_t x = c, y = c ? c << (lane - 1) : 0;
    const uint32_t own = y;
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t a = __shfl_up_sync(kAll, x, o), b = __shfl_up_sync(kAll, y, o);
      if (lane >= o) {
        x += a;
        y += b;
      }
    }
    __syncwarp();
    if (lane < kDecHufBits + 2) {
      S.nth[lane] = x - c;
      S.first[lane] = y - own;
    }
    if (__shfl_sync(kAll, y, kDecHufBits) != (1u << bits))
      return 0;
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int s = 32 * i + lane;
    if (s < nw && S.weight[s])
      S.sorted[S.nth[S.weight[s]] + rank[i]] = uint16_t(s);
  }
  __syncwarp();
  for (uint32_t u = uint32_t(lane); u < (1u << bits); u += 32) {
    int wt = 1;
    while (u >= S.first[wt + 1])
      ++wt;
    const uint32_t sym = S.sorted[S.nth[wt] + ((u - S.first[wt]) >> (wt - 1))];
    S.huf[u] = uint16_t(sym | uint32_t(bits + 1 - wt) << 8);
  }
  __syncwarp();
  return bits;
}

// `count` symbols of a Huffman stream to dst; false when the stream is not
// consumed exactly.  Whole aligned words are stored.
__device__ __forceinline__ bool zd_huf_stream(const uint8_t* p, uint32_t n, const uint8_t* lo, const uint8_t* hi,
                              uint8_t* dst, uint32_t count, ZLitTables& S, int bits)
{
  ZBits bi;
  if (!bi.init(p, n))
    return false;
  const int sh = 32 - bits;
  auto sym = [&]() -> uint32_t {
    const uint32_t e = S.huf[bi.hi >> sh];
    bi.drop(e >> 8);
    return e & 255;
  };
  while (count) {
    bi.stage(S.stage, lo, hi);
    uint32_t m = count < kLitStep ? count : kLitStep;
    count -= m;
    for (; m && (reinterpret_cast<uintptr_t>(dst) & 3); --m) {
      bi.fill(S.stage);
      *dst++ = uint8_t(sym());
    }
    for (; m >= 4; m -= 4, dst += 4) {
      bi.fill(S.stage); // 32 bits or more: two symbols of up to 11
      uint32_t v = sym();
      v |= sym() << 8;
      bi.fill(S.stage);
      v |= sym() << 16;
      v |= sym() << 24;
      *reinterpret_cast<uint32_t*>(dst) = v;
    }
    for (; m; --m) {
      bi.fill(S.stage);
      *dst++ = uint8_t(sym());
    }
    if (bi.left() < 0)
      return false;
  }
  return bi.left() == 0;
}

__global__ void __launch_bounds__(32 * kLitWarps, 1) zd_lit_k(ZWave W, uint32_t groups)
{
  CHUCKY_DYN_SHARED(uint4, sm);
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  ZLitTables& S = reinterpret_cast<ZLitTables*>(sm)[threadIdx.x >> 5];
  const uint64_t g = uint64_t(blockIdx.x) * kLitWarps + (threadIdx.x >> 5);
  const uint64_t f = g % W.n; // (in this order as in zd_seq_k)
  if (g / W.n >= groups)
    return; // the whole warp
  ZFrame& F = W.frames[f];
  const uint32_t nblk = F.nblk, b0 = uint32_t(g / W.n) * kLitBlocks;
  if (F.slow || b0 >= nblk)
    return;
  const uint8_t* const base = W.in + W.in_off[f];
  const uint8_t* const end = base + W.in_size[f];
  uint8_t* const out = W.out + f * W.out_stride;
  const ZBlk* const blk = W.blocks + f * W.max_blk;
  // raw and RLE blocks and literals: by the whole warp
  for (uint32_t b = b0; b < b0 + kLitBlocks && b < nblk; ++b) {
    const uint32_t type = blk[b].type, lt = type == 2 ? blk[b].ltype : type;
    if (lt > 1)
      continue;
    const uint32_t n = blk[b].nlit;
    const uint8_t* src = base + blk[b].src + (type == 2 ? blk[b].lit_at : 0);
    uint8_t* dst = out + blk[b].out + (blk[b].regen - n);
    if (lt == 0) {
      copy_exact(dst, src, n, unsigned(lane), 32);
    } else {
      const uint32_t v = src[0] * 0x01010101u;
      uint32_t i = uint32_t(-reinterpret_cast<uintptr_t>(dst)) & 15;
      i = i < n ? i : n;
      if (uint32_t(lane) < i)
        dst[lane] = uint8_t(v);
      for (uint32_t k = i + 16 * uint32_t(lane); k + 16 <= n; k += 512)
        *reinterpret_cast<uint4*>(dst + k) = make_uint4(v, v, v, v);
      const uint32_t tail = i + (n - i) / 16 * 16;
      if (tail + uint32_t(lane) < n)
        dst[tail + lane] = uint8_t(v);
    }
  }
  // Huffman literals: lane 4 k + s decodes stream s of block k
  const uint32_t b = b0 + uint32_t(lane >> 2), s = uint32_t(lane & 3);
  const bool has = b < nblk && blk[b].type == 2 && blk[b].ltype >= 2;
  const uint8_t* sp = nullptr;
  uint8_t* dst = nullptr;
  uint32_t sn = 0, count = 0;
  int huf = -1;
  bool good = true, mine = false;
  if (has) {
    const uint8_t* q = base + blk[b].src + blk[b].lit_at;
    const uint32_t qn = blk[b].lit_len, n = blk[b].nlit;
    huf = blk[b].huf;
    dst = out + blk[b].out + (blk[b].regen - n);
    if (blk[b].streams == 1) {
      mine = s == 0;
      sp = q;
      sn = qn;
      count = n;
    } else {
      mine = true;
      const uint32_t seg = (n + 3) / 4;
      good = qn >= 6 && seg * 3 <= n;
      if (good) {
        uint32_t l[3], at = 6;
        for (int k = 0; k < 3; ++k)
          l[k] = q[2 * k] | (uint32_t(q[2 * k + 1]) << 8);
        good = 6 + l[0] + l[1] + l[2] <= qn;
        for (uint32_t k = 0; k < s; ++k)
          at += l[k];
        sp = q + at;
        sn = s < 3 ? l[s] : qn - at;
        dst += s * seg;
        count = s < 3 ? seg : n - 3 * seg;
      }
    }
  }
  // tables one after another, every lane that uses one at the same time
  bool todo = mine && good;
  int built = -1, bits = 0;
  for (;;) {
    const unsigned m = __ballot_sync(kAll, todo);
    if (!m)
      break;
    const int d = __shfl_sync(kAll, huf, __ffs(int(m)) - 1);
    if (d != built) {
      const ZBlk& D = blk[d];
      bits = zd_huffman(base + D.src + D.tree_at, base, end, S);
      built = d;
    }
    if (todo && huf == d) {
      good = bits > 0 && zd_huf_stream(sp, sn, base, end, dst, count, S, bits);
      todo = false;
    }
    __syncwarp();
  }
  if (!__all_sync(kAll, good) && lane == 0)
    F.slow = 1;
}

// ---- execution ---------------------------------------------------------------

struct ZTok // as tile_run wants it, in one load
{
  uint32_t bound, off;
  int32_t dlit;
  uint32_t unused;
};

constexpr uint32_t kExecPer = 4; // sequences per thread and tile

// A block with sequences.
struct ZWork
{
  uint64_t out;
  uint32_t seq0, nseq, lits, rep[3]; // lits: where its literals are in its output
};

template<int NT>
struct ZExec
{
  static constexpr uint32_t kList = NT < 128 ? NT : 128;
  ZWork work[kList];
  uint16_t slot[kList];
  LzTile<NT> tile;
  alignas(16) ZTok tok[NT * kExecPer + 1];
  uint64_t warp_sum[32];
  uint32_t warp_sum32[32];
  uint32_t cut, cut_out, cut_ll;
  uint32_t bad;
};

template<int NT>
__global__ void __launch_bounds__(NT) zd_exec_k(ZWave W)
{
  CHUCKY_DYN_SHARED(uint4, sm);
  ZExec<NT>& S = *reinterpret_cast<ZExec<NT>*>(sm);
  constexpr uint32_t kExecList = ZExec<NT>::kList;
  const uint32_t tid = threadIdx.x;
  const uint64_t f = blockIdx.x;
  ZFrame& F = W.frames[f];
  if (F.slow)
    return; // the whole CTA
  const uint32_t nblk = F.nblk;
  const ZBlk* const blk = W.blocks + f * W.max_blk;
  uint8_t* const out = W.out + f * W.out_stride;
  if (tid == 0)
    S.bad = 0;
  uint64_t ahead[kExecPer]; // a block's first sequences, loaded during the one before
  auto fetch = [&](const ZWork& K) {
#pragma unroll
    for (uint32_t u = 0; u < kExecPer; ++u)
      ahead[u] = tid * kExecPer + u < K.nseq
                   ? W.seqs[f * W.max_seq + K.seq0 + tid * kExecPer + u]
                   : 0;
  };
  for (uint32_t bl = 0, i = 0, nwork = 0;; ++i) {
    if (i == nwork) { // the next blocks with sequences, in order
      if (bl >= nblk)
        break;
      __syncthreads();
      if (tid < kExecList) {
        const uint32_t b = bl + tid;
        const bool has = b < nblk && blk[b].type == 2 && blk[b].nseq != 0;
        const unsigned m = __ballot_sync(0xffffffffu, has);
        if ((tid & 31) == 0)
          S.warp_sum32[tid >> 5] = uint32_t(__popc(m));
        S.slot[tid] = has ? uint16_t(__popc(m & ((1u << (tid & 31)) - 1))) : 0xFFFFu;
      }
      __syncthreads();
      nwork = 0;
      for (uint32_t k = 0; k < kExecList / 32; ++k)
        nwork += S.warp_sum32[k];
      if (tid < kExecList && S.slot[tid] != 0xFFFFu) {
        const ZBlk& B = blk[bl + tid];
        uint32_t at = S.slot[tid];
        for (uint32_t k = 0; k < (tid >> 5); ++k)
          at += S.warp_sum32[k];
        S.work[at] = ZWork{ B.out, B.seq0, B.nseq, B.regen - B.nlit,
                            { B.rep[0], B.rep[1], B.rep[2] } };
      }
      __syncthreads();
      bl += kExecList;
      i = 0;
      if (nwork == 0) {
        i = ~0u; // (0 after the increment)
        continue;
      }
      fetch(S.work[0]);
    }
    const ZWork K = S.work[i];
    const uint32_t nseq = K.nseq;
    const uint64_t* const seq = W.seqs + f * W.max_seq + K.seq0;
    const uint32_t r0 = K.rep[0], r1 = K.rep[1], r2 = K.rep[2];
    uint8_t* const bo = out + K.out;
    const uint64_t before = K.out;
    uint32_t op = 0, lp = K.lits; // next output, next literal
    for (uint32_t s0 = 0; s0 < nseq;) {
      const uint32_t left = nseq - s0;
      const uint32_t take = left < NT * kExecPer ? left : NT * kExecPer;
      uint32_t ll[kExecPer], ml[kExecPer], of[kExecPer];
      uint64_t sum = 0; // output bytes, literals << 32
      uint64_t qs[kExecPer];
#pragma unroll
      for (uint32_t u = 0; u < kExecPer; ++u)
        qs[u] = s0 == 0 ? ahead[u] : (tid * kExecPer + u < take ? seq[s0 + tid * kExecPer + u] : 0);
      if (s0 == 0 && i + 1 < nwork) // the next block's first sequences
        fetch(S.work[i + 1]);
#pragma unroll
      for (uint32_t u = 0; u < kExecPer; ++u) {
        const uint32_t e = tid * kExecPer + u;
        ll[u] = ml[u] = of[u] = 0;
        if (e < take) {
          const uint64_t q = qs[u];
          ll[u] = uint32_t(q) & 0x1FFFF;
          ml[u] = uint32_t(q >> 17) & 0x3FFFF;
          const uint32_t o = uint32_t(q >> 35);
          of[u] = (o & kSymOff)
                    ? zd_rep(kSym | ((o >> 26) & 3) << 29 | (o & 0x3FFFFFFu), r0, r1, r2)
                    : o;
          sum += uint64_t(ll[u] + ml[u]) | uint64_t(ll[u]) << 32;
        }
      }
      tile_clear(S.tile);
      if (tid == 0)
        S.cut = ~0u;
      uint64_t total;
      const uint64_t ex = cta_scan<NT>(sum, S.warp_sum, total);
      const uint32_t shd = uint32_t(reinterpret_cast<uintptr_t>(bo + op) & 15);
      uint32_t o = uint32_t(ex), l = uint32_t(ex >> 32);
#pragma unroll
      for (uint32_t u = 0; u < kExecPer; ++u) {
        const uint32_t i = tid * kExecPer + u, len = ll[u] + ml[u];
        if (i >= take)
          continue;
        if (o + len <= LzTile<NT>::kBytes) {
          S.tok[i + 1] = ZTok{ shd + o + ll[u], of[u], int32_t(lp + l) - int32_t(op + o), 0 };
          tile_mark(S.tile, shd, o);
        } else if (o <= LzTile<NT>::kBytes) { // the first past the tile
          S.cut = i;
          S.cut_out = o;
          S.cut_ll = l;
        }
        // (offsets of all of them: they are the block's sequences)
        if (of[u] == 0 || of[u] > before + op + o + ll[u])
          S.bad = 1;
        o += len;
        l += ll[u];
      }
      __syncthreads();
      if (S.bad) { // the whole CTA
        if (tid == 0)
          F.slow = 1;
        return;
      }
      const bool cut = S.cut != ~0u;
      const uint32_t n = cut ? S.cut : take;
      const uint32_t nout = cut ? S.cut_out : uint32_t(total);
      const uint32_t nll = cut ? S.cut_ll : uint32_t(total >> 32);
      if (n == 0) { // one sequence longer than a tile
        const uint64_t q = seq[s0];
        const uint32_t gl = uint32_t(q) & 0x1FFFF, gm = uint32_t(q >> 17) & 0x3FFFF;
        const uint32_t o29 = uint32_t(q >> 35);
        const uint32_t off =
          (o29 & kSymOff)
            ? zd_rep(kSym | ((o29 >> 26) & 3) << 29 | (o29 & 0x3FFFFFFu), r0, r1, r2)
            : o29;
        // its literals move down (never past themselves): a piece is read
        // before any of it is written
        for (uint32_t c = 0; c < gl && lp != op; c += NT * 16) {
          uint8_t v[16];
#pragma unroll
          for (uint32_t u = 0; u < 16; ++u)
            if (c + u * NT + tid < gl)
              v[u] = bo[lp + c + u * NT + tid];
          __syncthreads();
#pragma unroll
          for (uint32_t u = 0; u < 16; ++u)
            if (c + u * NT + tid < gl)
              bo[op + c + u * NT + tid] = v[u];
          __syncthreads();
        }
        __syncthreads();
        cta_match<NT>(bo + op + gl, off, gm);
        op += gl + gm;
        lp += gl;
        s0 += 1;
      } else {
        // (literals lie in the output: their places are relative to the tile)
        tile_run<NT, 9>(S.tile, S.warp_sum32, S.tok, bo + op - shd, bo + op, nout);
        op += nout;
        lp += nll;
        s0 += n;
      }
      __syncthreads();
    }
  }
  if (tid == 0)
    W.status[f] = kZOk;
}

cudaError_t zd_launch(const ZWave& W, cudaStream_t st)
{
  const unsigned wf = unsigned((W.n + kParseWarps - 1) / kParseWarps);
  note_launches(5);
  CHUCKY_LAUNCH(zd_parse_k, wf, 32 * kParseWarps, 0, st, W);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return e;
  // Blocks per warp: one lane each when they share their tables, so more of
  // them cost no more instructions; but a sequence takes 250 cycles on its
  // lane, so a few warps per scheduler are wanted first (12 per SM).  Blocks of
  // 8 KiB are assumed, as this library's encoder makes them: stock frames of
  // 128 KiB blocks are sixteen times fewer, and share no tables either.
  const uint64_t share = W.n * ((W.chunk_bytes >> 13) + 1) / (uint64_t(device_sm_count()) * 12);
  uint32_t per = 1;
  while (per < 32 && per <= share)
    per *= 2;
  const uint32_t runs = (W.max_blk + per - 1) / per;
  constexpr size_t seq_smem = sizeof(ZSeqTables) * kSeqWarps;
  constexpr size_t lit_smem = sizeof(ZLitTables) * kLitWarps;
  if ((e = cudaFuncSetAttribute(zd_seq_k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                int(seq_smem))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(zd_lit_k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                int(lit_smem))) != cudaSuccess)
    return e;
  CHUCKY_LAUNCH(zd_seq_k, unsigned((W.n * runs + kSeqWarps - 1) / kSeqWarps), 32 * kSeqWarps,
                seq_smem, st, W, runs, per);
  if ((e = cudaGetLastError()) != cudaSuccess)
    return e;
  CHUCKY_LAUNCH(zd_place_k, wf, 32 * kParseWarps, 0, st, W);
  if ((e = cudaGetLastError()) != cudaSuccess)
    return e;
  const uint32_t groups = (W.max_blk + kLitBlocks - 1) / kLitBlocks;
  CHUCKY_LAUNCH(zd_lit_k, unsigned((W.n * groups + kLitWarps - 1) / kLitWarps), 32 * kLitWarps,
                lit_smem, st, W, groups);
  if ((e = cudaGetLastError()) != cudaSuccess)
    return e;
  if (W.chunk_bytes <= (16u << 10)) {
    constexpr int NT = CHUCKY_DECODE_THREADS;
    constexpr size_t smem = sizeof(ZExec<NT>);
    if ((e = cudaFuncSetAttribute(zd_exec_k<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(smem))) != cudaSuccess)
      return e;
    CHUCKY_LAUNCH(zd_exec_k<NT>, unsigned(W.n), NT, smem, st, W);
  } else {
    constexpr int NT = CHUCKY_ZSTD_EXEC_THREADS;
    constexpr size_t smem = sizeof(ZExec<NT>);
    if ((e = cudaFuncSetAttribute(zd_exec_k<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(smem))) != cudaSuccess)
      return e;
    CHUCKY_LAUNCH(zd_exec_k<NT>, unsigned(W.n), NT, smem, st, W);
  }
  return cudaGetLastError();
}

} // namespace

} // namespace chucky
