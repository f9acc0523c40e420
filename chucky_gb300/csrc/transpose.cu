// (a) Scatter a row-major epoch into chunk-contiguous tiles.
//
// Element e of an epoch goes to ravel(e) over the lifted shape
// (c0, k0, c1, k1, ...) with the lifted strides of the level layout, exactly
// as src/gpu/transpose.cu:85-137 and src/cpu/transpose.cpp:10-105 of the
// reference.  The innermost lifted pair (count, chunk) spans one input row
// of `width` elements, so dst(e) = row_off[e / width] + col_off[e % width]:
// the two small tables replace the per-element unravel.  (Where that pair
// is narrow -- few channels innermost -- a row takes in the pairs above it.)
// When the chunk
// extent of the innermost dim is a multiple of 16 bytes and that dim is
// innermost in storage, every 16-byte input vector lands in one contiguous,
// aligned run of its chunk row: one 16-byte load and one 16-byte store per
// thread, fully coalesced on both sides.
#include "kernels.hpp"

namespace chucky {

namespace {

constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads)
transpose_vec16_k(TransposeArgs a, uint64_t nvec)
{
  const uint32_t per = 16u / a.bpe;
  for (uint64_t v = blockIdx.x * uint64_t(kThreads) + threadIdx.x; v < nvec;
       v += uint64_t(gridDim.x) * kThreads) {
    const uint64_t e = v * per;
    uint64_t row, x;
    a.width.divmod(e, row, x);
    const uint64_t o = __ldg(a.row_off + row) + __ldg(a.col_off + x);
    const uint4 val = __ldg(reinterpret_cast<const uint4*>(a.src) + v);
    *reinterpret_cast<uint4*>(a.dst + o * a.bpe) = val;
  }
}

// Interleaved channels (2 to 4 innermost elements, chunks planar): a thread
// takes 16 bytes' worth of pixels, one 16-byte load per channel, sorts them by
// channel in registers and stores 16 bytes to each channel's chunk row.  The
// host takes this path only where every such run is contiguous and aligned,
// so there is no remainder.  Bound by the latency of its loads at this size
// (34-37 % of the DRAM rate): 31.5 MB of RGB bytes into 256 x 256 chunks take 11
// us, element by element 57.
template<int kBpe, int C>
__device__ __forceinline__ uint32_t channel_word(const uint32_t (&w)[4 * C], int c, int j)
{
  if constexpr (kBpe == 1) {
    const int i0 = 4 * j * C + c, i1 = i0 + C, i2 = i1 + C, i3 = i2 + C;
    const uint32_t lo = __byte_perm(w[i0 / 4], w[i1 / 4], (i0 & 3) | (4 + (i1 & 3)) << 4);
    const uint32_t hi = __byte_perm(w[i2 / 4], w[i3 / 4], (i2 & 3) | (4 + (i3 & 3)) << 4);
    return __byte_perm(lo, hi, 0x5410);
  } else if constexpr (kBpe == 2) {
    const int i0 = 2 * j * C + c, i1 = i0 + C;
    return __byte_perm(w[i0 / 2], w[i1 / 2], (i0 & 1 ? 0x32 : 0x10) | (i1 & 1 ? 0x7600 : 0x5400));
  } else if constexpr (kBpe == 4) {
    return w[j * C + c];
  } else {
    return w[2 * ((j / 2) * C + c) + (j & 1)];
  }
}

template<int kBpe, int C>
__global__ void __launch_bounds__(kThreads)
transpose_planar_k(TransposeArgs a, uint64_t ngroups)
{
  constexpr uint32_t kGroup = 16 / kBpe * C; // elements per thread and step
  for (uint64_t g = blockIdx.x * uint64_t(kThreads) + threadIdx.x; g < ngroups;
       g += uint64_t(gridDim.x) * kThreads) {
    uint64_t row, x;
    a.width.divmod(g * kGroup, row, x);
    const uint4* src = reinterpret_cast<const uint4*>(a.src) + g * C;
    uint32_t w[4 * C];
#pragma unroll
    for (int k = 0; k < C; ++k) {
      const uint4 v = __ldg(src + k);
      w[4 * k] = v.x;
      w[4 * k + 1] = v.y;
      w[4 * k + 2] = v.z;
      w[4 * k + 3] = v.w;
    }
    const uint64_t o = __ldg(a.row_off + row) + __ldg(a.col_off + x);
#pragma unroll
    for (int c = 0; c < C; ++c)
      *reinterpret_cast<uint4*>(a.dst + (o + a.channel_off[c]) * kBpe) =
        make_uint4(channel_word<kBpe, C>(w, c, 0), channel_word<kBpe, C>(w, c, 1),
                   channel_word<kBpe, C>(w, c, 2), channel_word<kBpe, C>(w, c, 3));
  }
}

// Elements one by one, where vectors do not stay whole: kRun consecutive ones
// per thread (TransposeArgs::run), four read with one or two vector loads and
// one division.  Bound by its stores, an element each: neighbouring threads
// store side by side with one element each, four apart with four, which only
// pays where the elements go to different chunk rows anyway.  us for 540 x 959
// pixels x 4 frames, 1 and 4 per thread, u8 / u32, chunks of one channel and
// 100 columns: 2 channels 14 and 12 / 9 and 10, 3: 20 and 22 / 12 and 11, 4: 24
// and 18 / 16 and 15, 6: 39 and 33 / 44 and 36, 8: 57 and 36 / 59 and 39; 7
// columns, 2 channels: 16 and 23 / 15 and 18.  Rows of u8 cut every 100
// columns, 1080 x 2000 x 4 frames: 22 and 20; every 20: 22 and 29; every 5: 25
// and 59.  u16 every 100: 22 and 24.
template<typename T, uint32_t kRun>
__global__ void __launch_bounds__(kThreads)
transpose_scalar_k(TransposeArgs a, uint64_t first)
{
  struct alignas(sizeof(T) * kRun < 16 ? sizeof(T) * kRun : 16) Run
  {
    T v[kRun];
  };
  const T* src = reinterpret_cast<const T*>(a.src);
  T* dst = reinterpret_cast<T*>(a.dst);
  // (`first` keeps the 16-byte alignment of the epoch buffer, which is padded)
  for (uint64_t e = first + kRun * (blockIdx.x * uint64_t(kThreads) + threadIdx.x); e < a.n;
       e += kRun * uint64_t(gridDim.x) * kThreads) {
    const Run run = *reinterpret_cast<const Run*>(src + e);
    uint64_t row, x;
    a.width.divmod(e, row, x);
    uint64_t o = __ldg(a.row_off + row);
#pragma unroll
    for (uint32_t u = 0; u < kRun; ++u) {
      if (e + u >= a.n)
        break;
      dst[o + __ldg(a.col_off + x)] = run.v[u];
      if (++x == a.width.d && e + u + 1 < a.n) {
        x = 0;
        o = __ldg(a.row_off + ++row);
      }
    }
  }
}

int grid_for(uint64_t work)
{
  // persistent-style grid: a multiple of the SM count, capped by the work
  const uint64_t blocks = (work + kThreads - 1) / kThreads;
  const uint64_t cap = uint64_t(device_sm_count()) * 8;
  return int(blocks < cap ? (blocks ? blocks : 1) : cap);
}

template<typename T>
cudaError_t launch_scalar(const TransposeArgs& a, uint64_t first, cudaStream_t st)
{
  const int g = grid_for((a.n - first + a.run - 1) / a.run);
  if (a.run == 4)
    transpose_scalar_k<T, 4><<<g, kThreads, 0, st>>>(a, first);
  else
    transpose_scalar_k<T, 1><<<g, kThreads, 0, st>>>(a, first);
  note_launches(1);
  return cudaGetLastError();
}

template<int kBpe>
cudaError_t launch_planar(const TransposeArgs& a, cudaStream_t st)
{
  const uint64_t n = a.n / (16 / kBpe * a.channels);
  const int g = grid_for(n);
  switch (a.channels) {
    case 2:
      transpose_planar_k<kBpe, 2><<<g, kThreads, 0, st>>>(a, n);
      break;
    case 3:
      transpose_planar_k<kBpe, 3><<<g, kThreads, 0, st>>>(a, n);
      break;
    default:
      transpose_planar_k<kBpe, 4><<<g, kThreads, 0, st>>>(a, n);
      break;
  }
  note_launches(1);
  return cudaGetLastError();
}

} // namespace

cudaError_t launch_transpose(const TransposeArgs& a, cudaStream_t st)
{
  if (a.n == 0)
    return cudaSuccess;
  if (a.channels)
    switch (a.bpe) {
      case 1:
        return launch_planar<1>(a, st);
      case 2:
        return launch_planar<2>(a, st);
      case 4:
        return launch_planar<4>(a, st);
      case 8:
        return launch_planar<8>(a, st);
      default:
        return cudaErrorInvalidValue;
    }
  uint64_t first = 0;
  if (a.vector_ok) {
    const uint64_t per = 16u / a.bpe;
    const uint64_t nvec = a.n / per;
    if (nvec) {
      transpose_vec16_k<<<grid_for(nvec), kThreads, 0, st>>>(a, nvec);
      note_launches(1);
      first = nvec * per;
    }
  }
  if (first < a.n) {
    switch (a.bpe) {
      case 1:
        return launch_scalar<uint8_t>(a, first, st);
      case 2:
        return launch_scalar<uint16_t>(a, first, st);
      case 4:
        return launch_scalar<uint32_t>(a, first, st);
      case 8:
        return launch_scalar<uint64_t>(a, first, st);
      default:
        return cudaErrorInvalidValue;
    }
  }
  return cudaGetLastError();
}

} // namespace chucky
