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

// Elements one by one, where vectors do not stay whole: kRun consecutive ones
// per thread, read with one or two vector loads and one division.  Bound by
// its stores (an element each): RGB frames into planar u8 chunks (12.4 MB
// epochs) took 67 us with a division and two table look-ups per byte, a table
// entry per three bytes among them.
constexpr uint32_t kRun = 4;
template<typename T>
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

} // namespace

cudaError_t launch_transpose(const TransposeArgs& a, cudaStream_t st)
{
  if (a.n == 0)
    return cudaSuccess;
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
    const int g = grid_for((a.n - first + kRun - 1) / kRun);
    note_launches(1);
    switch (a.bpe) {
      case 1:
        transpose_scalar_k<uint8_t><<<g, kThreads, 0, st>>>(a, first);
        break;
      case 2:
        transpose_scalar_k<uint16_t><<<g, kThreads, 0, st>>>(a, first);
        break;
      case 4:
        transpose_scalar_k<uint32_t><<<g, kThreads, 0, st>>>(a, first);
        break;
      case 8:
        transpose_scalar_k<uint64_t><<<g, kThreads, 0, st>>>(a, first);
        break;
      default:
        return cudaErrorInvalidValue;
    }
  }
  return cudaGetLastError();
}

} // namespace chucky
