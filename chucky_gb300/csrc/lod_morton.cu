// (b) LOD pyramid, general path: Morton-ordered level buffers.
//
// Works for any number of LOD dims and levels.  Per epoch:
//   gather  : values[b*n0 + m] = linear[fixed[b] + lut[m]]
//             (src/cpu/lod.cpp:241-267, src/gpu/lod.cu:224-304)
//   reduce  : parent i of level l+1 = reduce(child window
//             [ends[i-1], ends[i]) of level l), sequential in window order
//             (src/cpu/lod.cpp:55-127, 269-296; src/gpu/lod.cu:414-528)
//   fold    : dim-0 accumulators of levels >= 1
//             (src/cpu/lod.cpp:366-414; src/gpu/lod.cu:904-941)
//   emit    : accumulators -> level values (src/cpu/lod.cpp:416-438)
//   scatter : level values -> chunk slot via per-level LUTs
//             (src/cpu/lod.cpp:298-359, src/gpu/lod.cu:347-364)
// Arithmetic per dtype matches the reference bit for bit: widened sums for
// mean (u8/u16 -> u32, u32 -> u64, i8/i16 -> i32, i32 -> i64, f16 -> f32),
// insertion-sort median (upper median), second-extreme with >= / <= ties.
#include "kernels.hpp"
#include "lod_ops.cuh"

namespace chucky {

namespace lod {

constexpr int kThreads = 256;

template<typename T>
__global__ void __launch_bounds__(kThreads)
gather_k(const T* __restrict__ linear,
         T* __restrict__ values,
         const uint32_t* __restrict__ lut,
         const uint64_t* __restrict__ fixed,
         FastDiv n0,
         uint64_t total)
{
  for (uint64_t g = blockIdx.x * uint64_t(kThreads) + threadIdx.x; g < total;
       g += uint64_t(gridDim.x) * kThreads) {
    uint64_t b, m;
    n0.divmod(g, b, m);
    values[g] = linear[fixed[b] + lut[m]];
  }
}

// One level from the one below: element g of all slices.
struct ReduceLevel
{
  const uint64_t* ends;
  uint64_t src_beg, dst_beg;
  uint64_t src_n, dst_n;
  FastDiv div; // by dst_n
  uint64_t total;
};

template<typename T>
__device__ __forceinline__ void reduce_one(T* values, const ReduceLevel& L, uint64_t g, int method)
{
  uint64_t b, i;
  L.div.divmod(g, b, i);
  const uint64_t lo = i ? L.ends[i - 1] : 0, hi = L.ends[i];
  const T* src = values + L.src_beg + b * L.src_n + lo;
  T v;
  if (hi - lo == 8) { // a whole window of three dims stays in registers
    T w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      w[k] = src[k];
    v = reduce_full<T, 8>(w, method);
  } else {
    v = reduce_window<T>(src, hi - lo, method);
  }
  values[L.dst_beg + g] = v;
}

template<typename T>
__global__ void __launch_bounds__(kThreads) reduce_k(T* values, ReduceLevel L, int method)
{
  for (uint64_t g = blockIdx.x * uint64_t(kThreads) + threadIdx.x; g < L.total;
       g += uint64_t(gridDim.x) * kThreads)
    reduce_one(values, L, g, method);
}

// The pyramid's top, levels of at most kTailElems elements, in one CTA: a
// launch each cost 4 to 6 us for work of a few hundred windows.  All levels of
// the i16 volume of 16 x 200 x 328 reduced, by kTailElems: 22.2 us with 0 (a
// launch each), 20.2 with 1024, 19.9 with 4096, 20.3 with 16384, 33.6 with 65536;
// of 32 x 400 x 656: 39.7, 33.5, 33.8, 33.8, 52.3.
constexpr uint64_t kTailElems = 4096;
constexpr int kTailThreads = 1024, kTailLevels = 16;
struct ReduceTail
{
  int n;
  ReduceLevel lv[kTailLevels];
};
template<typename T>
__global__ void __launch_bounds__(kTailThreads) reduce_tail_k(T* values, ReduceTail t, int method)
{
  for (int l = 0; l < t.n; ++l) {
    for (uint64_t g = threadIdx.x; g < t.lv[l].total; g += kTailThreads)
      reduce_one(values, t.lv[l], g, method);
    __syncthreads();
  }
}

template<typename T>
__global__ void __launch_bounds__(kThreads)
fold_k(T* __restrict__ accum,
       const T* __restrict__ x,
       uint64_t n,
       uint32_t count,
       int level,
       int method)
{
  for (uint64_t g = blockIdx.x * uint64_t(kThreads) + threadIdx.x; g < n;
       g += uint64_t(gridDim.x) * kThreads)
    accum[g] = count == 0 ? x[g] : fold_one<T>(accum[g], x[g], level, method);
}

template<typename T>
__global__ void __launch_bounds__(kThreads)
emit_k(T* __restrict__ dst,
       const T* __restrict__ accum,
       uint64_t n,
       uint32_t count,
       int method)
{
  for (uint64_t g = blockIdx.x * uint64_t(kThreads) + threadIdx.x; g < n;
       g += uint64_t(gridDim.x) * kThreads)
    dst[g] = emit_one<T>(accum[g], count, method);
}

// The active levels' values to their chunks, one launch for all of them (six
// of 2 to 6 us before).
struct ChunkLevel
{
  uint64_t first;  // of the launch's elements
  uint64_t beg;    // of the level's values
  FastDiv n;       // values per slice
  const uint32_t* lut;
  const uint64_t* fixed;
};
struct ChunkLevels
{
  int n;
  uint64_t total;
  ChunkLevel lv[32];
};
template<typename T>
__global__ void __launch_bounds__(kThreads)
to_chunks_k(const T* __restrict__ values, T* __restrict__ slot, ChunkLevels c)
{
  for (uint64_t e = blockIdx.x * uint64_t(kThreads) + threadIdx.x; e < c.total;
       e += uint64_t(gridDim.x) * kThreads) {
    int l = 0; // (levels shrink fast: most elements stop at the first)
    while (l + 1 < c.n && e >= c.lv[l + 1].first)
      ++l;
    const ChunkLevel& L = c.lv[l];
    const uint64_t g = e - L.first;
    uint64_t b, i;
    L.n.divmod(g, b, i);
    slot[L.fixed[b] + L.lut[i]] = values[L.beg + g];
  }
}

inline int grid_for(uint64_t work)
{
  const uint64_t blocks = (work + kThreads - 1) / kThreads;
  const uint64_t cap = uint64_t(device_sm_count()) * 16;
  return int(blocks < cap ? (blocks ? blocks : 1) : cap);
}

} // namespace lod

using namespace lod;

cudaError_t launch_lod_gather(const LodMortonArgs& a,
                              const uint8_t* linear,
                              uint8_t* values,
                              cudaStream_t st)
{
  const uint64_t n0 = a.lod_nelem[0], total = a.fixed_count * n0;
  CHUCKY_DISPATCH_DTYPE(a.dtype,
                        (gather_k<T><<<grid_for(total), kThreads, 0, st>>>(
                          reinterpret_cast<const T*>(linear),
                          reinterpret_cast<T*>(values),
                          a.d_gather_lut,
                          a.d_gather_fixed,
                          FastDiv(n0),
                          total)));
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_lod_reduce(const LodMortonArgs& a,
                              uint8_t* values,
                              cudaStream_t st)
{
  auto level = [&](int l) { // level l from level l - 1
    ReduceLevel L{};
    L.ends = a.d_ends + a.ends_beg[l];
    L.src_beg = a.level_beg[l - 1];
    L.dst_beg = a.level_beg[l];
    L.src_n = a.lod_nelem[l - 1];
    L.dst_n = a.lod_nelem[l];
    L.div = FastDiv(L.dst_n);
    L.total = a.fixed_count * L.dst_n;
    return L;
  };
  int l = 1;
  for (; l < a.nlod; ++l) {
    const ReduceLevel L = level(l);
    if (L.total <= kTailElems && a.nlod - l <= kTailLevels)
      break;
    CHUCKY_DISPATCH_DTYPE(a.dtype, (reduce_k<T><<<grid_for(L.total), kThreads, 0, st>>>(
                                     reinterpret_cast<T*>(values), L, a.reduce_method)));
    note_launches(1);
  }
  if (l < a.nlod) { // (higher levels are smaller still)
    ReduceTail t{};
    for (; l < a.nlod; ++l)
      t.lv[t.n++] = level(l);
    CHUCKY_DISPATCH_DTYPE(a.dtype, (reduce_tail_k<T><<<1, kTailThreads, 0, st>>>(
                                     reinterpret_cast<T*>(values), t, a.reduce_method)));
    note_launches(1);
  }
  return cudaGetLastError();
}

cudaError_t launch_lod_fold(const LodMortonArgs& a,
                            int level,
                            uint32_t count,
                            const uint8_t* values,
                            uint8_t* accum,
                            cudaStream_t st)
{
  const uint64_t n = a.fixed_count * a.lod_nelem[level];
  CHUCKY_DISPATCH_DTYPE(
    a.dtype,
    (fold_k<T><<<grid_for(n), kThreads, 0, st>>>(
      reinterpret_cast<T*>(accum) + a.accum_beg[level],
      reinterpret_cast<const T*>(values) + a.level_beg[level],
      n,
      count,
      level,
      a.append_method)));
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_lod_emit(const LodMortonArgs& a,
                            int level,
                            uint32_t count,
                            const uint8_t* accum,
                            uint8_t* values,
                            cudaStream_t st)
{
  const uint64_t n = a.fixed_count * a.lod_nelem[level];
  CHUCKY_DISPATCH_DTYPE(
    a.dtype,
    (emit_k<T><<<grid_for(n), kThreads, 0, st>>>(
      reinterpret_cast<T*>(values) + a.level_beg[level],
      reinterpret_cast<const T*>(accum) + a.accum_beg[level],
      n,
      count,
      a.append_method)));
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_lod_to_chunks(const LodMortonArgs& a,
                                 uint32_t levels,
                                 const uint8_t* values,
                                 uint8_t* slot,
                                 cudaStream_t st)
{
  ChunkLevels c{};
  for (int l = 0; l < a.nlod; ++l)
    if (levels >> l & 1) {
      ChunkLevel& L = c.lv[c.n++];
      L.first = c.total;
      L.beg = a.level_beg[l];
      L.n = FastDiv(a.lod_nelem[l]);
      L.lut = a.d_chunk_lut[l];
      L.fixed = a.d_chunk_fixed[l];
      c.total += a.fixed_count * a.lod_nelem[l];
    }
  if (!c.n)
    return cudaSuccess;
  CHUCKY_DISPATCH_DTYPE(a.dtype, (to_chunks_k<T><<<grid_for(c.total), kThreads, 0, st>>>(
                                   reinterpret_cast<const T*>(values),
                                   reinterpret_cast<T*>(slot), c)));
  note_launches(1);
  return cudaGetLastError();
}

} // namespace chucky
