// Size table, overlap-add kernel and launch dispatch of the FFT3D filtering
// core; the FFT kernels themselves are instantiated in kern_*.cu.
#include <algorithm>
#include <mutex>
#include <vector>

#include "fft3d_kernels.cuh"
#include "fft3d_kernels_impl.cuh"
#include "kern_registry.h"

#include <set>
#include <tuple>

namespace fft3d {

cudaError_t set_smem_attr(const void* func, int bytes, bool prefer_shared) {
  static std::mutex mu;
  static std::set<std::tuple<const void*, int, int>> done;
  int dev = 0;
  cudaGetDevice(&dev);
  const auto key = std::make_tuple(func, dev, bytes);
  std::lock_guard<std::mutex> lk(mu);
  if (done.count(key)) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && prefer_shared)
    e = cudaFuncSetAttribute(func, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) done.insert(key);
  return e;
}

namespace {

std::vector<SizeEntry>& table() {
  static std::vector<SizeEntry> t;
  return t;
}

constexpr int kOlaTx = 32, kOlaTy = 8;
constexpr int kOla4BatchRows = 4 * kOlaTy;  // rows of one batched 4-pixel overlap-add item

// V adjacent pixels (V = 1, 2 or 4) of R rows per thread, frame blockIdx.z of
// fs (one frame per call, or a frame group's frames in one launch). V > 1
// where the V pixels share their blocks and overlap case and their samples go
// out in one store (overlap_add_width); the block column, its overlap case and
// the synthesis windows along x are found once for the R rows (ola_pixels).
// The planes whose block step is not a multiple of 4 (the filter's default
// overlap of 10 with 32 x 32 blocks) had one launch per frame and one pixel per
// thread: 344 us for 16 frames of 720p 16-bit 4:2:0, against 112 us here.
template <typename T, int V, int R>
__global__ void __launch_bounds__(kOlaTx * kOlaTy) k_overlap_add_rows(OlaArgs a, const __grid_constant__ OlaFrameSet fs) {
  const int x0 = V * (blockIdx.x * kOlaTx + threadIdx.x), j = blockIdx.z;
  if (x0 >= a.g.W) return;
  const OlaColumn<V> c(a, x0);
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int k = (blockIdx.y * R + r) * kOlaTy + threadIdx.y;
    if (k < a.g.H) ola_pixels<T, V, false>(a, c, fs.tdom[j], fs.dst[j], fs.dst_stride[j], x0, k);
  }
}

// Pixels per thread of the overlap-add: as many as share their blocks and
// overlap case everywhere in the plane and are aligned in every frame.
int overlap_add_width(const OlaArgs& a, const OlaFrameSet& fs, int bytes) {
  for (int v = 4; v > 1; v /= 2) {
    bool ok = a.g.sx % v == 0 && a.g.ow % v == 0 && a.g.W % v == 0 && a.g.bw % v == 0;
    for (int j = 0; j < fs.count && ok; j++)
      ok = reinterpret_cast<uintptr_t>(fs.tdom[j]) % (4 * v) == 0 &&
           reinterpret_cast<uintptr_t>(fs.dst[j]) % (v * bytes) == 0 && fs.dst_stride[j] % (v * bytes) == 0;
    if (ok) return v;
  }
  return 1;
}

template <typename T, int V>
void overlap_add_rows(const OlaArgs& a, const OlaFrameSet& fs, cudaStream_t s) {
  const dim3 block(kOlaTx, kOlaTy);
  const int gx = (a.g.W / V + kOlaTx - 1) / kOlaTx + (a.g.W % V != 0), gy = (a.g.H + kOlaTy - 1) / kOlaTy;
  // 4 rows a thread while that still leaves four CTAs for each SM
  if ((long long)gx * ((gy + 3) / 4) * fs.count >= 4 * 148)
    k_overlap_add_rows<T, V, 4><<<dim3(gx, (gy + 3) / 4, fs.count), block, 0, s>>>(a, fs);
  else
    k_overlap_add_rows<T, V, 1><<<dim3(gx, gy, fs.count), block, 0, s>>>(a, fs);
}

template <typename T>
void overlap_add_typed(const OlaArgs& a, const OlaFrameSet& fs, cudaStream_t s) {
  const int v = overlap_add_width(a, fs, (int)sizeof(T));
  if (v == 4) overlap_add_rows<T, 4>(a, fs, s);
  else if (v == 2) overlap_add_rows<T, 2>(a, fs, s);
  else overlap_add_rows<T, 1>(a, fs, s);
}

// Batched overlap-add: work item = (plane, 32x8 tile in row-major tile order).
template <typename T>
__global__ void __launch_bounds__(kOlaTx * kOlaTy) k_overlap_add_batch(const OlaArgs* __restrict__ args,
                                                                      const int2* __restrict__ items, int nitems) {
  for (int i = blockIdx.x; i < nitems; i += gridDim.x) {
    const int2 it = items[i];
    const OlaArgs a = args[it.x];  // private copy: fields stay in registers
    const int tx = (a.g.W + kOlaTx - 1) / kOlaTx;
    const int ty = it.y / tx, t = it.y - ty * tx;
    const int x0 = t * kOlaTx + threadIdx.x, k = ty * kOlaTy + threadIdx.y;
    if (x0 < a.g.W && k < a.g.H) ola_pixels<T, 1, false>(a, OlaColumn<1>(a, x0), a.tdom, a.dst, a.dst_stride, x0, k);
  }
}

// Batched 4-pixel overlap-add: work item = (plane, 128x8-pixel tile); every
// plane of the launch meets the 4-pixel kernel's geometry and alignment rules
// (batch_overlap_add4_ok).
template <typename T>
__global__ void __launch_bounds__(kOlaTx * kOlaTy) k_overlap_add4_batch(const OlaArgs* __restrict__ args,
                                                                       const int2* __restrict__ items, int nitems) {
  for (int i = blockIdx.x; i < nitems; i += gridDim.x) {
    const int2 it = items[i];
    const OlaArgs a = args[it.x];  // private copy: fields stay in registers
    const int tx = (a.g.W + 4 * kOlaTx - 1) / (4 * kOlaTx);
    const int ty = it.y / tx, t = it.y - ty * tx;
    // kOla4BatchRows rows per item, so that the argument loads and the column
    // are shared by several pixel quads per thread
    const int x0 = 4 * (t * kOlaTx + threadIdx.x);
    if (x0 >= a.g.W) continue;
    const OlaColumn<4> c(a, x0);
#pragma unroll
    for (int r = 0; r < kOla4BatchRows; r += kOlaTy) {
      const int k = ty * kOla4BatchRows + r + threadIdx.y;
      if (k < a.g.H) ola_pixels<T, 4, false>(a, c, a.tdom, a.dst, a.dst_stride, x0, k);
    }
  }
}

}  // namespace

bool register_size(const SizeEntry& e) {
  table().push_back(e);
  return true;
}

const SizeEntry* find_size(int bw, int bh) {
  for (const auto& e : table())
    if (e.bw == bw && e.bh == bh) return &e;
  return nullptr;
}

int registered_sizes(SizeEntry* out, int max) {
  int n = 0;
  for (const auto& e : table())
    if (n < max) out[n++] = e;
  return (int)table().size();
}

bool block_size_supported(int bw, int bh) { return find_size(bw, bh) != nullptr; }

cudaError_t upload_twiddles() {
  for (const auto& e : table()) {
    cudaError_t err = e.upload();
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

cudaError_t launch_forward(const ForwardArgs& a, int bytes, cudaStream_t s) {
  const SizeEntry* e = find_size(a.g.bw, a.g.bh);
  return e ? e->fwd(a, bytes, s) : cudaErrorInvalidValue;
}

cudaError_t launch_filter_inverse(const InverseArgs& a, int mode, cudaStream_t s) {
  const SizeEntry* e = find_size(a.g.bw, a.g.bh);
  return e ? e->inv(a, mode, s) : cudaErrorInvalidValue;
}

cudaError_t launch_forward_frames(const ForwardArgs& a, const FwdFrameSet& fs, int bytes, cudaStream_t s) {
  const SizeEntry* e = find_size(a.g.bw, a.g.bh);
  return e ? e->fwd_frames(a, fs, bytes, s) : cudaErrorInvalidValue;
}

cudaError_t launch_filter_inverse_frames(const InverseArgs& a, const FrameSet& fs, int mode, cudaStream_t s) {
  const SizeEntry* e = find_size(a.g.bw, a.g.bh);
  return e ? e->inv_frames(a, fs, mode, s) : cudaErrorInvalidValue;
}

cudaError_t launch_filter_bins(const InverseArgs& a, float2* F, int mode, cudaStream_t s) {
  const int bins = a.g.bh * a.g.nh;
  const size_t pairs = (size_t)a.g.nblocks * bins / 2;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = (int)std::min<size_t>((pairs + 255) / 256, (size_t)sms * 8);
  switch (mode) {
    case MODE_KALMAN: k_filter_bins<MODE_KALMAN><<<grid, 256, 0, s>>>(a, F, bins); break;
    case 1: k_filter_bins<1><<<grid, 256, 0, s>>>(a, F, bins); break;
    case 2: k_filter_bins<2><<<grid, 256, 0, s>>>(a, F, bins); break;
    case 3: k_filter_bins<3><<<grid, 256, 0, s>>>(a, F, bins); break;
    case 4: k_filter_bins<4><<<grid, 256, 0, s>>>(a, F, bins); break;
    case 5: k_filter_bins<5><<<grid, 256, 0, s>>>(a, F, bins); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_filter_inverse_group(const InverseArgs& a, const TemporalSet& ts, int mode, cudaStream_t s,
                                        const OlaFuse* of) {
  const SizeEntry* e = find_size(a.g.bw, a.g.bh);
  return e ? e->inv_group(a, ts, mode, s, of) : cudaErrorInvalidValue;
}

cudaError_t launch_filter_frames(const InverseArgs& a, const FilterFrameSet& fs, int mode, cudaStream_t s) {
  if (fs.count < 1 || fs.count > kMaxGroupFrames) return cudaErrorInvalidValue;
  const int bins = a.g.bh * a.g.nh;
  const size_t pairs = (size_t)a.g.nblocks * bins / 2;
  const int grid = (int)((pairs + 255) / 256);
  switch (mode) {
    case MODE_KALMAN: k_filter_frames<MODE_KALMAN><<<grid, 256, 0, s>>>(a, fs, bins); break;
    case 1: k_filter_frames<1><<<grid, 256, 0, s>>>(a, fs, bins); break;
    case 2: k_filter_frames<2><<<grid, 256, 0, s>>>(a, fs, bins); break;
    case 3: k_filter_frames<3><<<grid, 256, 0, s>>>(a, fs, bins); break;
    case 4: k_filter_frames<4><<<grid, 256, 0, s>>>(a, fs, bins); break;
    case 5: k_filter_frames<5><<<grid, 256, 0, s>>>(a, fs, bins); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_frame(const FrameArgs& a, int mode, int bytes, cudaStream_t s) {
  const SizeEntry* e = find_size(a.v.g.bw, a.v.g.bh);
  return e ? e->frame(a, mode, bytes, s) : cudaErrorInvalidValue;
}

cudaError_t launch_forward_batch(int bw, int bh, const BatchLaunch& l, int bytes, cudaStream_t s) {
  const SizeEntry* e = find_size(bw, bh);
  return e ? e->fwd_batch(l, bytes, s) : cudaErrorInvalidValue;
}

cudaError_t launch_filter_inverse_batch(int bw, int bh, const BatchLaunch& l, int mode, cudaStream_t s) {
  const SizeEntry* e = find_size(bw, bh);
  return e ? e->inv_batch(l, mode, s) : cudaErrorInvalidValue;
}

cudaError_t launch_filter_inverse_group_batch(int bw, int bh, const BatchLaunch& l, int mode, cudaStream_t s) {
  const SizeEntry* e = find_size(bw, bh);
  return e ? e->inv_group_batch(l, mode, s) : cudaErrorInvalidValue;
}

cudaError_t launch_overlap_add_batch(const BatchLaunch& l, int bytes, cudaStream_t s) {
  dim3 block(kOlaTx, kOlaTy);
  const auto* args = static_cast<const OlaArgs*>(l.args);
  if (bytes >= kOla4Var) {  // the 4-pixel form
    bytes -= kOla4Var;
    if (bytes == 1) k_overlap_add4_batch<uint8_t><<<l.grid, block, 0, s>>>(args, l.items, l.nitems);
    else if (bytes == 2) k_overlap_add4_batch<uint16_t><<<l.grid, block, 0, s>>>(args, l.items, l.nitems);
    else k_overlap_add4_batch<float><<<l.grid, block, 0, s>>>(args, l.items, l.nitems);
    return cudaGetLastError();
  }
  if (bytes == 1) k_overlap_add_batch<uint8_t><<<l.grid, block, 0, s>>>(args, l.items, l.nitems);
  else if (bytes == 2) k_overlap_add_batch<uint16_t><<<l.grid, block, 0, s>>>(args, l.items, l.nitems);
  else k_overlap_add_batch<float><<<l.grid, block, 0, s>>>(args, l.items, l.nitems);
  return cudaGetLastError();
}

// Batched plane copies: work item = (copy, row); 16-byte moves when both
// rows are 16-byte aligned, bytes otherwise.
__global__ void __launch_bounds__(256) k_copy_batch(const CopyArgs* __restrict__ args, const int2* __restrict__ items,
                                                    int nitems) {
  for (int i = blockIdx.x; i < nitems; i += gridDim.x) {
    const int2 it = items[i];
    const CopyArgs c = args[it.x];
    const char* s = static_cast<const char*>(c.src) + (long long)it.y * c.spitch;
    char* d = static_cast<char*>(c.dst) + (long long)it.y * c.dpitch;
    if ((((uintptr_t)s | (uintptr_t)d) & 15) == 0) {
      const long long n16 = c.width / 16;
      for (long long x = threadIdx.x; x < n16; x += blockDim.x)
        reinterpret_cast<uint4*>(d)[x] = reinterpret_cast<const uint4*>(s)[x];
      for (long long x = n16 * 16 + threadIdx.x; x < c.width; x += blockDim.x) d[x] = s[x];
    } else {
      for (long long x = threadIdx.x; x < c.width; x += blockDim.x) d[x] = s[x];
    }
  }
}

cudaError_t launch_copy_batch(const BatchLaunch& l, cudaStream_t s) {
  k_copy_batch<<<l.grid, 256, 0, s>>>(static_cast<const CopyArgs*>(l.args), l.items, l.nitems);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(128) k_pattern_scores(const float2* __restrict__ spec,
                                                        const float2* __restrict__ grid,
                                                        const float* __restrict__ pwin, int nox, int noy,
                                                        int bins, float degrid, float* scores) {
  const int wx = nox - 4, wy = noy - 4;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= wx * wy) return;
  const int by = 2 + i / wx, bx = 2 + i % wx;
  const float2* s = spec + ((size_t)by * nox + bx) * bins;
  const float gcur = __fdiv_rn(__fmul_rn(degrid, s[0].x), grid[0].x);
  float acc = 0.f;
  for (int k = 0; k < bins; k++) {
    const float2 v = s[k], gs = grid[k];
    const float c0 = __fsub_rn(v.x, __fmul_rn(gcur, gs.x)), c1 = __fsub_rn(v.y, __fmul_rn(gcur, gs.y));
    acc = __fadd_rn(acc, __fmul_rn(__fadd_rn(__fmul_rn(c0, c0), __fmul_rn(c1, c1)), pwin[k]));
  }
  scores[i] = acc;
}

cudaError_t launch_pattern_scores(const float2* spec, const float2* grid, const float* pwin, int nox, int noy,
                                  int bins, float degrid, float* scores, cudaStream_t s) {
  const int n = (nox - 4) * (noy - 4);
  if (n <= 0) return cudaSuccess;
  k_pattern_scores<<<(n + 127) / 128, 128, 0, s>>>(spec, grid, pwin, nox, noy, bins, degrid, scores);
  return cudaGetLastError();
}

int batch_items_forward(const Geom& g) {
  const SizeEntry* e = find_size(g.bw, g.bh);
  return e ? e->ctas(g.nblocks) : 0;
}

int batch_items_overlap_add(const Geom& g) {
  return ((g.W + kOlaTx - 1) / kOlaTx) * ((g.H + kOlaTy - 1) / kOlaTy);
}

int batch_items_overlap_add4(const Geom& g) {
  return ((g.W + 4 * kOlaTx - 1) / (4 * kOlaTx)) * ((g.H + kOla4BatchRows - 1) / kOla4BatchRows);
}

bool batch_overlap_add4_ok(const OlaArgs& a, int bytes) {
  return a.g.sx % 4 == 0 && a.g.ow % 4 == 0 && a.g.W % 4 == 0 && a.g.bw % 4 == 0 &&
         reinterpret_cast<uintptr_t>(a.tdom) % 16 == 0 && reinterpret_cast<uintptr_t>(a.dst) % (4 * bytes) == 0 &&
         a.dst_stride % (4 * bytes) == 0;
}

int batch_occupancy(int bw, int bh, int which, int mode_or_bytes) {
  if (which == 4) return 8;  // plane copies
  if (which == 2) {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_overlap_add_batch<uint8_t>, kOlaTx * kOlaTy, 0);
    return n > 0 ? n : 1;
  }
  const SizeEntry* e = find_size(bw, bh);
  return e ? e->occupancy(which, mode_or_bytes) : 1;
}

int overlap_add_pixels(const OlaArgs& a, const OlaFrameSet& fs, int bytes) { return overlap_add_width(a, fs, bytes); }

__global__ void k_fill(float* p, float v, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

cudaError_t launch_fill(float* p, float v, size_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int grid = (int)std::min<size_t>((n + 255) / 256, 4096);
  k_fill<<<grid, 256, 0, s>>>(p, v, n);
  return cudaGetLastError();
}

cudaError_t launch_overlap_add_frames(const OlaArgs& a, const OlaFrameSet& fs, int bytes, cudaStream_t s) {
  if (fs.count < 1 || fs.count > kMaxGroupFrames) return cudaErrorInvalidValue;
  if (bytes == 1) overlap_add_typed<uint8_t>(a, fs, s);
  else if (bytes == 2) overlap_add_typed<uint16_t>(a, fs, s);
  else overlap_add_typed<float>(a, fs, s);
  return cudaGetLastError();
}

cudaError_t launch_overlap_add(const OlaArgs& a, int bytes, cudaStream_t s) {
  OlaFrameSet fs{};
  fs.tdom[0] = a.tdom;
  fs.dst[0] = a.dst;
  fs.dst_stride[0] = a.dst_stride;
  fs.count = 1;
  return launch_overlap_add_frames(a, fs, bytes, s);
}

// The bytes of bs.count planes outside an interior rectangle (the crop borders,
// which the overlap-add does not write), from their source planes: one launch
// for a call's frames. Rows are cut into slots of U bytes, U the alignment that
// all the frames' rows share; the slots of the rows above and below the
// interior and those that hold the ends of the rows beside it are numbered
// through, so that a thread has one slot, or four at a time of a large border,
// however the border is shaped. A slot that is border in part goes in aligned
// pieces of less than U bytes.
// Bound by the latency of its loads. One-frame calls, us per frame with a copy
// of the whole plane (cudaMemcpy2DAsync) / a warp per row, words or bytes / now:
// 1080p 16-bit, a quarter of the width and an eighth of the height off each
// side, 45.2 / 57.9 / 38.5; 4K 10-bit, 8 rows off top and bottom, 218 / 204 / 172;
// 1080p 8-bit, 6 to 10 pixels off all sides, 108 / 70 / 63.
template <int N>
struct Bytes;
template <>
struct Bytes<16> { using V = uint4; };
template <>
struct Bytes<8> { using V = uint2; };
template <>
struct Bytes<4> { using V = uint32_t; };
template <>
struct Bytes<2> { using V = uint16_t; };
template <>
struct Bytes<1> { using V = uint8_t; };

// A slot's next piece: N bytes of the row from x on if they lie before hi and,
// on the way up to a multiple of U, x has this bit set (on the way down N
// halves from piece to piece, so that x stays a multiple of it).
template <int U, int N, bool UP>
struct BorderPiece {
  typename Bytes<N>::V v;
  int at = -1;
  __device__ __forceinline__ BorderPiece(const char* row, int& x, int hi) {
    if (N >= U || x + N > hi || (UP && (x & N) == 0)) return;
    at = x;
    x += N;
    v = *reinterpret_cast<const typename Bytes<N>::V*>(row + at);
  }
  __device__ __forceinline__ void put(char* row) const {
    if (at >= 0) *reinterpret_cast<typename Bytes<N>::V*>(row + at) = v;
  }
};

// (small CTAs: the 2160 slots of a narrow border of 1080p go to 34 SMs)
constexpr int kBorderThreads = 64;

template <int U>
__global__ void __launch_bounds__(kBorderThreads) k_copy_borders(const __grid_constant__ BorderSet bs) {
  using V = typename Bytes<U>::V;
  const int f = blockIdx.y;
  const char* src = static_cast<const char*>(bs.src[f]);
  char* dst = static_cast<char*>(bs.dst[f]);
  const unsigned whole = (bs.width + U - 1) / U, left = (bs.x0 + U - 1) / U, right0 = bs.x1 / U;
  const unsigned ends = left + (bs.x1 < bs.width ? whole - right0 : 0);
  const unsigned rows = bs.y0 + bs.height - bs.y1, n = rows * whole + (bs.y1 - bs.y0) * ends;
  // slot i: its row, and its bytes [lo, hi) of the row
  auto slot = [&](unsigned i, int* y, int* lo, int* hi) {
    unsigned s, r;
    int b0 = 0, b1 = bs.width;
    if (i < rows * whole) {
      r = i / whole;
      s = i - r * whole;
      *y = (int)r < bs.y0 ? r : r - bs.y0 + bs.y1;
    } else {
      i -= rows * whole;
      r = i / ends;
      s = i - r * ends;
      *y = bs.y0 + r;
      if (s < left) {
        b1 = bs.x0;
      } else {
        s += right0 - left;
        b0 = bs.x1;
      }
    }
    *lo = max((int)(s * U), b0);
    *hi = min((int)(s * U) + U, b1);
  };
  const unsigned step = gridDim.x * kBorderThreads;
  for (unsigned i = blockIdx.x * kBorderThreads + threadIdx.x; i < n; i += 4 * step) {
    V v[4];
    V* to[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const unsigned k = i + u * step;
      to[u] = nullptr;
      if (k >= n) continue;
      int y, lo, hi;
      slot(k, &y, &lo, &hi);
      const char* p = src + y * bs.spitch[f];
      char* q = dst + y * bs.dpitch[f];
      if (hi - lo == U) {
        v[u] = *reinterpret_cast<const V*>(p + lo);
        to[u] = reinterpret_cast<V*>(q + lo);
      } else {
        int x = lo;
        const BorderPiece<U, 1, true> u1(p, x, hi);
        const BorderPiece<U, 2, true> u2(p, x, hi);
        const BorderPiece<U, 4, true> u4(p, x, hi);
        const BorderPiece<U, 8, true> u8(p, x, hi);
        const BorderPiece<U, 8, false> d8(p, x, hi);
        const BorderPiece<U, 4, false> d4(p, x, hi);
        const BorderPiece<U, 2, false> d2(p, x, hi);
        const BorderPiece<U, 1, false> d1(p, x, hi);
        u1.put(q), u2.put(q), u4.put(q), u8.put(q), d8.put(q), d4.put(q), d2.put(q), d1.put(q);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (to[u]) *to[u] = v[u];
  }
}

template <int U>
void copy_borders(const BorderSet& bs, cudaStream_t s) {
  const long long whole = (bs.width + U - 1) / U, ends = (bs.x0 + U - 1) / U + whole - bs.x1 / U;
  const long long slots = whole * (bs.y0 + bs.height - bs.y1) + ends * (bs.y1 - bs.y0);
  const long long most = std::max(1, 32 * 148 / bs.count);  // all SMs' threads, for all frames
  const int ctas = (int)std::min(most, (slots + kBorderThreads - 1) / kBorderThreads);
  k_copy_borders<U><<<dim3(std::max(1, ctas), bs.count), kBorderThreads, 0, s>>>(bs);
}

cudaError_t launch_copy_borders(const BorderSet& bs, cudaStream_t s) {
  if (bs.count < 1 || bs.count > kMaxGroupFrames) return cudaErrorInvalidValue;
  if (bs.width < 1 || bs.height < 1) return cudaSuccess;
  uintptr_t bits = 16;
  for (int j = 0; j < bs.count; j++)
    bits |= reinterpret_cast<uintptr_t>(bs.src[j]) | reinterpret_cast<uintptr_t>(bs.dst[j]) |
            (uintptr_t)bs.spitch[j] | (uintptr_t)bs.dpitch[j];
  switch (bits & (~bits + 1)) {  // the lowest bit: the alignment that all rows share, at most 16
    case 16: copy_borders<16>(bs, s); break;
    case 8: copy_borders<8>(bs, s); break;
    case 4: copy_borders<4>(bs, s); break;
    case 2: copy_borders<2>(bs, s); break;
    default: copy_borders<1>(bs, s); break;
  }
  return cudaGetLastError();
}

}  // namespace fft3d
