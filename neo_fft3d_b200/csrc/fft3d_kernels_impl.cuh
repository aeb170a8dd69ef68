// Kernel templates of the FFT3D filtering core (FP32 CUDA-core path).
// Included by the per-size translation units kern_*.cu, which instantiate the
// block sizes they own and register them in the size table (kern_registry.h).
#pragma once
#include <algorithm>
#include <cmath>

#include "fft3d_kernels.cuh"
#include "kern_registry.h"
#include "regfft.cuh"
#include "fft3d_attr.h"

namespace fft3d {
namespace {

constexpr int kWarps = 4;       // warps per CTA of the forward and filter/inverse kernels

// CTAs per SM that the filter/inverse kernels are compiled for, where their
// shared memory lets that many reside: walks of a Wiener 3D run (whose tiles
// allow 4 at 32 x 32 and bt = 5), and the others at 96 registers (at 6 CTAs and
// 80 registers they spill 52 bytes: 1080p bt=5 with its spatial edge frames
// 1820 us per 24 frames, 1763 at 5).
constexpr int kWalkCtas = 6, kShortCtas = 5;
// shared memory per SM, and what the runtime reserves per resident CTA
constexpr int kSmemPerSm = 228 * 1024, kSmemPerCtaReserved = 1024;
__host__ __device__ constexpr int ctas_for(int want, int smem_per_cta) {
  const int fit = kSmemPerSm / (smem_per_cta + kSmemPerCtaReserved);
  return fit < 1 ? 1 : (fit < want ? fit : want);
}

// reflect-101 of index s into [0, n): the cover's mirror margins
// (src/buffer.cpp:19-26, 65-79); repeated for planes narrower than a margin.
__device__ __forceinline__ int reflect101(int s, int n) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    if (s < 0) s = -s;
    if (s >= n) s = 2 * (n - 1) - s;
  }
  return s;
}

// processed-plane row k -> source row: progressive, or interlaced with field 1
// (even rows) first and field 2 bottom-up (src/buffer.cpp:31-63, 99-115)
__device__ __forceinline__ int field_row(int k, int H, int interlaced) {
  if (!interlaced) return k;
  int half = H >> 1;
  return k < half ? 2 * k : H - 1 - 2 * (k - half);
}

// The hardware's approximate reciprocal and reciprocal square root (PTX
// rcp.approx / rsqrt.approx, the instructions __fdividef and rsqrtf stand on).
// Every caller's argument is a normal float (a power spectrum plus 1e-15,
// a noise power of at least 1e-15, a ratio clamped to >= 1e-30), where the
// .ftz forms give the same result without the handling of denormal
// arguments that the plain forms carry.
__device__ __forceinline__ float rcp_nrm(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_nrm(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// n / d for 0 <= n < 2^24, d > 0 and a quotient below 2^20 (pixel and block
// coordinates over a block step or a row length), exact: the estimate
// n * (1/d) is within (n / d) * 2^-21 < 0.5 of n / d (reciprocal <= 2 ulp,
// one rounding), so truncating it and correcting by one step either way gives
// the integer quotient, in a few instructions instead of an integer division
// by a runtime value.
__device__ __forceinline__ int div_small(int n, int d) {
  int q = __float2int_rz(__int2float_rn(n) * rcp_nrm(__int2float_rn(d)));
  const int r = n - q * d;
  q += (r >= d) - (r < 0);
  return q;
}

template <typename T>
__device__ __forceinline__ float load_sample(const T* p) { return (float)p[0]; }
template <>
__device__ __forceinline__ float load_sample<uint8_t>(const uint8_t* p) { return (float)(int)__ldg(p); }
template <>
__device__ __forceinline__ float load_sample<uint16_t>(const uint16_t* p) { return (float)(int)__ldg(p); }
template <>
__device__ __forceinline__ float load_sample<float>(const float* p) { return __ldg(p); }

// Blocks per warp of the FFT kernels: enough that the bw/2 column transforms
// of all of them (DC and Nyquist columns share one complex transform) fill
// the 32 lanes (2 for bw = 32, 4 for bw = 16, 1 for bw = 48).
template <int BW>
__host__ __device__ constexpr int blocks_per_warp() {
  return (32 / (BW / 2)) < 1 ? 1 : ((32 / (BW / 2)) > 4 ? 4 : 32 / (BW / 2));
}

template <int BW, int BH>
__host__ __device__ constexpr int fft_smem_bytes() {
  return blocks_per_warp<BW>() * BH * (BW / 2 + 1) * 8;
}

// The BW samples at p as 32-bit words: 16-byte loads where p allows, else
// 4-byte loads of the words that hold them (never past the word of the last
// sample) and funnel shifts.
template <typename T, int BW>
__device__ __forceinline__ void load_words(const T* p, uint32_t (&w)[BW * sizeof(T) / 4]) {
  constexpr int WORDS = BW * (int)sizeof(T) / 4;
  static_assert(BW * sizeof(T) % 4 == 0, "whole words");
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  if (WORDS % 4 == 0 && (at & 15) == 0) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int v = 0; v < WORDS / 4; v++) {
      const uint4 u = __ldg(q + v);
      w[4 * v] = u.x, w[4 * v + 1] = u.y, w[4 * v + 2] = u.z, w[4 * v + 3] = u.w;
    }
    return;
  }
  const uint32_t* q = reinterpret_cast<const uint32_t*>(at & ~(uintptr_t)3);
#pragma unroll
  for (int v = 0; v < WORDS; v++) w[v] = __ldg(q + v);
  if constexpr (sizeof(T) < 4) {
    const int shift = 8 * (int)(at & 3);
    if (shift) {
      const uint32_t last = __ldg(q + WORDS);
#pragma unroll
      for (int v = 0; v < WORDS; v++) w[v] = __funnelshift_r(w[v], v + 1 < WORDS ? w[v + 1] : last, shift);
    }
  }
}

// Sample x of a row's words as a float of 2^23 + sample (8/16-bit samples: one
// byte permute into the low mantissa bits of 2^23, exact), or the sample itself.
template <typename T, int WORDS>
__device__ __forceinline__ float raw_sample(const uint32_t (&w)[WORDS], int x) {
  if constexpr (sizeof(T) == 1) return __uint_as_float(__byte_perm(w[x >> 2], 0x4B000000u, 0x7540u | (uint32_t)(x & 3)));
  else if constexpr (sizeof(T) == 2) return __uint_as_float(__byte_perm(w[x >> 1], 0x4B000000u, (x & 1) ? 0x7432u : 0x7410u));
  else return __uint_as_float(w[x]);
}

// ---------------------------------------------------------------- block FFT phases
// Sb points at one block's bh x (bw/2+1) complex tile in shared memory.

// Where a forward CTA reads its frame and writes its spectra: the launch
// arguments (one frame per launch), or pointers picked for one frame of a
// frame group (k_forward_frames).
struct ArgsFwd {
  const ForwardArgs& a;
  __device__ __forceinline__ const void* src() const { return a.src; }
  __device__ __forceinline__ long long stride() const { return a.src_stride; }
  __device__ __forceinline__ float2* spec() const { return a.spec; }
};
struct FrameFwd {
  const void* s;
  long long st;
  float2* sp;
  __device__ __forceinline__ const void* src() const { return s; }
  __device__ __forceinline__ long long stride() const { return st; }
  __device__ __forceinline__ float2* spec() const { return sp; }
};

// Source row of row y of block `blk` and the source column of its column 0;
// *row: the source row index (checked against the plane in the checked build).
template <typename T, class Win>
__device__ __forceinline__ const T* fwd_row_src(const ForwardArgs& a, const Win& win, int blk, int y, int* x0,
                                                int* row = nullptr) {
  const Geom& g = a.g;
  const int by = div_small(blk, g.nox), bx = blk - by * g.nox;
  const int k = reflect101(by * g.sy + y - g.sy, g.H);
  *x0 = bx * g.sx - g.sx;
  const int r = field_row(k, g.H, g.interlaced);
  if (row) *row = r;
  return reinterpret_cast<const T*>(static_cast<const char*>(win.src()) + (long long)r * win.stride());
}

// Row y of block `blk`: gather (mirrored at the plane edges), analysis window,
// r2c along x into row y of Sb. PARAM: the window along x comes as halves from
// the launch parameters, else from memory (a power of two leaves the products
// the same).
template <int BW, int BH, typename T, bool PARAM, class Win>
__device__ __forceinline__ void fwd_row(const ForwardArgs& a, const Win& win, int blk, int y, float2* Sb) {
  constexpr int NH = BW / 2 + 1;
  const Geom& g = a.g;
  int x0, srcrow;
  const T* srow = fwd_row_src<T>(a, win, blk, y, &x0, &srcrow);
  float r[BW];
  const bool row_ok = FFT3D_IN(srcrow >= 0 && srcrow < g.H, a.err);
  const float off = (sizeof(T) < 4 ? 8388608.0f : 0.f) + a.base;  // raw_sample's offset and the plane's: exact
  if (row_ok && x0 >= 0 && x0 + BW <= g.W) {
    uint32_t w[BW * sizeof(T) / 4];
    load_words<T, BW>(srow + x0, w);
#pragma unroll
    for (int x = 0; x < BW; x++) r[x] = raw_sample<T>(w, x) - off;
  } else {
#pragma unroll
    for (int x = 0; x < BW; x++) {
      const int xi = reflect101(x0 + x, g.W);
      r[x] = (row_ok && FFT3D_IN(xi >= 0 && xi < g.W, a.err)) ? load_sample<T>(srow + xi) - a.base : 0.f;
    }
  }
  const float wy = __ldg(a.wan_y + y) * (PARAM ? 2.f : 1.f);
#pragma unroll
  for (int x = 0; x < BW; x++) r[x] = r[x] * (PARAM ? a.wx_half[x].x : __ldg(a.wan_x + x)) * wy;
  float2 c[NH];
  rfft<BW>(r, c);
  float2* row = Sb + y * NH;
#pragma unroll
  for (int kk = 0; kk < NH; kk++) row[kk] = c[kk];
}

// Column c (0 < c < bw/2) forward DFT along y in place; c == 0 transforms the
// real columns 0 and bw/2 together as one complex sequence col0 + i colN.
// The lanes of a warp differ only in what they load and store: the FFT itself
// is one code path for all of them (no divergent second pass).
template <int BW, int BH>
__device__ __forceinline__ void fwd_col(float2* Sb, int c) {
  constexpr int NH = BW / 2 + 1, HC = BW / 2;
  float2 col[BH];
  const bool dc = c == 0;
#pragma unroll
  for (int y = 0; y < BH; y++) {
    const float2 v = Sb[y * NH + c];
    col[y] = dc ? make_float2(v.x, Sb[y * NH + HC].x) : v;
  }
  cfft<BH, -1>(col);
  if (dc) {
#pragma unroll
    for (int h = 0; h < BH; h++) {
      const float2 zh = col[h], zm = cconj(col[(BH - h) % BH]);
      Sb[h * NH] = make_float2(0.5f * (zh.x + zm.x), 0.5f * (zh.y + zm.y));
      const float2 d = csub(zh, zm);
      Sb[h * NH + HC] = make_float2(0.5f * d.y, -0.5f * d.x);
    }
  } else {
#pragma unroll
    for (int h = 0; h < BH; h++) Sb[h * NH + c] = col[h];
  }
}

// Column c inverse DFT along y in place; c == 0 handles columns 0 and bw/2
// together (both Hermitian, so both inverses are real).
template <int BW, int BH>
__device__ __forceinline__ void inv_col(float2* Sb, int c) {
  constexpr int NH = BW / 2 + 1, HC = BW / 2;
  float2 col[BH];
  const bool dc = c == 0;
#pragma unroll
  for (int h = 0; h < BH; h++) {
    const float2 x0 = Sb[h * NH + c];
    if (dc) {
      const float2 xn = Sb[h * NH + HC];
      col[h] = make_float2(x0.x - xn.y, x0.y + xn.x);  // x0 + i xn
    } else {
      col[h] = x0;
    }
  }
  cfft<BH, +1>(col);
  if (dc) {
#pragma unroll
    for (int y = 0; y < BH; y++) {
      Sb[y * NH] = make_float2(col[y].x, 0.f);
      Sb[y * NH + HC] = make_float2(col[y].y, 0.f);
    }
  } else {
#pragma unroll
    for (int y = 0; y < BH; y++) Sb[y * NH + c] = col[y];
  }
}

// Row y: c2r along x; the BW real samples overwrite the row's own storage in
// Sb (BW floats fit in the row's BW/2+1 complex), for a coalesced copy-out.
template <int BW, int BH>
__device__ __forceinline__ void inv_row_inplace(float2* Sb, int y) {
  constexpr int NH = BW / 2 + 1;
  float2* row = Sb + y * NH;
  float2 c[NH];
#pragma unroll
  for (int k = 0; k < NH; k++) c[k] = row[k];
  float r[BW];
  irfft<BW>(c, r);
#pragma unroll
  for (int x = 0; x < BW / 2; x++) row[x] = make_float2(r[2 * x], r[2 * x + 1]);
}

// Coalesced store of one block's time-domain rows (left in Sb by
// inv_row_inplace, row pitch NH complex) to out[BH][BW].
template <int BW, int BH>
__device__ __forceinline__ void store_tdom(const float2* Sb, float* out, int lane) {
  constexpr int NH = BW / 2 + 1, HALF = BW / 2;
  float2* o = reinterpret_cast<float2*>(out);
  for (int i = lane; i < BH * HALF; i += 32) {
    const int y = i / HALF, x = i - y * HALF;
    o[i] = Sb[y * NH + x];
  }
}


// ---------------------------------------------------------------- forward

// k_frame's forward part: the CTA transforms `count` consecutive blocks into
// the tiles at S (a row, then a column per thread) and copies them to the
// ring; the tiles stay for the filter. The caller's next barrier ends the copy.
template <int BW, int BH, typename T>
__device__ __forceinline__ void frame_forward(const ForwardArgs& a, int blk0, int count, float2* S) {
  constexpr int NH = BW / 2 + 1, HC = BW / 2, BINS = BH * NH, NT = kWarps * 32;
  const ArgsFwd win{a};
  const int t = threadIdx.x;
  for (int i = t; i < count * BH; i += NT) {
    const int b = i / BH;
    fwd_row<BW, BH, T, false>(a, win, blk0 + b, i - b * BH, S + b * BINS);
  }
  __syncthreads();
  for (int i = t; i < count * HC; i += NT) {
    const int b = i / HC;
    fwd_col<BW, BH>(S + b * BINS, i - b * HC);
  }
  __syncthreads();
  float4* dst = reinterpret_cast<float4*>(a.spec + (size_t)blk0 * BINS);
  const float4* src = reinterpret_cast<const float4*>(S);
  for (int i = t; i < count * BINS / 2; i += NT)
    if (FFT3D_IN((size_t)blk0 * BINS / 2 + i < (size_t)a.g.nblocks * BINS / 2 && a.spec != nullptr, a.err)) dst[i] = src[i];
}

// Blocks of a forward CTA, and its threads: one per column (DC and Nyquist
// columns count as one), so that the column transforms are one full round
// and the row pairs of square blocks too (48 x 48: 4 blocks, 96 threads; a
// warp per block left a quarter of its lanes idle in both).
template <int BW>
__host__ __device__ constexpr int fwd_blocks() { return kWarps * blocks_per_warp<BW>(); }
template <int BW>
__host__ __device__ constexpr int fwd_threads() { return fwd_blocks<BW>() * (BW / 2); }
// Whether a thread takes two rows at once, or one: pairs, unless a block has so
// few rows that its pairs fill half the threads or less, or two thirds where two
// rows of 48 samples take the registers of more than 96 a thread. us per frame
// with pairs / single rows: 32 x 16, 800 blocks 10.2 / 8.7, 16000 blocks 21.7 /
// 18.9; 48 x 16, 16000 blocks 38.6 / 30.5; 48 x 32, 3600 blocks 21.2 / 19.1, 16000
// blocks 50.2 / 45.5; 24 x 16, 1600 blocks 9.3 / 10.6, 16000 blocks 18.9 / 18.6; 32 x
// 32, 8000 blocks 20.7 / 21.4.
template <int BW, int BH>
__host__ __device__ constexpr bool fwd_pairs() { return BH * 4 > BW * (BW > 32 ? 3 : 2); }

// Forward transform of fwd_blocks<BW>() consecutive blocks per CTA.
//  rows: a thread takes one row, or (fwd_pairs) rows y and y + bh/2 of a block at
//   once, packed
//   (rfft_pair): gather with mirrored edges, analysis window, r2c; their
//   spectra go to shared memory interleaved, 16 bytes per bin {A.re, B.re,
//   A.im, B.im};
//  columns: a thread takes a column (bh/2 16-byte reads), transforms it and,
//   when every thread of the block has read its column, writes it back as
//   (re, im) rows;
//  one bulk copy of the contiguous spectra to global memory per group.
// Where a block's threads lie in one warp (square blocks of 8, 16 and 32) the
// stages are separated by __syncwarp, else by CTA barriers.
// Bound by issue and shared-memory traffic: 18.7 us per 1080p frame of 32 x 32
// blocks (all planes; 818 instructions per block with the copy-out by 16-byte
// loads and stores, then 21.1 us) against 21.2 (1166) with one row at a time.
template <int BW, int BH, typename T, class Win>
__device__ __forceinline__ void forward_blocks(const ForwardArgs& a, int cta, const Win& win) {
  constexpr int NH = BW / 2 + 1, HC = BW / 2, HB = BH / 2, BINS = BH * NH, NT = fwd_threads<BW>();
  constexpr bool PAIRS = fwd_pairs<BW, BH>();
  constexpr bool WARP = (PAIRS ? HB : BH) == HC && 32 % HC == 0;  // a block's work stays in one warp
  constexpr int GT = WARP ? 32 : NT, GB = GT / HC;  // threads and blocks of a group that synchronises
  constexpr int WORDS = BW * (int)sizeof(T) / 4;
  extern __shared__ __align__(16) float2 smem2[];
  const Geom& g = a.g;
  const int grp = threadIdx.x / GT, t = threadIdx.x - grp * GT;
  const int blk0 = cta * fwd_blocks<BW>() + grp * GB;
  const int nvalid = min(GB, g.nblocks - blk0);
  float2* S = smem2 + grp * GB * BINS;
  auto sync = [] {
    if constexpr (WARP) __syncwarp();
    else __syncthreads();
  };
  if (WARP && nvalid <= 0) return;
  if constexpr (!PAIRS)
    for (int i = t; i < GB * BH; i += GT) {
      const int b = i / BH;
      if (b < nvalid) fwd_row<BW, BH, T, true>(a, win, blk0 + b, i - b * BH, S + b * BINS);
    }
  for (int i = t; PAIRS && i < GB * HB; i += GT) {
    const int b = i / HB, y = i - b * HB;
    if (b >= nvalid) continue;
    float4* quads = reinterpret_cast<float4*>(S + b * BINS) + y * NH;
    int x0, rowA, rowB;
    const T* srcA = fwd_row_src<T>(a, win, blk0 + b, y, &x0, &rowA);
    const T* srcB = fwd_row_src<T>(a, win, blk0 + b, y + HB, &x0, &rowB);
    const bool okA = FFT3D_IN(rowA >= 0 && rowA < g.H, a.err), okB = FFT3D_IN(rowB >= 0 && rowB < g.H, a.err);
    f2x v[BW];
    const float off = (sizeof(T) < 4 ? 8388608.0f : 0.f) + a.base;  // exact: base <= 2^15
    const f2x noff = dup2(-off);
    if (x0 >= 0 && x0 + BW <= g.W && okA && okB) {
      uint32_t wA[WORDS], wB[WORDS];
      load_words<T, BW>(srcA + x0, wA);
      load_words<T, BW>(srcB + x0, wB);
#pragma unroll
      for (int x = 0; x < BW; x++) v[x] = pk2(raw_sample<T>(wA, x), raw_sample<T>(wB, x));
    } else {
      // mirrored columns: sample by sample through the thread's own part of
      // the tile (as samples plus the offset that the common path takes off)
      f2x* own = reinterpret_cast<f2x*>(quads);
      const float up = sizeof(T) < 4 ? 8388608.0f : 0.f;
#pragma unroll 8
      for (int x = 0; x < BW; x++) {
        const int xi = reflect101(x0 + x, g.W);
        const bool in = FFT3D_IN(xi >= 0 && xi < g.W, a.err);
        own[x] = pk2(in && okA ? load_sample<T>(srcA + xi) + up : off, in && okB ? load_sample<T>(srcB + xi) + up : off);
      }
#pragma unroll
      for (int x = 0; x < BW; x++) v[x] = own[x];
    }
    const f2x wy = pk2(__ldg(a.wan_y + y), __ldg(a.wan_y + y + HB));
#pragma unroll
    for (int x = 0; x < BW; x++)
      v[x] = mul2_kept(mul2(add2(v[x], noff), *reinterpret_cast<const f2x*>(&a.wx_half[x])), wy);
    f2x re[NH], im[NH];
    rfft_pair<BW>(v, re, im);
#pragma unroll
    for (int k = 0; k < NH; k++) {
      const float2 r = up2(re[k]), q = up2(im[k]);
      quads[k] = make_float4(r.x, r.y, q.x, q.y);
    }
  }
  sync();
  float2 col[BH];
  const int cb = t / HC, c = t - cb * HC;
  const bool mine = cb < nvalid;
  float2* Sb = S + cb * BINS;
  if constexpr (!PAIRS) {
    if (mine) fwd_col<BW, BH>(Sb, c);
  } else {
    if (mine) {
      const float4* quads = reinterpret_cast<const float4*>(Sb);
#pragma unroll
      for (int y = 0; y < HB; y++) {
        const float4 q = quads[y * NH + c];
        col[y] = make_float2(q.x, q.z);
        col[y + HB] = make_float2(q.y, q.w);
        if (c == 0) {  // real columns 0 and bw/2 as one complex sequence
          const float4 n = quads[y * NH + HC];
          col[y].y = n.x;
          col[y + HB].y = n.y;
        }
      }
    }
    sync();
    if (mine) {
      cfft<BH, -1>(col);
      if (c == 0) {
#pragma unroll
        for (int h = 0; h < BH; h++) {
          const float2 zh = col[h], zm = cconj(col[(BH - h) % BH]);
          Sb[h * NH] = make_float2(0.5f * (zh.x + zm.x), 0.5f * (zh.y + zm.y));
          const float2 d = csub(zh, zm);
          Sb[h * NH + HC] = make_float2(0.5f * d.y, -0.5f * d.x);
        }
      } else {
#pragma unroll
        for (int h = 0; h < BH; h++) Sb[h * NH + c] = col[h];
      }
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  sync();
  if (t == 0 && nvalid > 0 && FFT3D_IN(blk0 + nvalid <= g.nblocks && win.spec() != nullptr, a.err)) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(win.spec() + (size_t)blk0 * BINS),
                 "r"(smem_addr(S)), "r"(nvalid * BINS * 8)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the tiles are read before the CTA leaves them
  }
}

template <int BW, int BH>
__host__ __device__ constexpr int fwd_smem() { return fwd_blocks<BW>() * BH * (BW / 2 + 1) * 8; }
// CTAs per SM: two packed rows of 32 samples are 64 registers (20 warps, 96
// registers a thread), of 48 samples 96 (15 warps).
template <int BW, int BH>
__host__ __device__ constexpr int fwd_ctas() {
  return ctas_for((BW > 32 || BH > 32 ? 15 : 20) * 32 / fwd_threads<BW>(), fwd_smem<BW, BH>());
}

// The new frames of one or more output frames in one launch: CTA x transforms
// CTA x % fs.ctas of frame x / fs.ctas (one launch instead of one per frame,
// so the grid has no per-frame wave tail).
template <int BW, int BH, typename T>
__global__ void __launch_bounds__(fwd_threads<BW>(), (fwd_ctas<BW, BH>()))
    k_forward_frames(const __grid_constant__ ForwardArgs a, const __grid_constant__ FwdFrameSet fs) {
  const int j = blockIdx.x / fs.ctas, c = blockIdx.x - j * fs.ctas;
  forward_blocks<BW, BH, T>(a, c, FrameFwd{fs.src[j], fs.stride[j], fs.spec[j]});
}

// Batched forward: work item i = (plane, CTA of that plane); the grid walks
// the items (persistent when the grid is smaller than the item count).
template <int BW, int BH, typename T>
__global__ void __launch_bounds__(fwd_threads<BW>(), (ctas_for(16 * 32 / fwd_threads<BW>(), fwd_smem<BW, BH>() + (int)sizeof(ForwardArgs))))
    k_forward_batch(const ForwardArgs* __restrict__ args, const int2* __restrict__ items, int nitems) {
  // the item's arguments staged in shared memory: the body's stores cannot
  // alias them, and they cost no registers
  __shared__ __align__(16) ForwardArgs sa;
  static_assert(sizeof(ForwardArgs) % 4 == 0, "word copy");
  for (int i = blockIdx.x; i < nitems; i += gridDim.x) {
    const int2 it = items[i];
    __syncthreads();  // every warp is done with the previous item's arguments and tiles
    const int* src = reinterpret_cast<const int*>(args + it.x);
    int* dst = reinterpret_cast<int*>(&sa);
    for (int w = threadIdx.x; w < (int)(sizeof(ForwardArgs) / 4); w += blockDim.x) dst[w] = src[w];
    __syncthreads();
    forward_blocks<BW, BH, T>(sa, it.y, ArgsFwd{sa});
  }
}

// ---------------------------------------------------------------- filters

// The per-bin table values one bin's filter reads (the same for every
// block). Loaded before the filter arithmetic, so that their latency is
// hidden behind it instead of stalling the first use.
struct BinTab {
  float2 grid;  // gridsample, when degrid != 0
  float wsh;    // sharpen weight, when sharpen != 0
  float wdh;    // dehalo weight, when dehalo != 0
};
// Only the values that MODE's filter and the sharpen pass read are loaded
// (Kalman and sharpen-only read the grid only in a sharpen pass; the weights
// are read by a sharpen pass or by Wiener 2D's fused factor).
template <int MODE>
__device__ __forceinline__ BinTab bin_tab(const InverseArgs& a, int bin) {
  BinTab t{make_float2(0.f, 0.f), 0.f, 0.f};
  const bool sh = a.c.do_sharpen || (MODE == MODE_WIENER2D && a.c.fuse_sharpen);
  if (a.c.degrid != 0.f && (MODE >= 1 || a.c.do_sharpen)) t.grid = __ldg(a.t.grid + bin);
  if (sh && a.c.use_sharpen) t.wsh = __ldg(a.t.wsharpen + bin);
  if (sh && a.c.use_dehalo) t.wdh = __ldg(a.t.wdehalo + bin);
  return t;
}

// |c|^2 + 1e-15 of a bin (the reference's psd, src/code_impl/Apply.cpp:27-31)
__device__ __forceinline__ float bin_psd(float re, float im) { return fmaf(re, re, fmaf(im, im, 1.0e-15f)); }

__device__ __forceinline__ float sharpen_fact(const InverseArgs& a, float psd, float wsh) {
  // src/code_impl/Apply.cpp:129-131: 1 + sharpen * wsh * sqrt(r) with
  // r = psd * smax2n / ((psd + smin2n)(psd + smax2n)) in [0, 1), the ratio
  // first as in the reference (the product of its terms overflows float for
  // high bit depths), its square root as r * rsqrt(r) (the clamp keeps r = 0,
  // i.e. smax = 0, finite)
  const float r = psd * a.c.smax2n * rcp_nrm((psd + a.c.smin2n) * (psd + a.c.smax2n));
  return fmaf(a.c.sharpen * wsh, r * rsqrt_nrm(fmaxf(r, 1e-30f)), 1.f);
}
__device__ __forceinline__ float dehalo_fact(const InverseArgs& a, float psd, float wdh) {
  // src/code_impl/Apply.cpp:132
  return (psd + a.c.ht2n) * rcp_nrm((psd + a.c.ht2n) + a.c.dehalo * wdh * psd);
}

// limited Wiener factor applied to one temporal component, code_impl_C.h:34-40:
// max((psd - noise) / psd, lowlimit) as max(1 - noise / psd, lowlimit) with
// the fast reciprocal (<= 2 ulp, far inside the +-1 LSB output bar)
// (both parts scaled by one packed multiply)
__device__ __forceinline__ void wiener(float2& v, float noise, float lowlimit) {
  const float q = fmaf(-noise, rcp_nrm(bin_psd(v.x, v.y)), 1.f);
  const float f = fmaxf(q, lowlimit);
  v = __fmul2_rn(v, make_float2(f, f));
}

// Learned noise power of bin `bin` of the block at spectrum offset `off`.
__device__ __forceinline__ float learned_noise(const InverseArgs& a, size_t off, int bin) {
  return a.psd_scale * __ldg(a.psd + (a.psd_per_block ? off : 0) + bin);
}

// One Kalman step of one bin, src/code_impl/Kalman.cpp:27-64: the motion test
// per component (OR), then either a reset to the current value or the gain
// update; last/cv/cp are the bin's state (filtered value, covariance, process
// covariance), updated in place. `sigma` is the bin's noise power.
__device__ __forceinline__ void kalman_step(const InverseArgs& a, float2 cur, float sigma, float2& last, float& cv,
                                            float& cp) {
  const float dr = cur.x - last.x, di = cur.y - last.y;
  if (dr * dr > sigma * a.c.kratio2 || di * di > sigma * a.c.kratio2) {
    cv = sigma;
    cp = sigma;
    last = cur;
  } else {
    const float sum = cv + cp;
    const float gain = sum * rcp_nrm(sum + sigma);
    cp = gain * gain * sigma;
    cv = (1.f - gain) * sum;
    last.x = gain * cur.x + (1.f - gain) * last.x;
    last.y = gain * cur.y + (1.f - gain) * last.y;
  }
}

// Filtered value of one bin from its values w[0..4] in frames n-2..n+2 (only
// the window's entries are read). MODE: 1 = Wiener 2D, 2..5 = Wiener 3D,
// 0 = Kalman (updates the state when `commit`), -1 = sharpen only (identity).
template <int MODE>
__device__ __forceinline__ float2 filter_vals(const InverseArgs& a, const float2 (&w)[5], size_t off, int bin, float gf,
                                              const BinTab& tb, bool commit) {
  const float2 cur = w[2];
  if constexpr (MODE == MODE_SHARPEN_ONLY) {
    return cur;
  } else if constexpr (MODE == MODE_KALMAN) {
    // src/code_impl/Kalman.cpp:27-64; the state is read once and written
    // back by this thread: coherent loads that do not allocate in L1
    float2 last;
    float cv, cp;
    asm("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(last.x), "=f"(last.y) : "l"(a.kal_last + off + bin));
    asm("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(cv) : "l"(a.kal_covar + off + bin));
    asm("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(cp) : "l"(a.kal_covarp + off + bin));
    float sigma = a.c.sigma2n_2d;
    if (a.psd) {
      sigma = learned_noise(a, off, bin);
      if (sigma < 1e-15f) sigma = 1e-15f;
    } else if (a.c.pattern) {
      sigma = __ldg(a.t.pattern2d + bin);
      if (sigma < 1e-15f) sigma = 1e-15f;
    }
    kalman_step(a, cur, sigma, last, cv, cp);
    if (commit) {
      a.kal_last[off + bin] = last;
      a.kal_covar[off + bin] = cv;
      a.kal_covarp[off + bin] = cp;
    }
    return last;
  } else if constexpr (MODE == MODE_WIENER2D) {
    // src/code_impl/Apply.cpp:13-65
    float2 gc = make_float2(0.f, 0.f);
    if (a.c.degrid != 0.f) gc = make_float2(gf * tb.grid.x, gf * tb.grid.y);
    const float cr = cur.x - gc.x, ci = cur.y - gc.y;
    const float psd = bin_psd(cr, ci);
    const float noise = a.psd ? learned_noise(a, off, bin) : a.c.pattern ? __ldg(a.t.pattern2d + bin) : a.c.sigma2n;
    float f = fmaxf(fmaf(-noise, rcp_nrm(psd), 1.f), a.c.lowlimit);
    if (a.c.fuse_sharpen) {
      if (a.c.use_sharpen && a.c.use_dehalo) f *= sharpen_fact(a, psd, tb.wsh) * dehalo_fact(a, psd, tb.wdh);
      else if (a.c.use_sharpen) f *= sharpen_fact(a, psd, tb.wsh);
      else if (a.c.use_dehalo) f *= dehalo_fact(a, psd, tb.wdh);
    }
    return make_float2(cr * f + gc.x, ci * f + gc.y);
  } else {
    // Wiener 3D over MODE frames, src/code_impl/Apply.cpp:67-235. The short
    // temporal DFT works on (re, im) pairs with packed f32x2 adds and
    // multiplies (one instruction per complex sum or real-scaled term); the
    // terms and their signs are the reference's, the association of a few
    // sums differs (rounding only). gc * bt (src/code_impl/Apply.cpp:78-93)
    // uses gf * MODE, the same for every bin of the block.
    const float gk = gf * (float)MODE;
    float2 g = make_float2(0.f, 0.f);
    if (a.c.degrid != 0.f) g = __fmul2_rn(tb.grid, make_float2(gk, gk));
    const float noise = a.psd ? learned_noise(a, off, bin) : a.c.pattern ? __ldg(a.t.pattern3d + bin) : a.c.sigma2n;
    const float ll = a.c.lowlimit;
    auto wf = [&](float2& v) { wiener(v, noise, ll); };
    auto add = [](float2 x, float2 y) { return __fadd2_rn(x, y); };
    auto sub = [](float2 x, float2 y) { return __fadd2_rn(x, make_float2(-y.x, -y.y)); };
    auto rot = [](float2 v) { return make_float2(v.y, -v.x); };  // -i v
    if constexpr (MODE == 2) {
      const float2 pv = w[1];
      float2 f0 = sub(add(cur, pv), g), f1 = sub(cur, pv);
      wf(f0);
      wf(f1);
      return __fmul2_rn(add(add(f0, f1), g), make_float2(0.5f, 0.5f));
    } else if constexpr (MODE == 3) {
      const float sin120 = 0.86602540378443864676372317075294f;
      const float2 pv = w[1], nx = w[3];
      const float2 pn = add(pv, nx);
      float2 fc = sub(add(cur, pn), g);
      const float2 h = __ffma2_rn(pn, make_float2(-0.5f, -0.5f), cur);      // cur - pn / 2
      const float2 m = rot(__fmul2_rn(sub(pv, nx), make_float2(sin120, sin120)));  // (di, dr)
      float2 fp = add(h, m), fn = sub(h, m);
      wf(fc);
      wf(fp);
      wf(fn);
      const float third = 1.0f / 3.0f;
      return __fmul2_rn(add(add(add(fc, fp), fn), g), make_float2(third, third));
    } else if constexpr (MODE == 4) {
      const float2 p2 = w[0], pv = w[1], nx = w[3];
      const float2 cp = add(cur, p2), cm = sub(cur, p2), pn = add(pv, nx);
      const float2 d = rot(sub(pv, nx));  // (pv.y - nx.y, nx.x - pv.x)
      float2 fp2 = sub(cp, pn), fc = sub(add(cp, pn), g);
      float2 fp = add(cm, d), fn = sub(cm, d);
      wf(fp2);
      wf(fp);
      wf(fc);
      wf(fn);
      return __fmul2_rn(add(add(add(fp2, fp), add(fc, fn)), g), make_float2(0.25f, 0.25f));
    } else {
      const float sin72 = 0.95105651629515357211643933337938f, cos72 = 0.30901699437494742410229341718282f;
      const float sin144 = 0.58778525229247312916870595463907f, cos144 = -0.80901699437494742410229341718282f;
      const float2 p2 = w[0], pv = w[1], nx = w[3], n2 = w[4];
      const float2 a2 = add(p2, n2), a1 = add(pv, nx);  // outer and inner pair sums
      const float2 e2 = sub(n2, p2), e1 = sub(pv, nx);  // their differences
      const float2 s1 = add(__ffma2_rn(a2, make_float2(cos72, cos72), __fmul2_rn(a1, make_float2(cos144, cos144))), cur);
      const float2 s2 = add(__ffma2_rn(a2, make_float2(cos144, cos144), __fmul2_rn(a1, make_float2(cos72, cos72))), cur);
      // -i (e2 sin72 + e1 sin144) and -i (e1 sin72 - e2 sin144)
      const float2 t1 = rot(__ffma2_rn(e2, make_float2(sin72, sin72), __fmul2_rn(e1, make_float2(sin144, sin144))));
      const float2 t2 = rot(__ffma2_rn(e2, make_float2(-sin144, -sin144), __fmul2_rn(e1, make_float2(sin72, sin72))));
      float2 fp2 = add(s1, t1), fn2 = sub(s1, t1);
      float2 fp = add(s2, t2), fn = sub(s2, t2);
      float2 fc = sub(add(add(a2, a1), cur), g);
      wf(fp2);
      wf(fp);
      wf(fc);
      wf(fn);
      wf(fn2);
      return __fmul2_rn(add(add(add(add(fp2, fp), add(fc, fn)), fn2), g), make_float2(0.2f, 0.2f));
    }
  }
}

// Window slots 2 - MODE/2 .. 2 + (MODE-1)/2 of a MODE-frame Wiener 3D (the
// reference's apply_in[] table, src/fft3d_engine.h:634-644); one slot otherwise.
template <int MODE>
__host__ __device__ constexpr int win_lo() { return MODE >= 2 ? 2 - MODE / 2 : 2; }
template <int MODE>
__host__ __device__ constexpr int win_hi() { return MODE >= 2 ? 2 + (MODE - 1) / 2 : 2; }

// separate sharpen/dehalo pass on a filtered bin, src/code_impl/Sharpen.cpp:13-63
// (the grid term removed and restored with packed f32x2 operations)
__device__ __forceinline__ float2 sharpen_bin(const InverseArgs& a, float2 v, const BinTab& tb, float gf) {
  float2 gc = make_float2(0.f, 0.f);
  if (a.c.degrid != 0.f) gc = __fmul2_rn(tb.grid, make_float2(gf, gf));
  const float2 c = __fadd2_rn(v, make_float2(-gc.x, -gc.y));
  const float psd = bin_psd(c.x, c.y);
  float f;
  if (a.c.use_sharpen && a.c.use_dehalo) f = sharpen_fact(a, psd, tb.wsh) * dehalo_fact(a, psd, tb.wdh);
  else if (a.c.use_sharpen) f = sharpen_fact(a, psd, tb.wsh);
  else f = dehalo_fact(a, psd, tb.wdh);
  return __ffma2_rn(c, make_float2(f, f), gc);
}

// ---------------------------------------------------------------- filters, two bins at a time

__device__ __forceinline__ f2x rcp2(f2x v) {
  const float2 u = up2(v);
  return pk2(rcp_nrm(u.x), rcp_nrm(u.y));
}
__device__ __forceinline__ f2x max2(f2x v, float w) {
  const float2 u = up2(v);
  return pk2(fmaxf(u.x, w), fmaxf(u.y, w));
}

// Two neighbouring bins: their real parts and their imaginary parts, packed.
// The filter's arithmetic is the same for both bins, so every sum, product
// and fused multiply-add of the pair is one instruction, the turns by -i cost
// nothing (re and im change places), and the pair's Wiener factors come as a
// packed value that scales both parts. A pair gives what filter_vals and
// sharpen_bin give for its two bins, bit for bit.
struct Pair {
  f2x re, im;
};
// The filter's constants as pairs, read from the constant bank by the packed
// instructions.
__constant__ float2 c_pair[] = {
    {0.30901699437494742410229341718282f, 0.30901699437494742410229341718282f},    // kCos72
    {-0.80901699437494742410229341718282f, -0.80901699437494742410229341718282f},  // kCos144
    {0.95105651629515357211643933337938f, 0.95105651629515357211643933337938f},    // kSin72
    {0.58778525229247312916870595463907f, 0.58778525229247312916870595463907f},    // kSin144
    {-0.58778525229247312916870595463907f, -0.58778525229247312916870595463907f},  // kMinusSin144
    {0.86602540378443864676372317075294f, 0.86602540378443864676372317075294f},    // kSin120
    {-0.5f, -0.5f},                                                                // kMinusHalf
    {1.0e-15f, 1.0e-15f},                                                          // kPsdFloor
    {1.f, 1.f},                                                                    // kOne
    {0.5f, 0.5f},                                                                  // kHalf
    {1.0f / 3.0f, 1.0f / 3.0f},                                                    // kThird
    {0.25f, 0.25f},                                                                // kQuarter
    {0.2f, 0.2f},                                                                  // kFifth
};
enum PairConst { kCos72, kCos144, kSin72, kSin144, kMinusSin144, kSin120, kMinusHalf, kPsdFloor, kOne, kHalf, kThird, kQuarter, kFifth };
__device__ __forceinline__ f2x kc(PairConst k) { return reinterpret_cast<const f2x*>(c_pair)[k]; }

__device__ __forceinline__ Pair pair_of(const float4& v) { return Pair{pk2(v.x, v.z), pk2(v.y, v.w)}; }
__device__ __forceinline__ float4 bins_of(const Pair& p) {
  const float2 re = up2(p.re), im = up2(p.im);
  return make_float4(re.x, im.x, re.y, im.y);
}
__device__ __forceinline__ Pair padd(const Pair& x, const Pair& y) { return Pair{add2(x.re, y.re), add2(x.im, y.im)}; }
__device__ __forceinline__ Pair pscale_kept(const Pair& x, f2x s) { return Pair{mul2_kept(x.re, s), mul2_kept(x.im, s)}; }
__device__ __forceinline__ Pair psub(const Pair& x, const Pair& y) { return Pair{sub2(x.re, y.re), sub2(x.im, y.im)}; }
__device__ __forceinline__ Pair pscale(const Pair& x, f2x s) { return Pair{mul2(x.re, s), mul2(x.im, s)}; }
__device__ __forceinline__ Pair pfma(const Pair& x, f2x s, const Pair& y) { return Pair{fma2(x.re, s, y.re), fma2(x.im, s, y.im)}; }
// x - i v and x + i v
__device__ __forceinline__ Pair psub_i(const Pair& x, const Pair& v) { return Pair{add2(x.re, v.im), sub2(x.im, v.re)}; }
__device__ __forceinline__ Pair padd_i(const Pair& x, const Pair& v) { return Pair{sub2(x.re, v.im), add2(x.im, v.re)}; }
__device__ __forceinline__ f2x ppsd(const Pair& v) { return fma2(v.re, v.re, fma2(v.im, v.im, kc(kPsdFloor))); }
// The factors of wiener() for both bins; nn: minus their noise powers. The
// parts scaled by them are summed with fused multiply-adds, as the compiler
// contracts filter_vals' sums: fma(x, fx, y fy) for x fx + y fy.
__device__ __forceinline__ f2x pfactor(const Pair& v, f2x nn, float lowlimit) {
  return max2(fma2(nn, rcp2(ppsd(v)), kc(kOne)), lowlimit);
}
__device__ __forceinline__ Pair psum2(const Pair& x, f2x fx, const Pair& y, f2x fy) { return pfma(x, fx, pscale(y, fy)); }

// filter_vals of a Wiener 3D mode for a pair; w: the pair in the window's
// frames, grid: the pair's gridsample (zeros without degrid), gf: the block's
// grid fraction, nn: minus the pair's noise powers. (The last scaling is kept
// apart from the subtraction that a sharpen pass begins with; a half and a
// quarter are exact either way.)
template <int MODE>
__device__ __forceinline__ Pair filter_pair(const Pair (&w)[5], const Pair& grid, float gf, f2x nn, float ll) {
  static_assert(MODE >= 2 && MODE <= 5, "Wiener 3D");
  const Pair cur = w[2], g = pscale_kept(grid, dup2(gf * (float)MODE));
  auto factor = [&](const Pair& v) { return pfactor(v, nn, ll); };
  if constexpr (MODE == 2) {
    const Pair f0 = psub(padd(cur, w[1]), g), f1 = psub(cur, w[1]);
    return pscale(padd(psum2(f0, factor(f0), f1, factor(f1)), g), kc(kHalf));
  } else if constexpr (MODE == 3) {
    const Pair pn = padd(w[1], w[3]);
    const Pair fc = psub(padd(cur, pn), g);
    const Pair h = pfma(pn, kc(kMinusHalf), cur), d = pscale_kept(psub(w[1], w[3]), kc(kSin120));
    const Pair fp = psub_i(h, d), fn = padd_i(h, d);
    return pscale_kept(padd(pfma(fn, factor(fn), psum2(fc, factor(fc), fp, factor(fp))), g), kc(kThird));
  } else if constexpr (MODE == 4) {
    const Pair cp = padd(cur, w[0]), cm = psub(cur, w[0]), pn = padd(w[1], w[3]), d = psub(w[1], w[3]);
    const Pair fp2 = psub(cp, pn), fc = psub(padd(cp, pn), g);
    const Pair fp = psub_i(cm, d), fn = padd_i(cm, d);
    return pscale(padd(padd(psum2(fp2, factor(fp2), fp, factor(fp)), psum2(fc, factor(fc), fn, factor(fn))), g),
                  kc(kQuarter));
  } else {
    const Pair a2 = padd(w[0], w[4]), a1 = padd(w[1], w[3]);
    const Pair e2 = psub(w[4], w[0]), e1 = psub(w[1], w[3]);
    const Pair s1 = padd(pfma(a2, kc(kCos72), pscale(a1, kc(kCos144))), cur);
    const Pair s2 = padd(pfma(a2, kc(kCos144), pscale(a1, kc(kCos72))), cur);
    const Pair t1 = pfma(e2, kc(kSin72), pscale(e1, kc(kSin144)));
    const Pair t2 = pfma(e2, kc(kMinusSin144), pscale(e1, kc(kSin72)));
    const Pair fp2 = psub_i(s1, t1), fn2 = padd_i(s1, t1);
    const Pair fp = psub_i(s2, t2), fn = padd_i(s2, t2);
    const Pair fc = psub(padd(padd(a2, a1), cur), g);
    const Pair sum = padd(psum2(fp2, factor(fp2), fp, factor(fp)), psum2(fc, factor(fc), fn, factor(fn)));
    return pscale_kept(padd(pfma(fn2, factor(fn2), sum), g), kc(kFifth));
  }
}

// sharpen_fact x dehalo_fact (those that are on) of a pair of power spectra
__device__ __forceinline__ f2x sharpen_factor(const InverseArgs& a, f2x psd, f2x wsh, f2x wdh) {
  f2x f = kc(kOne);
  if (a.c.use_sharpen) {
    const f2x smax = dup2(a.c.smax2n);
    const f2x r = mul2(mul2(psd, smax), rcp2(mul2(add2(psd, dup2(a.c.smin2n)), add2(psd, smax))));
    const float2 m = up2(max2(r, 1e-30f));
    f = fma2(mul2(dup2(a.c.sharpen), wsh), mul2(r, pk2(rsqrt_nrm(m.x), rsqrt_nrm(m.y))), kc(kOne));
  }
  if (a.c.use_dehalo || !a.c.use_sharpen) {
    const f2x top = add2(psd, dup2(a.c.ht2n));
    const f2x d = mul2(top, rcp2(fma2(mul2(dup2(a.c.dehalo), wdh), psd, top)));
    f = a.c.use_sharpen ? mul2(f, d) : d;
  }
  return f;
}

// sharpen_bin of a pair; wsh, wdh: the pair's weights.
__device__ __forceinline__ Pair sharpen_pair(const InverseArgs& a, const Pair& v, const Pair& grid, f2x wsh, f2x wdh,
                                             float gf) {
  const Pair gc = pscale_kept(grid, dup2(gf)), c = psub(v, gc);
  const f2x f = sharpen_factor(a, ppsd(c), wsh, wdh);
  return Pair{fma2(c.re, f, gc.re), fma2(c.im, f, gc.im)};
}

// filter_vals<MODE_WIENER2D> of a pair, the sharpen/dehalo factors in its
// Wiener factor where the filter fuses them.
__device__ __forceinline__ Pair wiener2d_pair(const InverseArgs& a, const Pair& v, const Pair& grid, float gf, f2x nn,
                                              f2x wsh, f2x wdh) {
  const Pair gc = pscale_kept(grid, dup2(gf)), c = psub(v, gc);
  const f2x psd = ppsd(c);
  f2x f = max2(fma2(nn, rcp2(psd), kc(kOne)), a.c.lowlimit);
  if (a.c.fuse_sharpen && (a.c.use_sharpen || a.c.use_dehalo)) f = mul2(f, sharpen_factor(a, psd, wsh, wdh));
  return Pair{fma2(c.re, f, gc.re), fma2(c.im, f, gc.im)};
}

// The gridsample of bins bin, bin + 1, or zeros without degrid.
__device__ __forceinline__ Pair pair_grid(const InverseArgs& a, int bin) {
  if (a.c.degrid == 0.f) return Pair{0, 0};
  return pair_of(__ldg(reinterpret_cast<const float4*>(a.t.grid + bin)));
}
// Minus the noise powers of bins bin, bin + 1 of the block at `off`.
template <int MODE>
__device__ __forceinline__ f2x pair_noise(const InverseArgs& a, size_t off, int bin) {
  if (a.psd) return pk2(-learned_noise(a, off, bin), -learned_noise(a, off, bin + 1));
  if (a.c.pattern) {
    const float2 p = __ldg(reinterpret_cast<const float2*>((MODE >= 2 ? a.t.pattern3d : a.t.pattern2d) + bin));
    return pk2(-p.x, -p.y);
  }
  return dup2(-a.c.sigma2n);
}
// Two neighbouring weights of a per-bin table, or zeros where it is not used.
__device__ __forceinline__ f2x pair_weights(const float* table, bool use, int bin) {
  if (!use) return 0;
  const float2 w = __ldg(reinterpret_cast<const float2*>(table + bin));
  return pk2(w.x, w.y);
}

// One frame of one bin pair from its window's values r[LO .. HI]. Wiener and
// sharpen-only modes.
template <int MODE>
__device__ __forceinline__ float4 group_filter_one(const InverseArgs& a, size_t off, int bin, const float4 (&r)[5],
                                                   float gf) {
  constexpr int LO = win_lo<MODE>(), HI = win_hi<MODE>();
  if constexpr (MODE >= 2) {
    Pair w[5];
#pragma unroll
    for (int k = 0; k < 5; k++) w[k] = pair_of(r[k >= LO && k <= HI ? k : LO]);
    return bins_of(filter_pair<MODE>(w, pair_grid(a, bin), gf, pair_noise<MODE>(a, off, bin), a.c.lowlimit));
  } else if constexpr (MODE == MODE_WIENER2D) {
    const bool fuse = a.c.fuse_sharpen;
    return bins_of(wiener2d_pair(a, pair_of(r[2]), pair_grid(a, bin), gf, pair_noise<MODE>(a, off, bin),
                                 pair_weights(a.t.wsharpen, fuse && a.c.use_sharpen, bin),
                                 pair_weights(a.t.wdehalo, fuse && a.c.use_dehalo, bin)));
  } else {
    return r[2];
  }
}

// ---------------------------------------------------------------- filter (streaming)

// Two neighbouring bins of a window spectrum, read once per thread: not kept
// in L1 (the per-bin tables stay there).
__device__ __forceinline__ float4 ld_stream4(const float2* p) {
  float4 v;
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// Filter of every bin of every block as a flat stream: each thread takes two
// neighbouring bins (one 16-byte load per window frame, one 16-byte store of
// the filtered pair to F). No shared memory and few registers, so the SMs
// hold enough warps to keep the spectrum reads at HBM speed. The separate
// sharpen/dehalo pass, which needs each block's filtered DC, runs afterwards
// in k_filter_inverse<MODE_SHARPEN_ONLY> on F.
template <int MODE>
__global__ void __launch_bounds__(256) k_filter_bins(InverseArgs a, float2* F, int bins_per_block) {
  constexpr int LO = win_lo<MODE>(), NW = win_hi<MODE>() - win_lo<MODE>() + 1;
  const size_t pairs = (size_t)a.g.nblocks * bins_per_block / 2;
  const float gs0 = __ldg(&a.t.grid[0].x);
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < pairs; q += (size_t)gridDim.x * blockDim.x) {
    const size_t e = 2 * q;
    const int bin = (int)(e % bins_per_block);
    const size_t off = e - bin;
    float4 wv[NW];
#pragma unroll
    for (int k = 0; k < NW; k++) wv[k] = __ldg(reinterpret_cast<const float4*>(a.in[LO + k] + e));
    const float gf = (MODE >= 1) ? a.c.degrid * __ldg(&a.in[2][off].x) / gs0 : 0.f;
    float2 w0[5], w1[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
      const bool in = k >= LO && k < LO + NW;
      w0[k] = in ? make_float2(wv[k - LO].x, wv[k - LO].y) : make_float2(0.f, 0.f);
      w1[k] = in ? make_float2(wv[k - LO].z, wv[k - LO].w) : make_float2(0.f, 0.f);
    }
    const float2 v0 = filter_vals<MODE>(a, w0, off, bin, gf, bin_tab<MODE>(a, bin), true);
    const float2 v1 = filter_vals<MODE>(a, w1, off, bin + 1, gf, bin_tab<MODE>(a, bin + 1), true);
    reinterpret_cast<float4*>(F)[q] = make_float4(v0.x, v0.y, v1.x, v1.y);
  }
}

// Filter of a run of consecutive output frames of one plane (a frame group)
// in one launch: each thread takes two neighbouring bins of one block and
// walks the run's frames in order with the bins' temporal window in
// registers, so that every window spectrum is loaded once per run (not once
// per output frame), and a Kalman state once per run. fs.spec[s] is frame
// n0 - 2 + s; frame n0 + j's window is fs.spec[j + LO .. j + HI] and its
// filtered bins go to fs.out[j]. The sharpen/dehalo pass and the inverse
// transform follow per frame (k_filter_inverse_frames<MODE_SHARPEN_ONLY> on
// fs.out[j]). Few registers and no shared memory: the SMs hold enough warps
// to cover the load latency by themselves.
template <int MODE>
__global__ void __launch_bounds__(256) k_filter_frames(InverseArgs a, const __grid_constant__ FilterFrameSet fs,
                                                     int bins_per_block) {
  constexpr int LO = win_lo<MODE>(), HI = win_hi<MODE>(), NW = HI - LO + 1;
  const size_t pairs = (size_t)a.g.nblocks * bins_per_block / 2;
  const float gs0 = __ldg(&a.t.grid[0].x);
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < pairs; q += (size_t)gridDim.x * blockDim.x) {
    const size_t e = 2 * q;
    const int bin = (int)(e % bins_per_block);
    const size_t off = e - bin;
    const BinTab tb0 = bin_tab<MODE>(a, bin), tb1 = bin_tab<MODE>(a, bin + 1);
    if constexpr (MODE == MODE_KALMAN) {
      // the state of both bins stays in registers across the run's frames
      float4 lv;
      float2 cv, cp;
      asm("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
          : "=f"(lv.x), "=f"(lv.y), "=f"(lv.z), "=f"(lv.w) : "l"(a.kal_last + e));
      asm("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(cv.x), "=f"(cv.y) : "l"(a.kal_covar + e));
      asm("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(cp.x), "=f"(cp.y) : "l"(a.kal_covarp + e));
      float2 l0 = make_float2(lv.x, lv.y), l1 = make_float2(lv.z, lv.w);
      float s0 = a.c.sigma2n_2d, s1 = a.c.sigma2n_2d;
      if (a.c.pattern) {
        s0 = fmaxf(__ldg(a.t.pattern2d + bin), 1e-15f);
        s1 = fmaxf(__ldg(a.t.pattern2d + bin + 1), 1e-15f);
      }
      for (int j = 0; j < fs.count; j++) {
        const float4 c = ld_stream4(fs.spec[j + 2] + e);
        kalman_step(a, make_float2(c.x, c.y), s0, l0, cv.x, cp.x);
        kalman_step(a, make_float2(c.z, c.w), s1, l1, cv.y, cp.y);
        reinterpret_cast<float4*>(fs.out[j])[q] = make_float4(l0.x, l0.y, l1.x, l1.y);
      }
      reinterpret_cast<float4*>(a.kal_last)[q] = make_float4(l0.x, l0.y, l1.x, l1.y);
      reinterpret_cast<float2*>(a.kal_covar)[q] = cv;
      reinterpret_cast<float2*>(a.kal_covarp)[q] = cp;
    } else {
      float4 wv[NW];
#pragma unroll
      for (int k = 0; k < NW - 1; k++) wv[k] = ld_stream4(fs.spec[LO + k] + e);
      for (int j = 0; j < fs.count; j++) {
        wv[NW - 1] = ld_stream4(fs.spec[j + HI] + e);
        const float gf = (MODE >= 1) ? a.c.degrid * __ldg(&fs.spec[j + 2][off].x) / gs0 : 0.f;
        float2 w0[5], w1[5];
#pragma unroll
        for (int k = 0; k < 5; k++) {
          const bool in = k >= LO && k <= HI;
          w0[k] = in ? make_float2(wv[k - LO].x, wv[k - LO].y) : make_float2(0.f, 0.f);
          w1[k] = in ? make_float2(wv[k - LO].z, wv[k - LO].w) : make_float2(0.f, 0.f);
        }
        const float2 v0 = filter_vals<MODE>(a, w0, off, bin, gf, tb0, false);
        const float2 v1 = filter_vals<MODE>(a, w1, off, bin + 1, gf, tb1, false);
        reinterpret_cast<float4*>(fs.out[j])[q] = make_float4(v0.x, v0.y, v1.x, v1.y);
#pragma unroll
        for (int k = 0; k < NW - 1; k++) wv[k] = wv[k + 1];
      }
    }
  }
}

// The Kalman state of two neighbouring bins: filtered values, covariances,
// process covariances (loads that do not allocate in L1: each is read once and
// written back by this thread).
struct KalmanPair {
  float4 l;
  float2 cv, cp;
  __device__ __forceinline__ void load(const InverseArgs& a, size_t at) {
    asm("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(l.x), "=f"(l.y), "=f"(l.z), "=f"(l.w) : "l"(a.kal_last + at));
    asm("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(cv.x), "=f"(cv.y) : "l"(a.kal_covar + at));
    asm("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(cp.x), "=f"(cp.y) : "l"(a.kal_covarp + at));
  }
  // (a load that the compiler keeps before the stores that follow)
  __device__ __forceinline__ void load_before_stores(const InverseArgs& a, size_t at) {
    l = *reinterpret_cast<const float4*>(a.kal_last + at);
    cv = *reinterpret_cast<const float2*>(a.kal_covar + at);
    cp = *reinterpret_cast<const float2*>(a.kal_covarp + at);
  }
  __device__ __forceinline__ void store(const InverseArgs& a, size_t at) const {
    *reinterpret_cast<float4*>(a.kal_last + at) = l;
    *reinterpret_cast<float2*>(a.kal_covar + at) = cv;
    *reinterpret_cast<float2*>(a.kal_covarp + at) = cp;
  }
  // One frame's values of the pair (bins bin, bin + 1 of the block at `off`): the filtered ones.
  __device__ __forceinline__ float4 step(const InverseArgs& a, const float4& c, size_t off, int bin) {
    float s0 = a.c.sigma2n_2d, s1 = a.c.sigma2n_2d;
    if (a.psd) {
      s0 = fmaxf(learned_noise(a, off, bin), 1e-15f);
      s1 = fmaxf(learned_noise(a, off, bin + 1), 1e-15f);
    } else if (a.c.pattern) {
      s0 = fmaxf(__ldg(a.t.pattern2d + bin), 1e-15f);
      s1 = fmaxf(__ldg(a.t.pattern2d + bin + 1), 1e-15f);
    }
    float2 l0 = make_float2(l.x, l.y), l1 = make_float2(l.z, l.w);
    kalman_step(a, make_float2(c.x, c.y), s0, l0, cv.x, cp.x);
    kalman_step(a, make_float2(c.z, c.w), s1, l1, cv.y, cp.y);
    l = make_float4(l0.x, l0.y, l1.x, l1.y);
    return l;
  }
};

// A thread's walk over the bin pairs of consecutive blocks, `STEP` pairs at a
// time: block b and first bin, kept without divisions.
template <int BINS, int STEP>
struct PairCursor {
  int b, bin;
  __device__ __forceinline__ explicit PairCursor(int pair) : b(pair / (BINS / 2)), bin(2 * (pair % (BINS / 2))) {}
  __device__ __forceinline__ void step() {
    b += 2 * STEP / BINS;
    bin += 2 * STEP % BINS;
    if (bin >= BINS) bin -= BINS, b++;
  }
};

// ---------------------------------------------------------------- inverse

// One warp filters and inverse-transforms blocks_per_warp<BW>() blocks:
//  A. every bin, consecutive bin pairs on consecutive lanes (coalesced 16-byte
//     loads of the bt spectra), through the filter and the separate
//     sharpen/dehalo pass (whose grid fraction is the filtered DC); results to
//     shared memory. Block by block, or the warp's blocks as one stream
//     (stream_blocks);
//  B. one column per lane: inverse complex DFT along y (DC and Nyquist columns
//     together: both are Hermitian, so their inverses are real);
//  C. one row per lane: c2r along x, 16-byte stores of the time-domain rows.
template <int BW, int BH>
__host__ __device__ constexpr int fft_ctas(int nblocks) {
  return (nblocks + kWarps * blocks_per_warp<BW>() - 1) / (kWarps * blocks_per_warp<BW>());
}

// Where a CTA finds its window spectra and writes its time-domain blocks:
// the launch arguments (one output frame per launch), or pointers picked for
// one frame of a frame group (k_filter_inverse_frames).
struct ArgsWin {
  const InverseArgs& a;
  __device__ __forceinline__ const float2* in(int k) const { return a.in[k]; }
  __device__ __forceinline__ float* tdom() const { return a.tdom; }
};
struct FrameWin {
  const float2* p[5];
  float* t;
  __device__ __forceinline__ const float2* in(int k) const { return p[k]; }
  __device__ __forceinline__ float* tdom() const { return t; }
};

// Blocks that a warp filters as one stream: all its blocks where single blocks
// leave many lanes idle in their last round (16 x 16: 72 pairs are three rounds,
// four blocks' 288 are nine), more of them for a window of 2 to 4 frames, whose
// rounds the stream's block index and shuffles cost more. us per frame block by
// block / as a stream: 16 x 16, 16000 blocks, bt = 5 35 / 31, bt = 1 22 / 19, bt = 3
// 25.7 / 25.9; 24 x 16, 30000 blocks, bt = 5 78 / 67, bt = 3 55 / 56, bt = 2 41 / 50.
template <int BW, int BH, int MODE>
__host__ __device__ constexpr int stream_blocks() {
  constexpr int PAIRS = BH * (BW / 2 + 1) / 2, LANES = (PAIRS + 31) / 32 * 32;
  constexpr int percent = MODE == 2 || MODE == 3 ? 65 : (MODE == 4 ? 76 : 87);
  return 100 * PAIRS < percent * LANES ? blocks_per_warp<BW>() : 1;
}

template <int BW, int BH, int MODE, class Win>
__device__ __forceinline__ void filter_inverse_cta_w(const InverseArgs& a, int vcta, const Win& win) {
  constexpr int NH = BW / 2 + 1, HC = BW / 2, NBW = blocks_per_warp<BW>(), BINS = BH * NH, PAIRS = BINS / 2;
  extern __shared__ __align__(16) float2 smem2[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2* S = smem2 + warp * NBW * BINS;
  const Geom& g = a.g;
  const int cta = a.reverse ? fft_ctas<BW, BH>(g.nblocks) - 1 - vcta : vcta;
  const int blk0 = (cta * kWarps + warp) * NBW;
  if (blk0 >= g.nblocks) return;
  const float gs0 = __ldg(&a.t.grid[0].x);
  constexpr int LO = win_lo<MODE>(), HI = win_hi<MODE>(), NW = HI - LO + 1;
  // load-pipeline depth (rounds of 32 bin pairs in flight), fewer as the
  // window (and the registers per round) grows
  constexpr int GROUP = stream_blocks<BW, BH, MODE>();
  constexpr int ROUNDS = (GROUP * PAIRS + 31) / 32;
  constexpr int DW = NW <= 1 ? (MODE == MODE_KALMAN ? 3 : 4) : (NW == 2 ? 4 : (NW == 3 ? 3 : 2));
  constexpr int D = ROUNDS < DW ? ROUNDS : DW;
#pragma unroll 1
  for (int b0 = 0; b0 < NBW; b0 += GROUP) {
    if (blk0 + b0 >= g.nblocks) break;
    const size_t off0 = (size_t)(blk0 + b0) * BINS;
    const int pairs = GROUP == 1 ? PAIRS : min(GROUP, g.nblocks - blk0 - b0) * PAIRS;
    const int rounds = GROUP == 1 ? ROUNDS : (pairs + 31) / 32;
    auto fetch = [&](int q, float4(&dst)[NW]) {  // the window of pair q
#pragma unroll
      for (int k = 0; k < NW; k++)
        dst[k] = (q < pairs && FFT3D_IN(win.in(LO + k) != nullptr && off0 + 2 * q + 1 < (size_t)g.nblocks * BINS, a.err))
                     ? ld_stream4(win.in(LO + k) + off0 + 2 * q)
                     : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto filter = [&](const float4(&in)[NW], KalmanPair& state, size_t off, int bin, float gf) {
      if constexpr (MODE == MODE_KALMAN) {
        return state.step(a, in[0], off, bin);
      } else {
        float4 w[5];
#pragma unroll
        for (int k = 0; k < 5; k++) w[k] = (k >= LO && k < LO + NW) ? in[k - LO] : make_float4(0.f, 0.f, 0.f, 0.f);
        return group_filter_one<MODE>(a, off, bin, w, gf);
      }
    };
    // software pipeline: the window (and Kalman state) of round j + D is loaded
    // while round j is filtered, so D x NW loads per lane are always in flight
    float4 buf[D][NW];
    KalmanPair kal[MODE == MODE_KALMAN ? D : 1];
#pragma unroll
    for (int j = 0; j < D; j++) {
      fetch(lane + 32 * j, buf[j]);
      if (MODE == MODE_KALMAN && lane + 32 * j < pairs) kal[j].load(a, off0 + 2 * (lane + 32 * j));
    }
    // grid fractions of the block's DC and of its filtered DC: lane b's are block b0 + b's
    float gf_mine = 0.f, gsh_mine = 0.f;
    if (lane * PAIRS < pairs) {
      if constexpr (MODE >= 1) gf_mine = a.c.degrid * __ldg(&win.in(2)[off0 + lane * BINS].x) / gs0;
      if (GROUP > 1 && a.c.do_sharpen) {
        float4 dc[NW];
        fetch(lane * PAIRS, dc);
        KalmanPair state;
        if constexpr (MODE == MODE_KALMAN) state.load_before_stores(a, off0 + lane * BINS);
        gsh_mine = a.c.degrid * filter(dc, state, off0 + lane * BINS, 0, gf_mine).x / gs0;
      }
    }
    float gf = MODE >= 1 ? __shfl_sync(0xffffffffu, gf_mine, 0) : 0.f, gsh = 0.f;
    PairCursor<BINS, 32> at(lane);
    // (D rounds to a turn of the loop: all of it unrolled is many times the
    // code, and its instruction-cache misses cost more than the loop)
#pragma unroll 1
    for (int j0 = 0; j0 < rounds; j0 += D) {
#pragma unroll
      for (int u = 0; u < D; u++) {
        const int j = j0 + u, q = lane + 32 * j;
        if (j >= rounds) break;
        const bool in = q < pairs;
        const int bin = GROUP == 1 ? 2 * q : at.bin;
        const size_t off = GROUP == 1 ? off0 : off0 + at.b * BINS;
        if constexpr (GROUP > 1) {
          if (MODE >= 1) gf = __shfl_sync(0xffffffffu, gf_mine, at.b);
          if (a.c.do_sharpen) gsh = __shfl_sync(0xffffffffu, gsh_mine, at.b);
          at.step();
        }
        float4 w[NW];
#pragma unroll
        for (int k = 0; k < NW; k++) w[k] = buf[u][k];
        KalmanPair state;
        if constexpr (MODE == MODE_KALMAN) state = kal[u];
        if (j + D < rounds) {
          fetch(q + 32 * D, buf[u]);
          if (MODE == MODE_KALMAN && q + 32 * D < pairs) kal[u].load(a, off0 + 2 * (q + 32 * D));
        }
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in) {
          v = filter(w, state, off, bin, gf);
          if constexpr (MODE == MODE_KALMAN) state.store(a, off0 + 2 * q);
        }
        if (a.c.do_sharpen) {
          // one block's filtered DC is lane 0's first bin
          if (GROUP == 1 && j == 0) gsh = a.c.degrid * __shfl_sync(0xffffffffu, v.x, 0) / gs0;
          if (in)
            v = bins_of(sharpen_pair(a, pair_of(v), pair_grid(a, bin), pair_weights(a.t.wsharpen, a.c.use_sharpen, bin),
                                     pair_weights(a.t.wdehalo, a.c.use_dehalo, bin), gsh));
        }
        if (in) *reinterpret_cast<float4*>(S + b0 * BINS + 2 * q) = v;
      }
    }
  }
  __syncwarp();
  for (int t = lane; t < NBW * HC; t += 32) {
    const int b = t / HC, c = t - b * HC;
    if (blk0 + b < g.nblocks) inv_col<BW, BH>(S + b * BINS, c);
  }
  __syncwarp();
  for (int t = lane; t < NBW * BH; t += 32) {
    const int b = t / BH, y = t - b * BH;
    if (blk0 + b < g.nblocks) inv_row_inplace<BW, BH>(S + b * BINS, y);
  }
  __syncwarp();
  for (int b = 0; b < NBW && blk0 + b < g.nblocks; b++)
    if (FFT3D_IN(win.tdom() != nullptr, a.err)) store_tdom<BW, BH>(S + b * BINS, win.tdom() + (size_t)(blk0 + b) * BH * BW, lane);
  __syncwarp();  // S is reused by the warp's next work item
}

template <int BW, int BH, int MODE>
__device__ __forceinline__ void filter_inverse_cta(const InverseArgs& a, int vcta) {
  filter_inverse_cta_w<BW, BH, MODE, ArgsWin>(a, vcta, ArgsWin{a});
}

// Several consecutive output frames of one plane in one launch (a frame
// group). CTA x works on frame x % count, CTA-of-frame x / count: the
// resident CTAs of all the group's frames cover the same blocks at the same
// time, so a window spectrum shared by up to bt frames is read from HBM once
// and then hit in L2. The frames differ only in their window spectra and
// time-domain buffers (fs); everything else is in a.
template <int BW, int BH, int MODE>
__global__ void __launch_bounds__(kWarps * 32) k_filter_inverse_frames(InverseArgs a, FrameSet fs) {
  const int j = blockIdx.x % fs.count, c = blockIdx.x / fs.count;
  // the frame's pointers, selected with constant indices (a dynamic index
  // into the parameter space would copy it to local memory)
  FrameWin w;
#pragma unroll
  for (int k = 0; k < 5; k++) w.p[k] = nullptr;
  w.t = nullptr;
#pragma unroll
  for (int q = 0; q < kMaxGroupFrames; q++)
    if (q == j) {
#pragma unroll
      for (int k = 0; k < 5; k++) w.p[k] = fs.in[q][k];
      w.t = fs.tdom[q];
    }
  filter_inverse_cta_w<BW, BH, MODE, FrameWin>(a, c, w);
}

// CTAs per SM of k_filter_inverse: 6 at 80 registers where that spills little
// (24 x 16 blocks, bt = 2, 16000 of them: 29 us at 5, 24 at 6; 32 x 32, bt = 3, 8000:
// 39 at 5, 52 at 6).
template <int BH, int MODE>
__host__ __device__ constexpr int inv_ctas() { return (MODE == 2 || MODE == 3) && BH <= 16 ? 6 : 5; }

template <int BW, int BH, int MODE>
__global__ void __launch_bounds__(kWarps * 32, ctas_for(inv_ctas<BH, MODE>(), kWarps * fft_smem_bytes<BW, BH>()))
    k_filter_inverse(InverseArgs a) {
  filter_inverse_cta<BW, BH, MODE>(a, blockIdx.x);
}

// The work item's arguments are staged in shared memory: the body's global
// stores cannot alias them (a reference into global memory would be reloaded
// after every store), and unlike a by-value copy they cost no registers.
template <int BW, int BH, int MODE>
__global__ void __launch_bounds__(kWarps * 32) k_filter_inverse_batch(const InverseArgs* __restrict__ args,
                                                                     const int2* __restrict__ items, int nitems) {
  __shared__ __align__(16) InverseArgs sa;
  static_assert(sizeof(InverseArgs) % 4 == 0, "word copy");
  for (int i = blockIdx.x; i < nitems; i += gridDim.x) {
    const int2 it = items[i];
    __syncthreads();  // every warp is done with the previous item's arguments
    const int* src = reinterpret_cast<const int*>(args + it.x);
    int* dst = reinterpret_cast<int*>(&sa);
    for (int w = threadIdx.x; w < (int)(sizeof(InverseArgs) / 4); w += blockDim.x) dst[w] = src[w];
    __syncthreads();
    filter_inverse_cta<BW, BH, MODE>(sa, it.y);
  }
}

// ---------------------------------------------------------------- overlap-add pixels

// Time-domain block reads of the overlap-add. Blocks written by an earlier
// launch go through the read-only path without L1 allocation (each value is
// read once; the synthesis windows stay in L1). Blocks written by other CTAs
// of the same launch (L2 = true, the fused overlap-add of a frame group) are
// read at L2, the point where those CTAs' stores are visible.
template <bool L2>
__device__ __forceinline__ float ld_tdom(const float* p) {
  if constexpr (L2) return __ldcg(p);
  else return __ldg(p);
}
template <bool L2>
__device__ __forceinline__ float4 ld_tdom4(const float* p) {
  if constexpr (L2) {
    return __ldcg(reinterpret_cast<const float4*>(p));
  } else {
    float4 q;
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w)
        : "l"(p));
    return q;
  }
}

// Four samples, as one store.
template <typename T>
struct Pack4;
template <>
struct Pack4<uint8_t> {
  using V = uchar4;
};
template <>
struct Pack4<uint16_t> {
  using V = ushort4;
};
template <>
struct Pack4<float> {
  using V = float4;
};

template <typename T>
__device__ __forceinline__ T clamp_sample(float v, int maxval) {
  if constexpr (sizeof(T) == 4) {
    float c = v < 0.f ? 0.f : v;
    return c > 1.f ? 1.f : c;
  } else {
    int i = __float2int_rz(v);
    i = i < 0 ? 0 : (i > maxval ? maxval : i);
    return (T)i;
  }
}

// V adjacent pixels (V = 1, 2 or 4) of the processed region from column x0 on
// that share their blocks and overlap case and go out in one store: what they
// share along x ...
template <int V>
struct OlaColumn {
  int bx, x;  // block column, position inside the block step
  bool xov;
  float sxr[V], sxl[V];  // synthesis windows
  __device__ __forceinline__ OlaColumn(const OlaArgs& a, int x0) {
    const int X = a.g.sx + x0;
    bx = div_small(X, a.g.sx);
    x = X - bx * a.g.sx;
    xov = x < a.g.ow;
#pragma unroll
    for (int i = 0; i < V; i++) {
      sxr[i] = xov ? __ldg(a.t.wsyn_xr + x + i) : 0.f;
      sxl[i] = xov ? __ldg(a.t.wsyn_xl + x + i) : 0.f;
    }
  }
};
// ... and those pixels of row k: the (at most four) blocks covering them,
// weighted with the synthesis windows and the FFT normalisation in the
// association order of src/buffer.cpp:399-559, with its fused multiply-adds
// written out, so that every width rounds alike. Truncation toward zero, then
// the clamp (src/buffer.cpp:397-406).
template <typename T, int V, bool L2>
__device__ __forceinline__ void ola_pixels(const OlaArgs& a, const OlaColumn<V>& q, const float* tdom, void* dst,
                                           long long stride, int x0, int k) {
  const Geom& g = a.g;
  const int bw = g.bw, bh = g.bh, bx = q.bx, x = q.x;
  const float norm = a.norm;
  const int Y = g.sy + k, by = div_small(Y, g.sy), y = Y - by * g.sy;
  const bool yov = y < g.oh;
  auto at = [&](int bxx, int byy, int yy, int xx, float (&v)[V]) {
    if (!FFT3D_IN(bxx >= 0 && bxx < g.nox && byy >= 0 && byy < g.noy && yy >= 0 && yy < bh && xx >= 0 && xx + V <= bw,
                  a.err)) {
#pragma unroll
      for (int i = 0; i < V; i++) v[i] = 0.f;
      return;
    }
    const float* p = tdom + ((size_t)(byy * g.nox + bxx) * bh + yy) * bw + xx;
    if constexpr (V == 4) {
      const float4 u = ld_tdom4<L2>(p);
      v[0] = u.x, v[1] = u.y, v[2] = u.z, v[3] = u.w;
    } else if constexpr (V == 2) {
      if constexpr (L2) {
        const float2 u = __ldcg(reinterpret_cast<const float2*>(p));
        v[0] = u.x, v[1] = u.y;
      } else {
        asm("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(p));
      }
    } else {
      v[0] = ld_tdom<L2>(p);
    }
  };
  float v[V], aa[V], b[V], c[V], d[V];
  at(bx, by, y, x, d);
  if (q.xov) at(bx - 1, by, y, x + g.sx, c);
  if (!yov) {
#pragma unroll
    for (int i = 0; i < V; i++) {
      const float t = q.xov ? fmaf(c[i], q.sxr[i], __fmul_rn(d[i], q.sxl[i])) : d[i];
      v[i] = fmaf(t, norm, a.rounder) + a.base;
    }
  } else {
    at(bx, by - 1, y + g.sy, x, b);
    if (q.xov) at(bx - 1, by - 1, y + g.sy, x + g.sx, aa);
    const float wr = __fmul_rn(__ldg(a.t.wsyn_yr + y), norm), wl = __fmul_rn(__ldg(a.t.wsyn_yl + y), norm);
#pragma unroll
    for (int i = 0; i < V; i++) {
      const float u = q.xov ? fmaf(aa[i], q.sxr[i], __fmul_rn(b[i], q.sxl[i])) : b[i];
      const float t = q.xov ? fmaf(c[i], q.sxr[i], __fmul_rn(d[i], q.sxl[i])) : d[i];
      v[i] = fmaf(u, wr, __fmul_rn(t, wl)) + a.rounder + a.base;
    }
  }
  const int fr = field_row(k, g.H, g.interlaced);
  if (!FFT3D_IN(fr >= 0 && fr < g.H && x0 + V <= g.W, a.err)) return;
  T o[V];
#pragma unroll
  for (int i = 0; i < V; i++) o[i] = clamp_sample<T>(v[i], a.maxval);
  T* px = reinterpret_cast<T*>(static_cast<char*>(dst) + (long long)fr * stride) + x0;
  if constexpr (V == 4) {
    typename Pack4<T>::V w;
    w.x = o[0], w.y = o[1], w.z = o[2], w.w = o[3];
    *reinterpret_cast<typename Pack4<T>::V*>(px) = w;
  } else if constexpr (V == 2) {
    if constexpr (sizeof(T) == 1) *reinterpret_cast<uchar2*>(px) = make_uchar2(o[0], o[1]);
    else if constexpr (sizeof(T) == 2) *reinterpret_cast<ushort2*>(px) = make_ushort2(o[0], o[1]);
    else *reinterpret_cast<float2*>(px) = make_float2(o[0], o[1]);
  } else {
    *px = o[0];
  }
}

// ---------------------------------------------------------------- bulk copies

constexpr int kBulkSpin = 1 << 22;  // bounded mbarrier wait (then error flag 2)

__device__ __forceinline__ bool bulk_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done = 0;
  for (int it = 0; it < kBulkSpin && !done; it++)
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
  return done != 0;
}

// One mbarrier for one arrival, made ready for the CTA's bulk copies.
__device__ __forceinline__ void bulk_init(uint64_t* bar) {
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}

// ---------------------------------------------------------------- runs of frames, a few blocks per CTA

// Spectrum tiles one CTA of k_filter_inverse_group works on (blocks x frames
// of the run): as many as its 128 threads have columns for in one round of
// the column transforms, within 36 KB, and at least the longest run's frames
// (staged runs add their window's extra ones, run_tiles; run_ctas says how many
// CTAs then reside per SM).
template <int BW, int BH>
__host__ __device__ constexpr int group_tiles() {
  const int lanes = kWarps * 32 / (BW / 2), fit = 36 * 1024 / (BH * (BW / 2 + 1) * 8);
  const int t = lanes < fit ? lanes : fit, run = group_run_frames(BW, BH);
  return t > run ? t : run;
}
// Two grid fractions per tile, in front of the tiles (16-byte aligned).
template <int BW, int BH>
__host__ __device__ constexpr int group_head_floats() { return (2 * group_tiles<BW, BH>() + 3) / 4 * 4; }
// Dynamic shared memory of k_filter_inverse_group.
template <int BW, int BH>
__host__ __device__ constexpr int group_smem_bytes(int tiles) {
  return group_head_floats<BW, BH>() * 4 + tiles * BH * (BW / 2 + 1) * 8;
}

// A run's window spectrum s, bins bin and bin + 1 of the block at `off`
// (checked build: the spectrum exists and the pair lies in the plane).
__device__ __forceinline__ float4 group_load(const InverseArgs& a, const TemporalSet& ts, int s, size_t off, int bin) {
  if (!FFT3D_IN(s >= 0 && s < kGroupTile + 4 && ts.spec[s] != nullptr &&
                    off + bin + 1 < (size_t)a.g.nblocks * a.g.bh * a.g.nh,
                a.err))
    return make_float4(0.f, 0.f, 0.f, 0.f);
  return ld_stream4(ts.spec[s] + off + bin);
}

// Bins bin, bin + 1 of the block at `off` through all the run's frames, in
// order: Wiener 3D with the window of MODE frames in registers (each spectrum
// read once, the next frame's bins loaded one frame ahead) and the separate
// sharpen/dehalo pass, or Kalman with the state in registers. load(s): the
// pair in the run's window spectrum s; gfs, gsh: the grid fractions of the
// block's first frame, before and after the filter, tile: the pair's place in
// its tile; all `stride` tiles apart from frame to frame.
template <int MODE, int BINS, class Load>
__device__ __forceinline__ void group_filter_pair(const InverseArgs& a, size_t off, int bin, int count,
                                                  const float* gfs, const float* gsh, float2* tile, int stride,
                                                  const Load& load) {
  if constexpr (MODE == MODE_KALMAN) {
    float4 lv;
    float2 cv, cp;
    asm("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(lv.x), "=f"(lv.y), "=f"(lv.z), "=f"(lv.w) : "l"(a.kal_last + off + bin));
    asm("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(cv.x), "=f"(cv.y) : "l"(a.kal_covar + off + bin));
    asm("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(cp.x), "=f"(cp.y) : "l"(a.kal_covarp + off + bin));
    float2 l0 = make_float2(lv.x, lv.y), l1 = make_float2(lv.z, lv.w);
    float s0 = a.c.sigma2n_2d, s1 = a.c.sigma2n_2d;
    if (a.psd) {
      s0 = fmaxf(learned_noise(a, off, bin), 1e-15f);
      s1 = fmaxf(learned_noise(a, off, bin + 1), 1e-15f);
    } else if (a.c.pattern) {
      s0 = fmaxf(__ldg(a.t.pattern2d + bin), 1e-15f);
      s1 = fmaxf(__ldg(a.t.pattern2d + bin + 1), 1e-15f);
    }
    float4 nxt = load(2);
    for (int j = 0; j < count; j++) {
      const float4 c = nxt;
      if (j + 1 < count) nxt = load(j + 3);
      kalman_step(a, make_float2(c.x, c.y), s0, l0, cv.x, cp.x);
      kalman_step(a, make_float2(c.z, c.w), s1, l1, cv.y, cp.y);
      *reinterpret_cast<float4*>(tile + j * stride * BINS) = make_float4(l0.x, l0.y, l1.x, l1.y);
    }
    *reinterpret_cast<float4*>(a.kal_last + off + bin) = make_float4(l0.x, l0.y, l1.x, l1.y);
    *reinterpret_cast<float2*>(a.kal_covar + off + bin) = cv;
    *reinterpret_cast<float2*>(a.kal_covarp + off + bin) = cp;
  } else if constexpr (MODE >= 2) {
    constexpr int LO = win_lo<MODE>(), HI = win_hi<MODE>(), NW = HI - LO + 1;
    const Pair grid = pair_grid(a, bin);
    const f2x nn = pair_noise<MODE>(a, off, bin);
    const bool sh = a.c.do_sharpen;
    const f2x wsh = pair_weights(a.t.wsharpen, sh && a.c.use_sharpen, bin),
              wdh = pair_weights(a.t.wdehalo, sh && a.c.use_dehalo, bin);
    // spectrum s (frame n0 - 2 + s) lives in r[s % NW]; frame j reads
    // s = j + LO .. j + HI; with j = j0 + u and j0 a multiple of NW every
    // index below is a compile-time constant
    Pair r[NW];
#pragma unroll
    for (int k = 0; k < NW - 1; k++) r[(LO + k) % NW] = pair_of(load(LO + k));
    float4 nxt = load(HI);
    // (left by a return from inside the unrolled steps: with a condition around
    // each step the window's registers are moved at every join)
    for (int j = 0;;) {
#pragma unroll
      for (int u = 0; u < NW; u++) {
        r[(u + HI) % NW] = pair_of(nxt);
        if (j + 1 < count) nxt = load(j + 1 + HI);
        Pair w[5];
#pragma unroll
        for (int k = 0; k < 5; k++) w[k] = r[(u + (k >= LO && k <= HI ? k : LO)) % NW];
        Pair v = filter_pair<MODE>(w, grid, gfs[j * stride], nn, a.c.lowlimit);
        if (a.c.do_sharpen) v = sharpen_pair(a, v, grid, wsh, wdh, gsh[j * stride]);
        *reinterpret_cast<float4*>(tile + j * stride * BINS) = bins_of(v);
        if (++j == count) return;
      }
    }
  }
}

// The overlap-add of output tile (tx, ty) (OlaFuse) for the run's frames, V
// pixels per thread, the blocks read from L2.
template <typename T, int V>
__device__ __forceinline__ void group_ola_tile_v(const OlaFuse& of, const TemporalSet& ts, int count, int tx, int ty) {
  const Geom& g = of.o.g;
  const int x_lo = (tx - 1) * g.sx, y_lo = (ty - 1) * g.sy;
  const int wd = min(g.sx, g.W - x_lo) / V, ht = min(g.sy, g.H - y_lo);
  // (V divides the step and the width: wd is exact)
  const int per = wd * ht;
  for (int i = threadIdx.x; i < count * per; i += blockDim.x) {
    const int j = i / per, r = i - j * per, yy = r / wd, x0 = x_lo + V * (r - yy * wd);
    ola_pixels<T, V, true>(of.o, OlaColumn<V>(of.o, x0), ts.tdom[j], of.dst[j], of.dst_stride[j], x0, y_lo + yy);
  }
}
template <typename T>
__device__ __noinline__ void group_ola_tile(const OlaFuse& of, const TemporalSet& ts, int count, int tx, int ty) {
  if (of.px == 4) group_ola_tile_v<T, 4>(of, ts, count, tx, ty);
  else if (of.px == 2) group_ola_tile_v<T, 2>(of, ts, count, tx, ty);
  else group_ola_tile_v<T, 1>(of, ts, count, tx, ty);
}

// Window spectra beyond the run's own frames that a staged run keeps in shared memory.
template <int MODE>
__host__ __device__ constexpr int win_extra() { return MODE >= 2 ? win_hi<MODE>() - win_lo<MODE>() : 0; }
// Whether runs of this block size and mode fetch their window spectra by bulk
// copies into their tiles: where the longest run's tiles and its window's
// extra ones still let 4 CTAs reside per SM.
template <int BW, int BH, int MODE>
__host__ __device__ constexpr bool run_staged() {
  return ctas_for(4, group_smem_bytes<BW, BH>(group_run_frames(BW, BH) + win_extra<MODE>())) >= 4;
}
// Tiles of shared memory of a CTA, and the CTAs per SM its kernel is compiled for.
template <int BW, int BH, int MODE, bool STAGED>
__host__ __device__ constexpr int run_tiles() {
  const int most = group_run_frames(BW, BH) + win_extra<MODE>();
  return STAGED && most > group_tiles<BW, BH>() ? most : group_tiles<BW, BH>();
}
template <int BW, int BH, int MODE, bool STAGED>
__host__ __device__ constexpr int run_ctas(int extra) {
  return ctas_for(STAGED && MODE >= 2 ? kWalkCtas : kShortCtas,
                  group_smem_bytes<BW, BH>(run_tiles<BW, BH, MODE, STAGED>()) + extra);
}

// A run of count <= kGroupTile consecutive output frames of one plane with
// one mode; CTA `cta` takes ts.nb consecutive blocks, so it makes count x
// ts.nb spectrum tiles in shared memory (tile j * blocks + b: frame j of block
// b). Each stage is spread over the whole CTA, with a barrier between stages:
//  0. STAGED: one bulk copy per window spectrum brings its blocks into the
//     tiles (the window's spectra beyond the run's frames into extra tiles);
//     the filter then works in place, since frame j's window begins with the
//     spectrum whose tile it overwrites and one thread takes a pair through
//     all frames. Otherwise the filter reads the spectra from global memory;
//  1. the grid fractions of each tile (its block's DC in its frame, and that
//     DC filtered, for the sharpen pass), then the filter with the separate
//     sharpen/dehalo pass. Wiener 3D runs of 2 frames and more, and Kalman:
//     each thread takes two neighbouring bins and walks the run's frames in
//     order, its window in registers, so that each of the block's count +
//     MODE - 1 window spectra is read once for the run (and a Kalman state
//     once); pairs beyond the last whole round of the CTA's threads, and all
//     pairs of shorter or window-less runs, are spread over all threads as
//     single (pair, frame) items;
//  2. Kalman only: the sharpen/dehalo pass, once the filtered DCs are known;
//  3. the inverse column DFTs of every tile (DC and Nyquist columns as one
//     complex transform), 4. the c2r rows, 5. coalesced stores of the
//     time-domain blocks.
// bar: an initialised mbarrier (STAGED), whose parity is `phase`. False when
// the bounded wait on it ran out (the whole CTA then leaves). NEWEST (one
// frame, not staged): the window's newest spectrum is not read from the window
// but from the tiles, where k_frame's forward transform left it.
template <int BW, int BH, int MODE, bool STAGED, bool NEWEST = false>
__device__ __forceinline__ bool filter_inverse_group_cta(const InverseArgs& a, const TemporalSet& ts, int cta,
                                                         uint64_t* bar, uint32_t phase, const OlaFuse* of = nullptr) {
  constexpr int NH = BW / 2 + 1, HC = BW / 2, BINS = BH * NH, PAIRS = BINS / 2, NT = kWarps * 32;
  constexpr int LO = win_lo<MODE>(), HI = win_hi<MODE>();
  static_assert(BINS % 2 == 0, "bin pairs");
  extern __shared__ __align__(16) float2 smem2[];
  float* gfs = reinterpret_cast<float*>(smem2);  // grid fraction of each tile's block
  float* gsh = gfs + group_tiles<BW, BH>();      // ... and of its filtered block (sharpen pass)
  float2* S = smem2 + group_head_floats<BW, BH>() / 2;  // [tile][BINS], 16-byte aligned
  const int count = ts.count;
  const int blk0 = cta * ts.nb, nbv = min(ts.nb, a.g.nblocks - blk0);
  if (nbv <= 0) return true;
  const int tiles = nbv * count, npairs = nbv * PAIRS;
  const size_t off0 = (size_t)blk0 * BINS;
  const float gs0 = __ldg(&a.t.grid[0].x);
  const int t = threadIdx.x;
  bool landed = true;
  if constexpr (STAGED) {
    const int slots = count + win_extra<MODE>();
    const uint32_t bytes = (uint32_t)nbv * BINS * 8;
    auto there = [&](int k) { return FFT3D_IN(ts.spec[LO + k] != nullptr && blk0 + nbv <= a.g.nblocks, a.err); };
    if (t == 0) {
      uint32_t total = 0;
      for (int k = 0; k < slots; k++) total += there(k) ? bytes : 0;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(total) : "memory");
      for (int k = 0; k < slots; k++)
        if (there(k))
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                  smem_addr(S + k * nbv * BINS)),
              "l"(ts.spec[LO + k] + off0), "r"(bytes), "r"(smem_addr(bar))
              : "memory");
    }
    landed = bulk_wait(bar, phase);
  }
  auto load = [&](int s, int b, int bin) {
    if constexpr (STAGED) return *reinterpret_cast<const float4*>(S + ((s - LO) * nbv + b) * BINS + bin);
    else if (NEWEST && s == HI) return *reinterpret_cast<const float4*>(S + b * BINS + bin);
    else return group_load(a, ts, s, off0 + b * BINS, bin);
  };
  constexpr bool WALK = MODE == MODE_KALMAN || MODE >= 2;
  const bool walk = MODE == MODE_KALMAN || (MODE >= 2 && count > 1);
  int full = walk ? npairs : 0;
  if (MODE >= 2 && walk && (npairs % NT) * count <= NT) full = npairs / NT * NT;
  auto finish = [&](float4 v, int bin, float gf) {  // the separate sharpen/dehalo pass, src/code_impl/Sharpen.cpp:13-63
    if (MODE != MODE_KALMAN && a.c.do_sharpen)
      v = bins_of(sharpen_pair(a, pair_of(v), pair_grid(a, bin), pair_weights(a.t.wsharpen, a.c.use_sharpen, bin),
                               pair_weights(a.t.wdehalo, a.c.use_dehalo, bin), gf));
    return v;
  };
  // 1. pass 0: a thread per tile, bins 0 and 1: the tile's grid fraction (its
  //    DC) and, for the sharpen pass, the filtered DC's. Pass 1: a thread per
  //    pair and frame of the pairs left after the whole rounds of a walk,
  //    read before the barrier (no tile is overwritten yet), filtered after
  float4 r[5];
  if constexpr (MODE != MODE_KALMAN) {
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
      const int rest = pass == 0 ? nbv : (walk ? npairs - full : 0);
      const bool item = t < rest * count;
      int j = 0, p = 0;
      if (item) {
        j = div_small(t, rest);
        p = t - j * rest;
        p = pass == 0 ? p * PAIRS : full + p;
      }
      const int b = p / PAIRS, bin = 2 * (p - b * PAIRS), tile = j * nbv + b;
      if (item && landed) {
#pragma unroll
        for (int k = LO; k <= HI; k++) r[k] = load(j + k, b, bin);
      }
      if (pass == 1) {
        if constexpr (STAGED) {
          if (__syncthreads_or(landed ? 0 : 1)) {
            // the copies never completed: flag it, give them one more bounded
            // wait (they target this CTA's shared memory), and stop
            if (t == 0 && a.err) atomicOr(a.err, 2);
            bulk_wait(bar, phase);
            return false;
          }
        } else {
          __syncthreads();
        }
      }
      if (item && landed) {
        const float gf = pass == 0 ? a.c.degrid * r[2].x / gs0 : gfs[tile];
        if (pass == 1 || a.c.do_sharpen) {
          const float4 v = group_filter_one<MODE>(a, off0 + b * BINS, bin, r, gf);
          if (pass == 0) gsh[tile] = a.c.degrid * v.x / gs0;
          else *reinterpret_cast<float4*>(S + tile * BINS + bin) = finish(v, bin, gsh[tile]);
        }
        if (pass == 0) gfs[tile] = gf;
      }
    }
  } else if constexpr (STAGED) {
    if (__syncthreads_or(landed ? 0 : 1)) {
      if (t == 0 && a.err) atomicOr(a.err, 2);
      bulk_wait(bar, phase);
      return false;
    }
  } else if constexpr (NEWEST) {
    __syncthreads();  // the tiles' copies to the ring are done
  }
  using Cursor = PairCursor<BINS, NT>;
  if constexpr (WALK) {
    Cursor c(t);
    for (int q = t; q < full; q += NT, c.step()) {
      const int b = c.b, bin = c.bin;
      group_filter_pair<MODE, BINS>(a, off0 + b * BINS, bin, count, gfs + b, gsh + b, S + 2 * q, nbv,
                                    [&](int s) { return load(s, b, bin); });
      if (MODE == MODE_KALMAN && a.c.do_sharpen && bin == 0)
        for (int j = 0; j < count; j++) gsh[j * nbv + b] = a.c.degrid * S[(j * nbv + b) * BINS].x / gs0;
    }
  }
  if (!walk) {  // single (pair, frame) items, tile after tile, the next one's window loaded ahead
    if constexpr (MODE != MODE_KALMAN) {
      // (c.b counts tiles: frame cj, block c.b - cj * nbv)
      Cursor c(t);
      int cj = 0;
      while (c.b >= (cj + 1) * nbv) cj++;
      float4 nx[5];
      auto fetch = [&]() {
#pragma unroll
        for (int k = LO; k <= HI; k++) nx[k] = load(cj + k, c.b - cj * nbv, c.bin);
      };
      const int total = tiles * PAIRS;
      if (t < total) fetch();
      for (int q = t; q < total; q += NT) {
        const int tile = c.b, bin = c.bin, b = tile - cj * nbv;
#pragma unroll
        for (int k = LO; k <= HI; k++) r[k] = nx[k];
        c.step();
        while (c.b >= (cj + 1) * nbv) cj++;
        if (q + NT < total) fetch();
        const float4 v = group_filter_one<MODE>(a, off0 + b * BINS, bin, r, MODE >= 1 ? gfs[tile] : 0.f);
        *reinterpret_cast<float4*>(S + tile * BINS + bin) = finish(v, bin, a.c.do_sharpen ? gsh[tile] : 0.f);
      }
    }
  }
  __syncthreads();
  // 2. Kalman's sharpen/dehalo pass (its filtered DCs are known only now)
  if (MODE == MODE_KALMAN && a.c.do_sharpen) {
    Cursor c(t);
    for (int q = t; q < npairs; q += NT, c.step()) {
      const Pair grid = pair_grid(a, c.bin);
      const f2x wsh = pair_weights(a.t.wsharpen, a.c.use_sharpen, c.bin),
                wdh = pair_weights(a.t.wdehalo, a.c.use_dehalo, c.bin);
      for (int j = 0; j < count; j++) {
        float4* at = reinterpret_cast<float4*>(S + j * nbv * BINS + 2 * q);
        *at = bins_of(sharpen_pair(a, pair_of(*at), grid, wsh, wdh, gsh[j * nbv + c.b]));
      }
    }
    __syncthreads();
  }
  // 3. inverse column DFTs
  for (int i = t; i < tiles * HC; i += NT) {
    const int k = i / HC;
    inv_col<BW, BH>(S + k * BINS, i - k * HC);
  }
  __syncthreads();
  // 4. c2r rows, in place
  for (int i = t; i < tiles * BH; i += NT) {
    const int k = i / BH;
    inv_row_inplace<BW, BH>(S + k * BINS, i - k * BH);
  }
  __syncthreads();
  // 5. time-domain blocks (rows of BW floats, left in the tiles with a pitch of NH complex)
  constexpr int HALF = BW / 2;
  for (int j = 0, k = 0; j < count; j++)
    for (int b = 0; b < nbv; b++, k++) {
      float2* o = reinterpret_cast<float2*>(ts.tdom[j] + (size_t)(blk0 + b) * BH * BW);
      if (!FFT3D_IN(ts.tdom[j] != nullptr && blk0 + b < a.g.nblocks, a.err)) continue;
      for (int r = t; r < BH * HALF; r += NT) {
        const int y = r / HALF, x = r - y * HALF;
        o[r] = S[k * BINS + y * NH + x];
      }
    }
  // 6. the overlap-adds of the output tiles whose last block this is (OlaFuse,
  //    one block per CTA): release (a barrier after the stores, then a fence
  //    before each tile arrival), acquire (a fence after the arrival that
  //    completes a tile, then a barrier); no waiting
  if (of) {
    const int blk = blk0;
    __shared__ int done[4];
    __syncthreads();  // the CTA's stores precede the arrivals below (the fence there is cumulative)
    const int bx = blk % a.g.nox, by = blk / a.g.nox;
    if (t < 4) {
      const int dx = t & 1, dy = t >> 1, tx = bx + dx, ty = by + dy;
      const unsigned need = (a.g.ow > 0 ? 2u : 1u) * (a.g.oh > 0 ? 2u : 1u);
      int last = 0;
      if ((dx == 0 || a.g.ow > 0) && (dy == 0 || a.g.oh > 0) && tx >= 1 && tx <= of->tiles_x && ty >= 1 &&
          ty <= of->tiles_y && FFT3D_IN(tx < a.g.nox && ty < a.g.noy, a.err)) {
        __threadfence();
        last = atomicAdd(of->cnt + ty * a.g.nox + tx, 1u) + 1u == need;
        if (last) {
          of->cnt[ty * a.g.nox + tx] = 0;  // ready for the next launch, a graph's replay too
          __threadfence();
        }
      }
      done[t] = last;
    }
    __syncthreads();
    for (int q = 0; q < 4; q++) {
      if (!done[q]) continue;
      const int tx = bx + (q & 1), ty = by + (q >> 1);
      if (of->bytes == 1) group_ola_tile<uint8_t>(*of, ts, count, tx, ty);
      else if (of->bytes == 2) group_ola_tile<uint16_t>(*of, ts, count, tx, ty);
      else group_ola_tile<float>(*of, ts, count, tx, ty);
    }
  }
  return true;
}

template <int BW, int BH, int MODE, bool STAGED>
__global__ void __launch_bounds__(kWarps * 32, run_ctas<BW, BH, MODE, STAGED>(0))
    k_filter_inverse_group(InverseArgs a, const __grid_constant__ TemporalSet ts, const __grid_constant__ OlaFuse of) {
  __shared__ uint64_t bar;
  if constexpr (STAGED) bulk_init(&bar);
  filter_inverse_group_cta<BW, BH, MODE, STAGED>(a, ts, a.reverse ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x,
                                                 &bar, 0, of.cnt ? &of : nullptr);
}

// Batched runs of many planes: work item (run, CTA of that run). The
// run's arguments are staged in shared memory behind the tiles, so the body's
// stores cannot alias them (a reference into global memory would be reloaded
// after every store) and they cost no registers.
template <int BW, int BH, int MODE>
__global__ void __launch_bounds__(kWarps * 32, run_ctas<BW, BH, MODE, run_staged<BW, BH, MODE>()>((int)sizeof(GroupRun)))
    k_filter_inverse_group_batch(const GroupRun* __restrict__ runs, const int2* __restrict__ items, int nitems) {
  constexpr bool STAGED = run_staged<BW, BH, MODE>();
  extern __shared__ __align__(16) float2 smem2[];
  __shared__ uint64_t bar;
  GroupRun* sr = reinterpret_cast<GroupRun*>(reinterpret_cast<char*>(smem2) +
                                             group_smem_bytes<BW, BH>(run_tiles<BW, BH, MODE, STAGED>()));
  static_assert(sizeof(GroupRun) % 4 == 0, "word copy");
  if constexpr (STAGED) bulk_init(&bar);
  uint32_t phase = 0;
  for (int i = blockIdx.x; i < nitems; i += gridDim.x) {
    const int2 it = items[i];
    __syncthreads();  // every thread is done with the previous item's arguments and tiles
    const int* src = reinterpret_cast<const int*>(runs + it.x);
    int* dst = reinterpret_cast<int*>(sr);
    for (int w = threadIdx.x; w < (int)(sizeof(GroupRun) / 4); w += blockDim.x) dst[w] = src[w];
    __syncthreads();
    if (!filter_inverse_group_cta<BW, BH, MODE, STAGED>(sr->a, sr->ts, it.y, &bar, phase)) return;
    phase ^= 1;
  }
}

// ---------------------------------------------------------------- inverse (bulk-staged)

constexpr int kBulkWarps = 4;
template <int BW, int BH, int MODE>
__host__ __device__ constexpr int bulk_warp_bytes() {
  return (win_hi<MODE>() - win_lo<MODE>() + 2) * BH * (BW / 2 + 1) * 8;
}

// Filter + inverse with the window's spectra fetched by bulk copies: each
// warp walks its blocks (block = warp index + k * all warps, or mirrored for
// the reverse order) with a stage holding the block's window spectra (one
// contiguous BH x NH run per frame, one cp.async.bulk each, completing on
// the warp's mbarrier). The filter reads the stage and writes the block's
// filtered spectrum to S; lane 0 then refills the stage with the next
// block's spectra, which land while the warp runs the inverse transform of S
// and stores the time-domain block. Wiener and sharpen-only modes.
template <int BW, int BH, int MODE>
__global__ void __launch_bounds__(kBulkWarps * 32) k_filter_inverse_bulk(InverseArgs a) {
  constexpr int NH = BW / 2 + 1, HC = BW / 2, BINS = BH * NH, PER = (BINS + 31) / 32;
  constexpr int LO = win_lo<MODE>(), NW = win_hi<MODE>() - win_lo<MODE>() + 1;
  constexpr uint32_t SPEC_BYTES = BINS * 8;
  static_assert(SPEC_BYTES % 16 == 0, "bulk copies move multiples of 16 bytes");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2* stage = reinterpret_cast<float2*>(smem_raw + 128 + (size_t)warp * bulk_warp_bytes<BW, BH, MODE>());
  float2* S = stage + NW * BINS;
  uint64_t* bar = bars + warp;
  const Geom& g = a.g;
  const int nwarps = gridDim.x * kBulkWarps;
  const int first = blockIdx.x * kBulkWarps + warp;
  if (first >= g.nblocks) return;
  auto block_of = [&](int idx) { return a.reverse ? g.nblocks - 1 - idx : idx; };
  auto fetch = [&](int blk) {  // lane 0
    const size_t off = (size_t)blk * BINS;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(NW * SPEC_BYTES)
                 : "memory");
#pragma unroll
    for (int k = 0; k < NW; k++)
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              smem_addr(stage + k * BINS)),
          "l"(a.in[LO + k] + off), "r"(SPEC_BYTES), "r"(smem_addr(bar))
          : "memory");
  };
  if (lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fetch(block_of(first));
  }
  __syncwarp();
  const float gs0 = __ldg(&a.t.grid[0].x);
  uint32_t phase = 0;
  for (int idx = first; idx < g.nblocks; idx += nwarps) {
    const int blk = block_of(idx);
    if (!__all_sync(0xffffffffu, bulk_wait(bar, phase))) {
      // the copies never completed: flag it, give them one more bounded wait
      // (they target this warp's shared memory), and stop
      if (lane == 0) atomicOr(a.err, 2);
      bulk_wait(bar, phase);
      return;
    }
    phase ^= 1;
    const size_t off = (size_t)blk * BINS;
    const float gf = (MODE >= 1) ? a.c.degrid * stage[(2 - LO) * BINS].x / gs0 : 0.f;
    float gsh = 0.f;
#pragma unroll 1
    for (int j = 0; j < PER; j++) {
      const int i = lane + 32 * j;
      float2 v = make_float2(0.f, 0.f);
      BinTab tb{make_float2(0.f, 0.f), 0.f, 0.f};
      if (i < BINS) {
        tb = bin_tab<MODE>(a, i);
        float2 w[5];
#pragma unroll
        for (int k = 0; k < 5; k++)
          w[k] = (k >= LO && k < LO + NW) ? stage[(k - LO) * BINS + i] : make_float2(0.f, 0.f);
        v = filter_vals<MODE>(a, w, off, i, gf, tb, true);
      }
      if (a.c.do_sharpen) {
        if (j == 0) gsh = a.c.degrid * __shfl_sync(0xffffffffu, v.x, 0) / gs0;
        if (i < BINS) v = sharpen_bin(a, v, tb, gsh);
      }
      if (i < BINS) S[i] = v;
    }
    __syncwarp();
    if (lane == 0 && idx + nwarps < g.nblocks) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      fetch(block_of(idx + nwarps));
    }
    for (int c = lane; c < HC; c += 32) inv_col<BW, BH>(S, c);
    __syncwarp();
    for (int y = lane; y < BH; y += 32) inv_row_inplace<BW, BH>(S, y);
    __syncwarp();
    store_tdom<BW, BH>(S, a.tdom + (size_t)blk * BH * BW, lane);
    __syncwarp();
  }
}

// ---------------------------------------------------------------- one launch per frame

// One output frame in one launch: each CTA transforms the window's newest frame
// for its blocks (the spectra go to the ring for the next output frames and
// stay in its tiles), filters them with the older frames' spectra from the
// ring and inverse-transforms them; with `of`, the CTA that completes an
// output tile does its overlap-add. For small planes, whose frames cost their
// launches and the latency of three kernels' chains rather than any
// throughput.
template <int BW, int BH, typename T, int MODE>
__global__ void __launch_bounds__(kWarps * 32, ctas_for(5, group_smem_bytes<BW, BH>(1)))
    k_frame(const __grid_constant__ ForwardArgs f, const __grid_constant__ InverseArgs a,
            const __grid_constant__ TemporalSet ts, const __grid_constant__ OlaFuse of) {
  extern __shared__ __align__(16) float2 smem2[];
  const int blk0 = blockIdx.x * ts.nb;
  frame_forward<BW, BH, T>(f, blk0, min(ts.nb, a.g.nblocks - blk0), smem2 + group_head_floats<BW, BH>() / 2);
  filter_inverse_group_cta<BW, BH, MODE, false, true>(a, ts, blockIdx.x, nullptr, 0, of.cnt ? &of : nullptr);
}

// ---------------------------------------------------------------- launchers

template <int BW, int BH>
int fft_grid(int nblocks) {
  return fft_ctas<BW, BH>(nblocks);
}

// Batched launches of one kernel variant over many planes (see k_forward_batch).
template <int BW, int BH, typename T>
cudaError_t fwd_batch_typed(const BatchLaunch& l, cudaStream_t s) {
  const cudaError_t e = fft3d::smem_attr(k_forward_batch<BW, BH, T>, fwd_smem<BW, BH>());
  if (e != cudaSuccess) return e;
  k_forward_batch<BW, BH, T><<<l.grid, fwd_threads<BW>(), fwd_smem<BW, BH>(), s>>>(static_cast<const ForwardArgs*>(l.args),
                                                                                   l.items, l.nitems);
  return cudaGetLastError();
}
template <int BW, int BH>
cudaError_t fwd_batch(const BatchLaunch& l, int bytes, cudaStream_t s) {
  if (bytes == 1) return fwd_batch_typed<BW, BH, uint8_t>(l, s);
  if (bytes == 2) return fwd_batch_typed<BW, BH, uint16_t>(l, s);
  return fwd_batch_typed<BW, BH, float>(l, s);
}

template <int BW, int BH, int MODE>
cudaError_t inv_batch_mode(const BatchLaunch& l, cudaStream_t s) {
  const int smem = kWarps * fft_smem_bytes<BW, BH>();
  cudaError_t e = fft3d::smem_attr(k_filter_inverse_batch<BW, BH, MODE>, smem);
  if (e != cudaSuccess) return e;
  k_filter_inverse_batch<BW, BH, MODE><<<l.grid, kWarps * 32, smem, s>>>(static_cast<const InverseArgs*>(l.args),
                                                                         l.items, l.nitems);
  return cudaGetLastError();
}

template <int BW, int BH>
cudaError_t inv_batch(const BatchLaunch& l, int mode, cudaStream_t s) {
  switch (mode) {
    case MODE_SHARPEN_ONLY: return inv_batch_mode<BW, BH, MODE_SHARPEN_ONLY>(l, s);
    case MODE_KALMAN: return inv_batch_mode<BW, BH, MODE_KALMAN>(l, s);
    case 1: return inv_batch_mode<BW, BH, 1>(l, s);
    case 2: return inv_batch_mode<BW, BH, 2>(l, s);
    case 3: return inv_batch_mode<BW, BH, 3>(l, s);
    case 4: return inv_batch_mode<BW, BH, 4>(l, s);
    case 5: return inv_batch_mode<BW, BH, 5>(l, s);
  }
  return cudaErrorInvalidValue;
}

// CTAs of one plane's unbatched launch (the work items per plane of a batch)
template <int BW, int BH>
int ctas_per_plane(int nblocks) {
  return fft_ctas<BW, BH>(nblocks);
}

// Occupancy (resident CTAs per SM) of the batched kernels.
template <int BW, int BH>
int occupancy_of(int which, int mode_or_bytes) {
  const int smem = kWarps * fft_smem_bytes<BW, BH>();
  int n = 0;
  if (which == 0) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_forward_batch<BW, BH, uint8_t>, fwd_threads<BW>(), fwd_smem<BW, BH>());
  } else if (which == 3) {
    const int gsmem = group_smem_bytes<BW, BH>(run_tiles<BW, BH, 5, run_staged<BW, BH, 5>()>()) + (int)sizeof(GroupRun);
    fft3d::smem_attr(k_filter_inverse_group_batch<BW, BH, 5>, gsmem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_filter_inverse_group_batch<BW, BH, 5>, kWarps * 32, gsmem);
  } else {
    switch (mode_or_bytes) {
      case MODE_KALMAN:
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_filter_inverse_batch<BW, BH, MODE_KALMAN>, kWarps * 32, smem);
        break;
      case 5:
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_filter_inverse_batch<BW, BH, 5>, kWarps * 32, smem);
        break;
      default:
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_filter_inverse_batch<BW, BH, 3>, kWarps * 32, smem);
    }
  }
  return n > 0 ? n : 1;
}

template <int BW, int BH, typename T>
cudaError_t fwd_typed(const ForwardArgs& a, const FwdFrameSet& fs, cudaStream_t s) {
  const cudaError_t e = fft3d::smem_attr(k_forward_frames<BW, BH, T>, fwd_smem<BW, BH>());
  if (e != cudaSuccess) return e;
  k_forward_frames<BW, BH, T><<<fs.ctas * fs.count, fwd_threads<BW>(), fwd_smem<BW, BH>(), s>>>(a, fs);
  return cudaGetLastError();
}
template <int BW, int BH>
cudaError_t fwd_frames(const ForwardArgs& a, const FwdFrameSet& fs, int bytes, cudaStream_t s) {
  if (fs.count < 1 || fs.count > kMaxFwdFrames) return cudaErrorInvalidValue;
  FwdFrameSet f = fs;
  f.ctas = (a.g.nblocks + fwd_blocks<BW>() - 1) / fwd_blocks<BW>();
  if (bytes == 1) return fwd_typed<BW, BH, uint8_t>(a, f, s);
  if (bytes == 2) return fwd_typed<BW, BH, uint16_t>(a, f, s);
  return fwd_typed<BW, BH, float>(a, f, s);
}
// one frame: a set of one
template <int BW, int BH>
cudaError_t fwd_sized(const ForwardArgs& a, int bytes, cudaStream_t s) {
  FwdFrameSet fs{};
  fs.src[0] = a.src;
  fs.stride[0] = a.src_stride;
  fs.spec[0] = a.spec;
  fs.count = 1;
  return fwd_frames<BW, BH>(a, fs, bytes, s);
}

inline bool ola_fuse_ok(const OlaFuse& of, const Geom& g) {
  return of.cnt && of.tiles_x >= 1 && of.tiles_y >= 1 && of.tiles_x < g.nox && of.tiles_y < g.noy &&
         (of.bytes == 1 || of.bytes == 2 || of.bytes == 4);
}

// Blocks per CTA of a run whose block takes `count` tiles, over nblocks
// blocks: as many as the CTA has tiles for, but no more than keep every CTA
// slot of the chip filled (run_ctas per SM), down to one block per CTA for
// small planes.
template <int BW, int BH, int MODE, bool STAGED>
int group_blocks_per_cta(int nblocks, int count) {
  const int most = std::max(1, run_tiles<BW, BH, MODE, STAGED>() / count);
  const int slots = 148 * run_ctas<BW, BH, MODE, STAGED>(0);
  return std::max(1, std::min(most, nblocks / slots));
}

template <int BW, int BH, int MODE, bool STAGED>
cudaError_t inv_group_launch(const InverseArgs& a, const TemporalSet& ts, const OlaFuse& of, cudaStream_t s) {
  cudaError_t e = fft3d::smem_attr(k_filter_inverse_group<BW, BH, MODE, STAGED>,
                                   group_smem_bytes<BW, BH>(run_tiles<BW, BH, MODE, STAGED>()));
  if (e != cudaSuccess) return e;
  TemporalSet t = ts;
  const int per = ts.count + (STAGED ? win_extra<MODE>() : 0);
  t.nb = of.cnt ? 1 : group_blocks_per_cta<BW, BH, MODE, STAGED>(a.g.nblocks, per);
  k_filter_inverse_group<BW, BH, MODE, STAGED><<<(a.g.nblocks + t.nb - 1) / t.nb, kWarps * 32,
                                                 group_smem_bytes<BW, BH>(t.nb * per), s>>>(a, t, of);
  return cudaGetLastError();
}

// The staged form where it is built and a wait for its copies that ran out can
// be told (a.err): without a flag, as in the allocation-free call, the form
// that waits for nothing.
template <int BW, int BH, int MODE>
cudaError_t inv_group_mode(const InverseArgs& a, const TemporalSet& ts, const OlaFuse& of, cudaStream_t s) {
  if constexpr (run_staged<BW, BH, MODE>()) {
    if (a.err && (MODE < 2 || ts.count > 1)) return inv_group_launch<BW, BH, MODE, true>(a, ts, of, s);
  }
  if constexpr (MODE != MODE_KALMAN || !run_staged<BW, BH, MODE>())  // (a Kalman filter's plane has a flag)
    return inv_group_launch<BW, BH, MODE, false>(a, ts, of, s);
  return cudaErrorInvalidValue;
}

// One output frame: many blocks by k_filter_inverse (a warp owns its blocks; no
// barriers, the loads of 2 to 4 rounds in flight per lane), few by
// k_filter_inverse_group with a CTA per block or more, which fills the chip with
// fewer blocks and has a quarter of the serial work per thread. The line lies
// where both take as long, us by CTAs / by warps: at 8 x 8, 800 blocks 10.6 / 8.6
// (450 equal); wide blocks, whose few rows leave a CTA's threads idle: 32 x 16, 800
// blocks 12.7 / 12.3, 3600 blocks 17.7 / 14.9; tall ones, whose columns are a warp's
// longer chains: 16 x 32, 3600 blocks 18.9 / 19.4, 24 x 32, 2400 blocks 18.8 / 18.0;
// 32 x 32 at bt = 3, 1600 blocks 18.6 / 17.8, at bt = 5, 2400 blocks 25.0 / 24.9, 3600
// blocks 31.1 / 27.5. 48 x 48 at bt = 1 or -1 has one spectrum to read, by a bulk
// copy, and the tiles of four resident CTAs: 8000 blocks 62 / 68. Kalman: 32 x 32,
// 8000 blocks 51 / 37.
template <int BW, int BH, int MODE>
bool one_frame_by_warps(int nblocks) {
  if (BW * BH >= 48 * 48 && (MODE == MODE_WIENER2D || MODE == MODE_SHARPEN_ONLY)) return false;
  constexpr int square = MODE >= 4 ? 3000 : 1500;
  return nblocks > (BW < 12 ? 400 : BW > BH ? 700 : BW == BH ? square : BW < 24 ? 4000 : 2000);
}

template <int BW, int BH, int MODE>
cudaError_t inv_mode(const InverseArgs& a, cudaStream_t s) {
  constexpr int bulk_smem = 128 + kBulkWarps * bulk_warp_bytes<BW, BH, MODE>();
  if (MODE != MODE_KALMAN && a.bulk && a.err && bulk_smem <= 160 * 1024) {
    cudaError_t e = fft3d::smem_attr(k_filter_inverse_bulk<BW, BH, MODE>, bulk_smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0, dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_filter_inverse_bulk<BW, BH, MODE>, kBulkWarps * 32,
                                                  bulk_smem);
    const int need = (a.g.nblocks + kBulkWarps - 1) / kBulkWarps;
    const int grid = std::min(need, std::max(1, per_sm) * sms);
    k_filter_inverse_bulk<BW, BH, MODE><<<grid, kBulkWarps * 32, bulk_smem, s>>>(a);
    return cudaGetLastError();
  }
  if (one_frame_by_warps<BW, BH, MODE>(a.g.nblocks)) {
    const int smem = kWarps * fft_smem_bytes<BW, BH>();
    cudaError_t e = fft3d::smem_attr(k_filter_inverse<BW, BH, MODE>, smem);
    if (e != cudaSuccess) return e;
    k_filter_inverse<BW, BH, MODE><<<fft_grid<BW, BH>(a.g.nblocks), kWarps * 32, smem, s>>>(a);
    return cudaGetLastError();
  }
  // one frame is a run of one
  TemporalSet ts{};
  ts.count = 1;
  for (int k = 0; k < 5; k++) ts.spec[k] = a.in[k];
  ts.tdom[0] = a.tdom;
  return inv_group_mode<BW, BH, MODE>(a, ts, OlaFuse{}, s);
}

template <int BW, int BH, typename T, int MODE>
cudaError_t frame_mode(const FrameArgs& a, cudaStream_t s) {
  cudaError_t e = fft3d::smem_attr(k_frame<BW, BH, T, MODE>, group_smem_bytes<BW, BH>(group_tiles<BW, BH>()));
  if (e != cudaSuccess) return e;
  TemporalSet ts{};
  ts.count = 1;
  for (int k = 0; k < 5; k++) ts.spec[k] = a.v.in[k];
  ts.tdom[0] = a.v.tdom;
  ts.nb = a.of.cnt ? 1 : group_blocks_per_cta<BW, BH, MODE, false>(a.v.g.nblocks, 1);
  k_frame<BW, BH, T, MODE><<<(a.v.g.nblocks + ts.nb - 1) / ts.nb, kWarps * 32, group_smem_bytes<BW, BH>(ts.nb), s>>>(
      a.f, a.v, ts, a.of);
  return cudaGetLastError();
}

template <int BW, int BH, typename T>
cudaError_t frame_typed(const FrameArgs& a, int mode, cudaStream_t s) {
  switch (mode) {
    case MODE_SHARPEN_ONLY: return frame_mode<BW, BH, T, MODE_SHARPEN_ONLY>(a, s);
    case MODE_KALMAN: return frame_mode<BW, BH, T, MODE_KALMAN>(a, s);
    case 1: return frame_mode<BW, BH, T, 1>(a, s);
    case 2: return frame_mode<BW, BH, T, 2>(a, s);
    case 3: return frame_mode<BW, BH, T, 3>(a, s);
    case 4: return frame_mode<BW, BH, T, 4>(a, s);
    case 5: return frame_mode<BW, BH, T, 5>(a, s);
  }
  return cudaErrorInvalidValue;
}

template <int BW, int BH>
cudaError_t frame_sized(const FrameArgs& a, int mode, int bytes, cudaStream_t s) {
  if (a.of.cnt && !ola_fuse_ok(a.of, a.v.g)) return cudaErrorInvalidValue;
  if (bytes == 1) return frame_typed<BW, BH, uint8_t>(a, mode, s);
  if (bytes == 2) return frame_typed<BW, BH, uint16_t>(a, mode, s);
  return cudaErrorNotSupported;  // float samples use the unfused path
}

template <int BW, int BH, int MODE>
cudaError_t inv_frames_mode(const InverseArgs& a, const FrameSet& fs, cudaStream_t s) {
  const int smem = kWarps * fft_smem_bytes<BW, BH>();
  const int grid = fft_grid<BW, BH>(a.g.nblocks) * fs.count;
  cudaError_t e = fft3d::smem_attr(k_filter_inverse_frames<BW, BH, MODE>, smem);
  if (e != cudaSuccess) return e;
  k_filter_inverse_frames<BW, BH, MODE><<<grid, kWarps * 32, smem, s>>>(a, fs);
  return cudaGetLastError();
}

// frame groups: Wiener 3D windows (the modes whose frames share spectra)
template <int BW, int BH>
cudaError_t inv_frames(const InverseArgs& a, const FrameSet& fs, int mode, cudaStream_t s) {
  if (fs.count < 1 || fs.count > kMaxGroupFrames) return cudaErrorInvalidValue;
  switch (mode) {
    case MODE_SHARPEN_ONLY: return inv_frames_mode<BW, BH, MODE_SHARPEN_ONLY>(a, fs, s);
    case 2: return inv_frames_mode<BW, BH, 2>(a, fs, s);
    case 3: return inv_frames_mode<BW, BH, 3>(a, fs, s);
    case 4: return inv_frames_mode<BW, BH, 4>(a, fs, s);
    case 5: return inv_frames_mode<BW, BH, 5>(a, fs, s);
  }
  return cudaErrorInvalidValue;
}

template <int BW, int BH>
cudaError_t inv_group(const InverseArgs& a, const TemporalSet& ts, int mode, cudaStream_t s, const OlaFuse* ofp) {
  if (ts.count < 1 || ts.count > group_run_frames(BW, BH)) return cudaErrorInvalidValue;
  OlaFuse of{};
  if (ofp) {
    of = *ofp;
    if (!ola_fuse_ok(of, a.g)) return cudaErrorInvalidValue;
  }
  switch (mode) {
    case MODE_SHARPEN_ONLY: return inv_group_mode<BW, BH, MODE_SHARPEN_ONLY>(a, ts, of, s);
    case MODE_KALMAN: return inv_group_mode<BW, BH, MODE_KALMAN>(a, ts, of, s);
    case 1: return inv_group_mode<BW, BH, 1>(a, ts, of, s);
    case 2: return inv_group_mode<BW, BH, 2>(a, ts, of, s);
    case 3: return inv_group_mode<BW, BH, 3>(a, ts, of, s);
    case 4: return inv_group_mode<BW, BH, 4>(a, ts, of, s);
    case 5: return inv_group_mode<BW, BH, 5>(a, ts, of, s);
  }
  return cudaErrorInvalidValue;
}

template <int BW, int BH, int MODE>
cudaError_t inv_group_batch_mode(const BatchLaunch& l, cudaStream_t s) {
  const int smem = group_smem_bytes<BW, BH>(run_tiles<BW, BH, MODE, run_staged<BW, BH, MODE>()>()) + (int)sizeof(GroupRun);
  cudaError_t e = fft3d::smem_attr(k_filter_inverse_group_batch<BW, BH, MODE>, smem);
  if (e != cudaSuccess) return e;
  k_filter_inverse_group_batch<BW, BH, MODE><<<l.grid, kWarps * 32, smem, s>>>(static_cast<const GroupRun*>(l.args),
                                                                             l.items, l.nitems);
  return cudaGetLastError();
}

template <int BW, int BH>
cudaError_t inv_group_batch(const BatchLaunch& l, int mode, cudaStream_t s) {
  switch (mode) {
    case MODE_SHARPEN_ONLY: return inv_group_batch_mode<BW, BH, MODE_SHARPEN_ONLY>(l, s);
    case MODE_KALMAN: return inv_group_batch_mode<BW, BH, MODE_KALMAN>(l, s);
    case 1: return inv_group_batch_mode<BW, BH, 1>(l, s);
    case 2: return inv_group_batch_mode<BW, BH, 2>(l, s);
    case 3: return inv_group_batch_mode<BW, BH, 3>(l, s);
    case 4: return inv_group_batch_mode<BW, BH, 4>(l, s);
    case 5: return inv_group_batch_mode<BW, BH, 5>(l, s);
  }
  return cudaErrorInvalidValue;
}

template <int BW, int BH>
cudaError_t inv_sized(const InverseArgs& a, int mode, cudaStream_t s) {
  switch (mode) {
    case MODE_SHARPEN_ONLY: return inv_mode<BW, BH, MODE_SHARPEN_ONLY>(a, s);
    case MODE_KALMAN: return inv_mode<BW, BH, MODE_KALMAN>(a, s);
    case 1: return inv_mode<BW, BH, 1>(a, s);
    case 2: return inv_mode<BW, BH, 2>(a, s);
    case 3: return inv_mode<BW, BH, 3>(a, s);
    case 4: return inv_mode<BW, BH, 4>(a, s);
    case 5: return inv_mode<BW, BH, 5>(a, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

// Registers block size BW x BH of this translation unit in the size table.
#define FFT3D_REGISTER_SIZE(BW, BH)                                                                     \
  static const bool fft3d_reg_##BW##x##BH = register_size(                                             \
      SizeEntry{BW, BH, &fwd_sized<BW, BH>, &inv_sized<BW, BH>, &frame_sized<BW, BH>, &upload_twiddle_table, \
                &fwd_batch<BW, BH>, &inv_batch<BW, BH>, &ctas_per_plane<BW, BH>, &occupancy_of<BW, BH>,      \
                &inv_frames<BW, BH>, &fwd_frames<BW, BH>, &inv_group<BW, BH>, &inv_group_batch<BW, BH>});

}  // namespace fft3d
