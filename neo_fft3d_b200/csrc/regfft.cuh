// Register-resident mixed-radix FFTs for one thread (sm_100a).
//
// Every transform length is a compile-time constant, every loop is fully
// unrolled, so the data array lives in registers and every twiddle index is a
// constant: the twiddles are read from a __constant__ table whose operands the
// FFMA instructions take directly (constant-bank operands), with no loads.
//
// Algorithm: Stockham self-sorting passes (natural order in and out) with
// radix 4, 2 and 3 butterflies:
//   Y[j + L q + L P k] = sum_u W_P^{q u} (W_{L P}^{j u} X[j + L (k + R u)])
// for pass radix P, L = product of the earlier radices, R = N / (L P).
// Lengths: any N = 2^a 3^b dividing kTwN (384), so 2..128, 6, 12, 24, 48, 96.
#pragma once
#include <cuda_runtime.h>

namespace fft3d {

// Two floats in one 64-bit register pair, for the packed f32x2 instructions
// (each lane rounds like the scalar operation). Held as one 64-bit value and
// worked on with PTX: the same arithmetic on float2 and its intrinsics cost 50
// register moves per bin pair and frame at bt = 5 (188 instructions instead of
// 131), because the halves are then allocated one by one.
using f2x = unsigned long long;
__device__ __forceinline__ f2x pk2(float lo, float hi) {
  f2x r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f2x dup2(float v) { return pk2(v, v); }
__device__ __forceinline__ float2 up2(f2x v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2x add2(f2x a, f2x b) {
  f2x r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2x sub2(f2x a, f2x b) {
  f2x r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2x mul2(f2x a, f2x b) {
  f2x r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2x fma2(f2x a, f2x b, f2x c) {
  f2x r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// x * s with products that stay products: ptxas contracts a packed multiply
// into a packed add that follows (explicit rounding or not), which would round
// once where the scalar code rounds twice; two scalar multiplies
// are left alone, at the same cost on the FMA pipe.
__device__ __forceinline__ f2x mul2_kept(f2x v, f2x s) {
  const float2 a = up2(v), b = up2(s);
  return pk2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y));
}
constexpr int kTwN = 384;  // W_384^k = exp(-2 pi i k / 384), k < 384
// One copy per translation unit (whole-program compilation keeps __constant__
// memory per module); each TU that includes this header uploads it with
// upload_twiddle_table() once per device.
static __constant__ float2 c_tw[kTwN];
// The same factors for two transforms at once (rfft_pair): the real part, the
// imaginary part and their negatives, each as a pair that the packed
// instructions take from the constant bank.
struct TwPair {
  float2 re, im, nim, nre;
};
static __constant__ TwPair c_tw_pair[kTwN];

static inline cudaError_t upload_twiddle_table() {
  float2 h[kTwN];
  TwPair hp[kTwN];
  for (int k = 0; k < kTwN; k++) {
    double a = -2.0 * 3.14159265358979323846 * (double)k / (double)kTwN;
    h[k] = make_float2((float)__builtin_cos(a), (float)__builtin_sin(a));
    hp[k].re = make_float2(h[k].x, h[k].x);
    hp[k].im = make_float2(h[k].y, h[k].y);
    hp[k].nim = make_float2(-h[k].y, -h[k].y);
    hp[k].nre = make_float2(-h[k].x, -h[k].x);
  }
  const cudaError_t e = cudaMemcpyToSymbol(c_tw, h, sizeof(h));
  return e != cudaSuccess ? e : cudaMemcpyToSymbol(c_tw_pair, hp, sizeof(hp));
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// Complex adds as packed f32x2 operations (one instruction for both parts,
// each part rounded exactly as a scalar add).
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }

// W_N^m for SIGN = -1 (forward) or its conjugate for SIGN = +1.
template <int N, int SIGN>
__device__ __forceinline__ float2 tw(int m) {
  static_assert(kTwN % N == 0, "transform length must divide 384");
  float2 w = c_tw[(m % N) * (kTwN / N)];
  return SIGN < 0 ? w : cconj(w);
}

// small DFTs in place, sign SIGN
template <int P, int SIGN>
__device__ __forceinline__ void small_dft(float2 (&t)[P]) {
  if constexpr (P == 2) {
    float2 a = t[0], b = t[1];
    t[0] = cadd(a, b);
    t[1] = csub(a, b);
  } else if constexpr (P == 4) {
    float2 s02 = cadd(t[0], t[2]), d02 = csub(t[0], t[2]);
    float2 s13 = cadd(t[1], t[3]), d13 = csub(t[1], t[3]);
    // d13 * (SIGN * i)
    float2 j = SIGN < 0 ? make_float2(d13.y, -d13.x) : make_float2(-d13.y, d13.x);
    t[0] = cadd(s02, s13);
    t[1] = cadd(d02, j);
    t[2] = csub(s02, s13);
    t[3] = csub(d02, j);
  } else if constexpr (P == 3) {
    const float c = -0.5f;
    const float s = SIGN < 0 ? -0.86602540378443864676f : 0.86602540378443864676f;
    float2 a = t[0], b = t[1], d = t[2];
    float2 sum = cadd(b, d), dif = csub(b, d);
    float2 m = make_float2(a.x + c * sum.x, a.y + c * sum.y);
    // i * s * dif
    float2 r = make_float2(-s * dif.y, s * dif.x);
    t[0] = cadd(a, sum);
    t[1] = cadd(m, r);
    t[2] = csub(m, r);
  }
}

template <int N>
struct Radices {
  // first radix used for length N in the recursion below (4 while N%4==0 and N>=16 or N==4)
  static constexpr int first = (N % 4 == 0) ? 4 : ((N % 2 == 0) ? 2 : 3);
};

template <int N, int SIGN, int L>
__device__ __forceinline__ void stockham(float2 (&x)[N]) {
  if constexpr (L < N) {
    constexpr int rem = N / L;
    constexpr int P = Radices<rem>::first;
    constexpr int R = N / (L * P);
    float2 y[N];
#pragma unroll
    for (int k = 0; k < R; k++) {
#pragma unroll
      for (int j = 0; j < L; j++) {
        float2 t[P];
#pragma unroll
        for (int u = 0; u < P; u++) {
          float2 a = x[j + L * (k + R * u)];
          if (j * u != 0) a = cmul(a, tw<N, SIGN>(j * u * R));  // W_{LP}^{ju} = W_N^{ju R}
          t[u] = a;
        }
        small_dft<P, SIGN>(t);
#pragma unroll
        for (int q = 0; q < P; q++) y[j + L * q + L * P * k] = t[q];
      }
    }
#pragma unroll
    for (int i = 0; i < N; i++) x[i] = y[i];
    stockham<N, SIGN, L * P>(x);
  }
}

// Unnormalised complex DFT of length N in place (SIGN -1 forward, +1 inverse).
template <int N, int SIGN>
__device__ __forceinline__ void cfft(float2 (&x)[N]) {
  if constexpr (N > 1) stockham<N, SIGN, 1>(x);
}

// Real-to-complex DFT of length N (even): out[k], k = 0..N/2, through one
// complex DFT of length N/2 on z[m] = x[2m] + i x[2m+1].
template <int N>
__device__ __forceinline__ void rfft(const float (&x)[N], float2 (&out)[N / 2 + 1]) {
  constexpr int H = N / 2;
  float2 z[H];
#pragma unroll
  for (int m = 0; m < H; m++) z[m] = make_float2(x[2 * m], x[2 * m + 1]);
  cfft<H, -1>(z);
#pragma unroll
  for (int k = 0; k <= H; k++) {
    float2 zk = z[k % H], zc = cconj(z[(H - k) % H]);
    float2 e = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y + zc.y));
    // o = (zk - zc) / (2 i)
    float2 d = csub(zk, zc);
    float2 o = make_float2(0.5f * d.y, -0.5f * d.x);
    out[k] = (k == 0 || k == H) ? make_float2(e.x + (k == 0 ? o.x : -o.x), e.y + (k == 0 ? o.y : -o.y))
                                : cadd(e, cmul(o, tw<N, -1>(k)));
  }
}

// Complex-to-real inverse DFT of length N (unnormalised, like FFTW's c2r): the
// imaginary parts of in[0] and in[N/2] are ignored.
template <int N>
__device__ __forceinline__ void irfft(const float2 (&in)[N / 2 + 1], float (&x)[N]) {
  constexpr int H = N / 2;
  float2 z[H];
#pragma unroll
  for (int k = 0; k < H; k++) {
    float2 a = in[k], b = in[H - k];
    if (k == 0) { a.y = 0.f; b.y = 0.f; }
    float2 bc = cconj(b);
    float2 e = cadd(a, bc);
    float2 o = csub(a, bc);
    if (k != 0) o = cmul(o, tw<N, +1>(k));
    // z = e + i o
    z[k] = make_float2(e.x - o.y, e.y + o.x);
  }
  cfft<H, +1>(z);
#pragma unroll
  for (int m = 0; m < H; m++) {
    x[2 * m] = z[m].x;
    x[2 * m + 1] = z[m].y;
  }
}

// ---------------------------------------------------------------- two transforms at once

// Two sequences A and B in one thread: re[i] = (A_i.re, B_i.re) and im[i] =
// (A_i.im, B_i.im), packed. A turn by i only changes re and im about, and a
// twiddle costs four instructions for both sequences (one sequence as (re, im)
// pairs: four for one): two 32-sample rows take 233 instead of 349
// instructions through their 16-point transforms, 221 us instead of 309 in a
// loop of nothing else. Every operation rounds as in the scalar code; where
// that has a fused multiply-add, so has this.
// a * W, W = tw<N, SIGN>(m): re = fma(a.re, W.re, -(a.im W.im)), im = fma(a.im, W.re, a.re W.im)
template <int N, int SIGN>
__device__ __forceinline__ void cmul_pair(f2x& re, f2x& im, int m) {
  const TwPair& w = c_tw_pair[(m % N) * (kTwN / N)];
  const f2x wr = *reinterpret_cast<const f2x*>(&w.re);
  const f2x wi = *reinterpret_cast<const f2x*>(SIGN < 0 ? &w.im : &w.nim);
  const f2x nwi = *reinterpret_cast<const f2x*>(SIGN < 0 ? &w.nim : &w.im);
  const f2x r = fma2(re, wr, mul2(im, nwi)), i = fma2(im, wr, mul2(re, wi));
  re = r;
  im = i;
}

template <int P, int SIGN>
__device__ __forceinline__ void small_dft_pair(f2x (&a)[P], f2x (&b)[P]) {
  if constexpr (P == 2) {
    const f2x x = a[0], y = b[0];
    a[0] = add2(x, a[1]);
    b[0] = add2(y, b[1]);
    a[1] = sub2(x, a[1]);
    b[1] = sub2(y, b[1]);
  } else if constexpr (P == 4) {
    const f2x sa = add2(a[0], a[2]), sb = add2(b[0], b[2]), da = sub2(a[0], a[2]), db = sub2(b[0], b[2]);
    const f2x ta = add2(a[1], a[3]), tb = add2(b[1], b[3]), ea = sub2(a[1], a[3]), eb = sub2(b[1], b[3]);
    a[0] = add2(sa, ta);
    b[0] = add2(sb, tb);
    a[2] = sub2(sa, ta);
    b[2] = sub2(sb, tb);
    const f2x pa = add2(da, eb), pb = sub2(db, ea), qa = sub2(da, eb), qb = add2(db, ea);  // d -+ i e
    a[1] = SIGN < 0 ? pa : qa;
    b[1] = SIGN < 0 ? pb : qb;
    a[3] = SIGN < 0 ? qa : pa;
    b[3] = SIGN < 0 ? qb : pb;
  } else {
    static_assert(P == 3, "radix 2, 3 or 4");
    const f2x half = dup2(-0.5f), s = dup2(SIGN < 0 ? -0.86602540378443864676f : 0.86602540378443864676f);
    const f2x sa = add2(a[1], a[2]), sb = add2(b[1], b[2]), da = sub2(a[1], a[2]), db = sub2(b[1], b[2]);
    const f2x ma = fma2(half, sa, a[0]), mb = fma2(half, sb, b[0]);
    const f2x ra = mul2_kept(s, db), rb = mul2_kept(s, da);  // i s d = (-s d.im, s d.re)
    a[0] = add2(a[0], sa);
    b[0] = add2(b[0], sb);
    a[1] = sub2(ma, ra);
    b[1] = add2(mb, rb);
    a[2] = add2(ma, ra);
    b[2] = sub2(mb, rb);
  }
}

template <int N, int SIGN, int L>
__device__ __forceinline__ void stockham_pair(f2x (&x)[N], f2x (&y)[N]) {
  if constexpr (L < N) {
    constexpr int rem = N / L;
    constexpr int P = Radices<rem>::first;
    constexpr int R = N / (L * P);
    f2x u[N], v[N];
#pragma unroll
    for (int k = 0; k < R; k++) {
#pragma unroll
      for (int j = 0; j < L; j++) {
        f2x a[P], b[P];
#pragma unroll
        for (int q = 0; q < P; q++) {
          a[q] = x[j + L * (k + R * q)];
          b[q] = y[j + L * (k + R * q)];
          if (j * q != 0) cmul_pair<N, SIGN>(a[q], b[q], j * q * R);
        }
        small_dft_pair<P, SIGN>(a, b);
#pragma unroll
        for (int q = 0; q < P; q++) {
          u[j + L * q + L * P * k] = a[q];
          v[j + L * q + L * P * k] = b[q];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < N; i++) {
      x[i] = u[i];
      y[i] = v[i];
    }
    stockham_pair<N, SIGN, L * P>(x, y);
  }
}

// rfft of two sequences that come scaled by 1/2 (the caller's window holds the
// factor): the spectrum is then (z_k + conj z_{H-k}) - i W^k (z_k - conj
// z_{H-k}) with no further halving, which a power of two leaves bit for bit
// what rfft gives. The sums and differences of bins k and H - k are shared.
template <int N>
__device__ __forceinline__ void rfft_pair(const f2x (&x)[N], f2x (&re)[N / 2 + 1], f2x (&im)[N / 2 + 1]) {
  constexpr int H = N / 2;
  f2x zr[H], zi[H];
#pragma unroll
  for (int m = 0; m < H; m++) {
    zr[m] = x[2 * m];
    zi[m] = x[2 * m + 1];
  }
  if constexpr (H > 1) stockham_pair<H, -1, 1>(zr, zi);
  {
    // bins 0 and H: z_0 = a + i b gives e = 2 a, o = 2 b
    const f2x e = add2(zr[0], zr[0]), o = add2(zi[0], zi[0]);
    const f2x zero = dup2(0.f);
    re[0] = add2(e, o);
    re[H] = sub2(e, o);
    im[0] = zero;
    im[H] = zero;
  }
#pragma unroll
  for (int k = 1; 2 * k <= H; k++) {
    const int q = H - k;
    const f2x sr = add2(zr[k], zr[q]), si = sub2(zi[k], zi[q]);  // z_k + conj z_q
    const f2x dr = sub2(zr[k], zr[q]), di = add2(zi[k], zi[q]);  // z_k - conj z_q
    {
      const TwPair& w = c_tw_pair[k * (kTwN / N)];
      const f2x wr = *reinterpret_cast<const f2x*>(&w.re), wi = *reinterpret_cast<const f2x*>(&w.im);
      const f2x nwr = *reinterpret_cast<const f2x*>(&w.nre);
      re[k] = add2(sr, fma2(di, wr, mul2(dr, wi)));
      im[k] = add2(si, fma2(dr, nwr, mul2(di, wi)));
    }
    if (q != k) {
      const TwPair& w = c_tw_pair[q * (kTwN / N)];
      const f2x wr = *reinterpret_cast<const f2x*>(&w.re), wi = *reinterpret_cast<const f2x*>(&w.im),
                nwi = *reinterpret_cast<const f2x*>(&w.nim);
      re[q] = add2(sr, fma2(di, wr, mul2(dr, nwi)));
      im[q] = sub2(fma2(dr, wr, mul2(di, wi)), si);
    }
  }
}

}  // namespace fft3d
