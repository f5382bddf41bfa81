// ppb_fft.cuh — register DFTs of small lengths and the two-step split of a
// length N = 16 M, shared by the kernels of k_fft.cu.
//
// A length-N DFT is split N = 16 x M (Cooley-Tukey): one thread per residue
// transforms its elements in registers, multiplies by the twiddles and leaves
// them in shared memory; after one barrier a second set of threads reads
// across the residues and transforms those in registers.  Each element
// crosses shared memory once.  The register DFTs are built from the lengths
// 2, 3, 4, 5, 7, 11 by the same splitting, with twiddles that the compiler
// folds to constants.
#pragma once
#include <cuda_runtime.h>

namespace ppb {
namespace fft {

// cos and sin of 2 pi k / n at compile time (Taylor series after reduction to
// [0, pi/4] by symmetry; double precision)
struct CS {
  double c, s;
};
constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr CS taylor_cs(double x) {
  double c = 1.0, s = x, tc = 1.0, ts = x;
  for (int i = 1; i < 14; i++) {
    tc *= -x * x / ((2 * i - 1) * (2 * i));
    ts *= -x * x / ((2 * i) * (2 * i + 1));
    c += tc;
    s += ts;
  }
  return CS{c, s};
}
constexpr CS unit_root(int k, int n) {
  k %= n;
  // octant reduction: angle 2 pi k / n with 8 k / n in [0, 8)
  const int oct = 8 * k / n;
  if (oct == 0) return taylor_cs(kTwoPi * k / n);
  if (oct == 1 || oct == 2) {   // about pi/2: cos = -sin(x - pi/2)
    const CS t = taylor_cs(kTwoPi * (4 * k - n) / (4.0 * n));
    return CS{-t.s, t.c};
  }
  if (oct == 3 || oct == 4) {
    const CS t = taylor_cs(kTwoPi * (2 * k - n) / (2.0 * n));
    return CS{-t.c, -t.s};
  }
  if (oct == 5 || oct == 6) {
    const CS t = taylor_cs(kTwoPi * (4 * k - 3 * n) / (4.0 * n));
    return CS{t.s, -t.c};
  }
  return taylor_cs(kTwoPi * (k - n) / n);
}
// each root as float plus the float of what the rounding left.  A constant's
// rounding is the same in every transform, so it does not average out: with
// the rounded constants alone psi2 of the tile-local 2LPT, whose source
// cancels at low k, was 13, 8 and 21 % further from 64 bits than with cuFFT's
// transforms at 80^3, 96^3 and 144^3
template <int R> struct Roots {
  float c[R], s[R], cl[R], sl[R];
  constexpr Roots() : c(), s(), cl(), sl() {
    for (int k = 0; k < R; k++) {
      const CS t = unit_root(k, R);
      c[k] = (float)t.c;
      s[k] = (float)t.s;
      cl[k] = (float)(t.c - (double)c[k]);
      sl[k] = (float)(t.s - (double)s[k]);
    }
  }
};

__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a times c + i SIGN s
template <int SIGN> __device__ __forceinline__ float2 rot(float2 a, float c, float s) {
  const float t = SIGN * s;
  return make_float2(fmaf(a.x, c, -a.y * t), fmaf(a.x, t, a.y * c));
}
// acc + x (h + l), the constants known at compile time
__device__ __forceinline__ float fma2(float x, float h, float l, float acc) {
  return l == 0.f ? fmaf(x, h, acc) : fmaf(x, h, fmaf(x, l, acc));
}
// a times root k of R
template <int R, int SIGN> __device__ __forceinline__ float2 rot_root(float2 a, int k) {
  constexpr Roots<R> W;
  const float c = W.c[k], cl = W.cl[k], s = SIGN * W.s[k], sl = SIGN * W.sl[k];
  const float mx = fma2(a.y, s, sl, 0.f), my = fma2(a.y, c, cl, 0.f);
  return make_float2(fma2(a.x, c, cl, -mx), fma2(a.x, s, sl, my));
}

constexpr int first_factor(int R) {   // 4 before 2, then 3, 5, 7, else a prime (R < 64)
  return R % 4 == 0 && R != 4 ? 4 : R % 2 == 0 && R != 2 && R != 4 ? 2 : R % 3 == 0 ? 3 : R % 5 == 0 ? 5 : R % 7 == 0 ? 7 : R;
}

// v := sum_j v[j] exp(SIGN 2 pi i j k / R), natural order in and out
template <int R, int SIGN> __device__ __forceinline__ void dft(float2 (&v)[R]) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = add(a, b);
    v[1] = sub(a, b);
  } else if constexpr (R == 4) {
    const float2 s02 = add(v[0], v[2]), d02 = sub(v[0], v[2]), s13 = add(v[1], v[3]), d = sub(v[1], v[3]);
    const float2 d13 = make_float2(-SIGN * d.y, SIGN * d.x);   // i SIGN d
    v[0] = add(s02, s13);
    v[2] = sub(s02, s13);
    v[1] = add(d02, d13);
    v[3] = sub(d02, d13);
  } else if constexpr (first_factor(R) == R) {   // odd prime: symmetric pairs
    constexpr Roots<R> W;
    constexpr int H = (R - 1) / 2;
    float2 p[H], m[H];
#pragma unroll
    for (int j = 0; j < H; j++) {
      p[j] = add(v[j + 1], v[R - 1 - j]);
      m[j] = sub(v[j + 1], v[R - 1 - j]);
    }
    const float2 v0 = v[0];
    float2 t = v0;
#pragma unroll
    for (int j = 0; j < H; j++) t = add(t, p[j]);
    v[0] = t;
#pragma unroll
    for (int k = 1; k <= H; k++) {
      float2 a = v0, b = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < H; j++) {
        const int i = ((j + 1) * k) % R;
        const float c = W.c[i], cl = W.cl[i], s = SIGN * W.s[i], sl = SIGN * W.sl[i];
        a.x = fma2(p[j].x, c, cl, a.x);
        a.y = fma2(p[j].y, c, cl, a.y);
        b.x = fma2(m[j].y, -s, -sl, b.x);
        b.y = fma2(m[j].x, s, sl, b.y);
      }
      v[k] = add(a, b);
      v[R - k] = sub(a, b);
    }
  } else {
    constexpr int R1 = first_factor(R), R2 = R / R1;
    // v[R2 j1 + j2]: DFT over j1 for each j2, twiddle, DFT over j2
    float2 y[R1][R2];
#pragma unroll
    for (int j2 = 0; j2 < R2; j2++) {
      float2 u[R1];
#pragma unroll
      for (int j1 = 0; j1 < R1; j1++) u[j1] = v[R2 * j1 + j2];
      dft<R1, SIGN>(u);
#pragma unroll
      for (int k1 = 0; k1 < R1; k1++) y[k1][j2] = k1 * j2 ? rot_root<R, SIGN>(u[k1], k1 * j2) : u[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) {
      dft<R2, SIGN>(y[k1]);
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) v[k1 + R1 * k2] = y[k1][k2];
    }
  }
}

}  // namespace fft
}  // namespace ppb
