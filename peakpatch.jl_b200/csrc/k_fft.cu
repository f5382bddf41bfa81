// k_fft.cu — the transforms whose k-space and real-space work is fused into
// them: 2LPT (phi_ij, the source term, psi2), the Laplacian field and the
// filter bank's k^2-weighted twin, for grid sizes N = 16 M.
//
// Half spectra keep cuFFT's [kz][ky][kx] order, kx fastest; the intermediate
// arrays have rows of `hp` = n/2 + 1 rounded up to 4 elements, so that a run
// of 16 kx is four whole 32-byte sectors.  Columns (z or y) are transformed
// by col_kernel: a block owns 16 consecutive kx of one column plane; threads
// read their elements straight from global memory into registers (128-byte
// runs across the 16 kx), transform, cross shared memory once (ppb_fft.cuh)
// and store from registers.
//
// 2LPT (LPT.jl:86-191) in seven passes.  With q = |f|^2 (f the integer
// frequencies), phi_ab = -f_a f_b / q delta: along a z column f_x and f_y are
// constants, so z transforms of g = -delta / q and f_z g (and f_z^2 g) serve
// all six phi; the y pass applies f_y and f_y^2 before its transform, and f_x
// and f_x^2 are applied as the x pass reads.  phi_33 is taken from the trace
// (sum_a phi_aa = -delta) where the caller's formula allows.  src2_kernel
// transforms the phi rows of two (y, z) rows at a time to real space (two
// real rows as one complex transform), forms the source there and transforms
// it forward, so phi and src2 never go to memory.  In units of one half
// spectrum read or written the passes move 3 + 7 + 6.5 + 2 + 3 + 5 + 4.5 = 31;
// separate transforms (multiply, Hermitian projection, three passes each)
// move about 110.  Measured at 384^3 (231 MB per half spectrum): col_kernel
// 4.0-4.4 TB/s of HBM traffic in the y passes (the z passes are bound by
// instructions, the factor of every mode), src2_rows_kernel 0.74 ms (2.1
// TB/s; 15 warps per SM at 128 registers), mid_kernel 0.30 ms, row_kernel 3.2
// TB/s; 2LPT with the Laplacian 6.4 -> 2.7 ms.
#include <cstdint>

#include "ppb_fft.cuh"
#include "ppb_internal.h"

namespace ppb {
namespace {

using fft::dft;

constexpr int kColW = 16;   // kx per block of the column passes
template <int N> constexpr int kM = N / 16;
template <int N> constexpr int kLanes = kM<N> > 16 ? kM<N> : 16;   // threads per column or row pair
// blocks per SM the column kernels are compiled for
template <int N> constexpr int kColBlocks = kLanes<N> == 16 ? 4 : kLanes<N> <= 24 ? 2 : 1;
template <int N> constexpr int kPairs = (kLanes<N> > 24 ? 8 : 256 / kLanes<N>);   // row pairs per block

template <int SIGN> __device__ __forceinline__ float2 twid(float2 a, const float2* __restrict__ tw, int e) {
  const float2 w = __ldg(tw + e);
  return fft::rot<SIGN>(a, w.x, w.y);
}

// k-space factors as unevaluated sums of two floats (43 bits and more), applied
// with one rounding: the accuracy of a factor formed in FP64 without its
// conversions and division (fields with 2LPT and Laplacian at 384^3: 6.92 ms
// with factors rounded to float, 7.22 in FP64, 6.98 so)
struct Pair {
  float h, l;
};
Pair pair_of(double x) { return Pair{(float)x, (float)(x - (double)(float)x)}; }
__device__ __forceinline__ Pair operator*(const Pair& a, float b) {
  const float h = a.h * b;
  return Pair{h, fmaf(a.l, b, fmaf(a.h, b, -h))};
}
__device__ __forceinline__ Pair over(const Pair& a, int q) {   // a / q, 0 < q < 2^24
  // r is within 2 ulp of 1 / q, r + e within 2^-43
  const float r = __fdividef(1.f, (float)q), e = r * fmaf(-(float)q, r, 1.f), h = a.h * r;
  return Pair{h, fmaf(a.h, e, fmaf(a.l, r, fmaf(a.h, r, -h)))};
}
__device__ __forceinline__ float apply(float x, const Pair& s) { return fmaf(x, s.h, x * s.l); }

// elements t + M j (j < 16) of thread t < M -> elements q + 16 p (p < M) of
// thread q < 16, through sm[(q M + t) W]
template <int N, int SIGN> __device__ __forceinline__ void step_a(float2 (&v)[16], int t, float2* sm, int W,
                                                                 const float2* __restrict__ tw) {
  constexpr int M = kM<N>;
  dft<16, SIGN>(v);
#pragma unroll
  for (int q = 0; q < 16; q++) sm[(q * M + t) * W] = q ? twid<SIGN>(v[q], tw, t * q) : v[q];
}
template <int N, int SIGN> __device__ __forceinline__ void step_b(float2 (&u)[kM<N>], int q, const float2* sm, int W) {
  constexpr int M = kM<N>;
#pragma unroll
  for (int t = 0; t < M; t++) u[t] = sm[(q * M + t) * W];
  dft<M, SIGN>(u);
}

struct ColOut {
  const float2* in;
  float2* out;
  int pow;     // power of the column's own frequency
  int flim;    // frequencies above flim (on any axis) are taken as zero; N/2: none
};
struct ColArgs {
  ColOut o[kTwinGroup];
  const float2* tw;
  const float* win;       // kind 3: W_3 by q, wstride apart per output
  int64_t wstride;
  int nout;
  int kind;               // transfer applied as the input is read (z passes): 0 none, 1 ps / q, 2 q ps, 3 W_3(q) ps
  int zero_nyq;           // the transfer zeroes the Nyquist planes
  Pair ps;
  int fmax;               // largest flim
  int hp_in, hp;          // row pitches
  int64_t js_in, js;      // strides along the column (in, out)
  int64_t bs_in, bs;      // strides of the plane index
  int zpass;              // planes are ky (only |ky| <= fmax), else z
};

// Column transforms, one output per block (an input that serves two or three
// outputs is read by neighbouring blocks at the same time, from L2).  Bound:
// HBM, or L2 where the arrays fit it.
template <int N, int SIGN>
__global__ void __launch_bounds__(kColW* kLanes<N>, kColBlocks<N>) col_kernel(const __grid_constant__ ColArgs a) {
  constexpr int M = kM<N>;
  extern __shared__ float2 sm[];
  const int c = threadIdx.x & (kColW - 1), u = threadIdx.x / kColW;
  const int o = blockIdx.x % a.nout, kx = (blockIdx.x / a.nout) * kColW + c;
  const int flim = a.o[o].flim;
  const bool live = kx <= flim;
  int b = blockIdx.y;
  if (a.zpass && b > a.fmax) b += N - (int)gridDim.y;   // the negative ky kept
  if (kx - c > flim || (a.zpass && b > flim && N - b > flim)) return;   // the whole block
  if (u < M) {
    float2 v[16];
    const float2* src = a.o[o].in + b * a.bs_in + kx + u * a.js_in;
    const int64_t step = M * a.js_in;
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const int e = u + M * j;
      v[j] = live && (e <= flim || N - e <= flim) ? src[j * step] : make_float2(0.f, 0.f);
    }
    const int pw = a.o[o].pow;
    if (a.kind) {
      const int fb = b < N / 2 ? b : b - N, q0 = kx * kx + fb * fb;
      const bool znp = a.zero_nyq && (kx == N / 2 || b == N / 2);
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const int e = u + M * j, f = e < N / 2 ? e : e - N;
        const int q = q0 + f * f;
        const bool zero = znp || (a.zero_nyq && e == N / 2);
        if (a.kind == 3) {
          const float s = zero ? 0.f : __ldg(a.win + o * a.wstride + (live ? q : 0)) * a.ps.h;
          v[j].x *= s;
          v[j].y *= s;
        } else {   // the column's frequency goes into the factor
          Pair s = a.kind == 2 ? a.ps * (float)q : over(a.ps, max(q, 1));
          if (zero || q == 0) s = Pair{0.f, 0.f};
          if (pw) s = s * (float)(pw == 1 ? f : f * f);
          v[j].x = apply(v[j].x, s);
          v[j].y = apply(v[j].y, s);
        }
      }
    } else if (pw) {
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const int e = u + M * j;
        const float f = (float)(e < N / 2 ? e : e - N), s = pw == 1 ? f : f * f;
        v[j].x *= s;
        v[j].y *= s;
      }
    }
    step_a<N, SIGN>(v, u, sm + c, kColW, a.tw);
  }
  __syncthreads();
  if (u < 16) {
    float2 w[M];
    step_b<N, SIGN>(w, u, sm + c, kColW);
    if (live) {
      float2* dst = a.o[o].out + b * a.bs + kx + u * a.js;
      const int64_t step = 16 * a.js;
#pragma unroll
      for (int p = 0; p < M; p++) dst[p * step] = w[p];
    }
  }
}

// The z columns of psi2: forward transform of the source, times -i ps / q
// (zero at the DC mode and the Nyquist planes), and the inverse transforms of
// the result h and of f_z h, from one read
struct MidArgs {
  const float2* in;
  float2 *h0, *h1;
  const float2* tw;
  Pair ps;
  int hp;
};
template <int N>
__global__ void __launch_bounds__(kColW* kLanes<N>, 1) mid_kernel(const __grid_constant__ MidArgs a) {
  constexpr int M = kM<N>, nh = N / 2 + 1;
  extern __shared__ float2 sm[];
  const int c = threadIdx.x & (kColW - 1), u = threadIdx.x / kColW;
  const int kx = blockIdx.x * kColW + c, iy = blockIdx.y;
  const bool live = kx < nh;
  const int64_t js = (int64_t)N * a.hp, base = (int64_t)iy * a.hp + kx;
  if (u < M) {
    float2 d[16];
#pragma unroll
    for (int j = 0; j < 16; j++) d[j] = live ? __ldg(a.in + base + (u + M * j) * js) : make_float2(0.f, 0.f);
    step_a<N, -1>(d, u, sm + c, kColW, a.tw);
  }
  __syncthreads();
  const int fy = iy < N / 2 ? iy : iy - N, q0 = kx * kx + fy * fy;
  const bool z0 = kx == N / 2 || iy == N / 2;
  float2 h[M];
  if (u < 16) step_b<N, -1>(h, u, sm + c, kColW);   // kz = u + 16 p
  for (int o = 0; o < 2; o++) {
    __syncthreads();
    if (u < 16) {   // elements u + 16 p: transfer, DFT over p, twiddle, then across u
      float2 v[M];
#pragma unroll
      for (int p = 0; p < M; p++) {
        const int e = u + 16 * p, f = e < N / 2 ? e : e - N;
        const int q = q0 + f * f;
        Pair s = over(a.ps, max(q, 1));
        if (z0 || e == N / 2 || q == 0) s = Pair{0.f, 0.f};
        if (o) s = s * (float)f;
        v[p] = make_float2(apply(h[p].y, s), -apply(h[p].x, s));   // -i s h
      }
      dft<M, 1>(v);
#pragma unroll
      for (int r = 0; r < M; r++) sm[(r * 16 + u) * kColW + c] = r ? twid<1>(v[r], a.tw, u * r) : v[r];
    }
    __syncthreads();
    if (u < M) {
      float2 w[16];
#pragma unroll
      for (int q = 0; q < 16; q++) w[q] = sm[(u * 16 + q) * kColW + c];
      dft<16, 1>(w);
      if (live) {
        float2* dst = (o ? a.h1 : a.h0) + base;
#pragma unroll
        for (int s = 0; s < 16; s++) dst[(u + M * s) * js] = w[s];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// rows (x): two real rows as the real and imaginary parts of one length-N
// transform.  In: half rows A, B of z/y-transformed spectra, C[k] = A[k] + i
// B[k] (k <= N/2), conj A[N-k] + i conj B[N-k] beyond; at k = 0 and N/2 only
// the real parts of A and B enter, the Hermitian projection of those planes.
// Thread t < 16 of a pair holds k = t + 16 j (j < M); after step one (through
// sm[r 17 + t]) thread r < M holds x = r + M s, s < 16.
// ---------------------------------------------------------------------------
template <int N> constexpr int kRowSm = kM<N> * 17 > 16 * (kM<N> | 1) ? kM<N> * 17 : 16 * (kM<N> | 1);

template <int N>
__device__ __forceinline__ void rows_in(float2 (&v)[kM<N>], int t, const float2* __restrict__ A,
                                        const float2* __restrict__ B, int pw, float2* sm,
                                        const float2* __restrict__ tw) {
  constexpr int M = kM<N>;
#pragma unroll
  for (int j = 0; j < M; j++) {
    const int k = t + 16 * j, kk = k <= N / 2 ? k : N - k;
    float2 x = __ldg(A + kk), y = __ldg(B + kk);
    if (kk == 0 || kk == N / 2) x.y = y.y = 0.f;
    if (k > N / 2) { x.y = -x.y; y.y = -y.y; }
    const float f = (float)kk, s = pw == 0 ? 1.f : pw == 1 ? f : f * f;
    v[j] = make_float2(s * (x.x - y.y), s * (x.y + y.x));
  }
  dft<M, 1>(v);
#pragma unroll
  for (int r = 0; r < M; r++) sm[r * 17 + t] = r ? twid<1>(v[r], tw, t * r) : v[r];
}
template <int N> __device__ __forceinline__ void rows_out(float2 (&w)[16], int r, const float2* sm) {
#pragma unroll
  for (int q = 0; q < 16; q++) w[q] = sm[r * 17 + q];
  dft<16, 1>(w);
}

struct RowArgs {
  const float2* in[3];
  float* out[3];
  int pow[3];             // power of f_x
  const float2* tw;
  int hp;
};

// half rows -> real rows, one field per blockIdx.y
template <int N>
__global__ void __launch_bounds__(kLanes<N>* kPairs<N>, 3) row_kernel(const __grid_constant__ RowArgs a) {
  constexpr int M = kM<N>;
  __shared__ float2 smem[kPairs<N> * kRowSm<N>];
  const int t = threadIdx.x % kLanes<N>, pr = threadIdx.x / kLanes<N>;
  const int64_t row = 2 * ((int64_t)blockIdx.x * kPairs<N> + pr);   // rows row, row + 1
  const bool live = row < (int64_t)N * N;
  float2* sm = smem + pr * kRowSm<N>;
  const int f = blockIdx.y;
  if (live && t < 16) {
    float2 v[M];
    const float2* A = a.in[f] + row * a.hp;
    rows_in<N>(v, t, A, A + a.hp, a.pow[f], sm, a.tw);
  }
  __syncthreads();
  if (live && t < M) {
    float2 w[16];
    rows_out<N>(w, t, sm);
    float* o = a.out[f] + row * N + t;
#pragma unroll
    for (int s = 0; s < 16; s++) {
      o[M * s] = w[s].x;
      o[N + M * s] = w[s].y;
    }
  }
}

struct SrcArgs {
  const float2* o[6];     // Ty: g, f_y g, f_y^2 g, (f_z g), f_y (f_z g), f_z^2 g (null: from the trace)
  const float* delta;
  float2* out;            // the source's spectrum after the x pass
  const float2* tw;
  int hp;
};

// The x pass of 2LPT: phi rows to real space, the source, its forward row
// transform.  TRACE: phi_33 = -(delta + phi_11 + phi_22) and the source
// phi_11 phi_22 - phi_12^2 + ... of LPT.jl:141-143; else six phi and the
// trace-identity source delta^2/2 - sum phi_aa^2/2 - sum phi_ab^2 of
// MultiResolution.jl:804-831.  Registers hold one running value per x.
template <int N, bool TRACE>
__global__ void __launch_bounds__(kLanes<N>* kPairs<N>, 2) src2_rows_kernel(const __grid_constant__ SrcArgs a) {
  constexpr int M = kM<N>;
  __shared__ float2 smem[kPairs<N> * kRowSm<N>];
  const int t = threadIdx.x % kLanes<N>, pr = threadIdx.x / kLanes<N>;
  const int64_t row = 2 * ((int64_t)blockIdx.x * kPairs<N> + pr);
  const bool live = row < (int64_t)N * N;
  float2* sm = smem + pr * kRowSm<N>;
  float2 acc[16];
  // powers of f_x per array: phi_11 2, phi_12 1, phi_22 0, phi_13 1, phi_23 0, phi_33 0;
  // taken in the order 11, 22, (33,) 12, 13, 23
  for (int f = 0; f < (TRACE ? 5 : 6); f++) {
    const int id = TRACE ? (f == 0 ? 0 : f == 1 ? 2 : f == 2 ? 1 : f) : (f == 0 ? 0 : f == 1 ? 2 : f == 2 ? 5 : f == 3 ? 1 : f - 1);
    if (live && t < 16) {
      float2 v[M];
      const float2* A = a.o[id] + row * a.hp;
      rows_in<N>(v, t, A, A + a.hp, id == 0 ? 2 : (id == 1 || id == 3) ? 1 : 0, sm, a.tw);
    }
    __syncthreads();
    if (live && t < M) {
      float2 w[16];
      rows_out<N>(w, t, sm);
      if (TRACE) {
        if (f == 0) {
#pragma unroll
          for (int s = 0; s < 16; s++) acc[s] = w[s];
        } else if (f == 1) {
          const float* d = a.delta + row * N + t;
#pragma unroll
          for (int s = 0; s < 16; s++) {   // ab + (a + b) c, c = -(delta + a + b)
            const float sx = acc[s].x + w[s].x, sy = acc[s].y + w[s].y;
            const float cx = -(__ldg(d + M * s) + sx), cy = -(__ldg(d + N + M * s) + sy);
            acc[s].x = fmaf(acc[s].x, w[s].x, sx * cx);
            acc[s].y = fmaf(acc[s].y, w[s].y, sy * cy);
          }
        } else {
#pragma unroll
          for (int s = 0; s < 16; s++) {
            acc[s].x = fmaf(-w[s].x, w[s].x, acc[s].x);
            acc[s].y = fmaf(-w[s].y, w[s].y, acc[s].y);
          }
        }
      } else {
        if (f == 0) {
          const float* d = a.delta + row * N + t;
#pragma unroll
          for (int s = 0; s < 16; s++) {
            const float dx = __ldg(d + M * s), dy = __ldg(d + N + M * s);
            acc[s] = make_float2(0.5f * dx * dx, 0.5f * dy * dy);
          }
        }
        const float h = f < 3 ? 0.5f : 1.f;
#pragma unroll
        for (int s = 0; s < 16; s++) {
          acc[s].x = fmaf(-h * w[s].x, w[s].x, acc[s].x);
          acc[s].y = fmaf(-h * w[s].y, w[s].y, acc[s].y);
        }
      }
    }
    __syncthreads();
  }
  // forward: thread r holds x = r + M s; DFT over s, twiddle, then across r
  constexpr int P = M | 1;
  if (live && t < M) {
    dft<16, -1>(acc);
#pragma unroll
    for (int q = 0; q < 16; q++) sm[q * P + t] = q ? twid<-1>(acc[q], a.tw, t * q) : acc[q];
  }
  __syncthreads();
  float2 v[M];
  if (live && t < 16) {
#pragma unroll
    for (int r = 0; r < M; r++) v[r] = sm[t * P + r];
    dft<M, -1>(v);
  }
  __syncthreads();
  if (live && t < 16)
#pragma unroll
    for (int p = 0; p < M; p++) sm[t + 16 * p] = v[p];
  __syncthreads();
  if (live) {   // the two rows' half spectra from C[k] and conj C[N - k]
    float2* A = a.out + row * a.hp;
    float2* B = A + a.hp;
    for (int k = t; k <= N / 2; k += kLanes<N>) {
      const float2 x = sm[k], y = sm[k ? N - k : 0];
      A[k] = make_float2(0.5f * (x.x + y.x), 0.5f * (x.y - y.y));
      B[k] = make_float2(0.5f * (x.y + y.y), 0.5f * (y.x - x.x));
    }
  }
}

struct TwinArgs {
  const float2* w[kTwinGroup];   // z/y-transformed twins of filters f0, f0 + 1, ... in [z][y][kx] order
  int flim[kTwinGroup];
  const float2* tw;
  int n, hp, n1, n2, fbits, f0;
  const int64_t* woff;
  const int* first;
  PeakBuf pb;
};
// the twin at the peaks a group of filters appended (slots *first .. count -
// 1): sum over kx of c_k Re(L[kx] w^(kx x)), c = 1 at kx = 0 and n/2, else 2;
// one warp per peak, FP64 sum.  A peak's row is one contiguous run.  The
// key's window number (above fbits) gives the window's first cell on the n^3
// grid.
__global__ void __launch_bounds__(256) twin_rows_kernel(const __grid_constant__ TwinArgs a) {
  const int end = (int)min((int64_t)*a.pb.count, a.pb.cap);
  const int l = threadIdx.x & 31;
  const int nw = gridDim.x * (blockDim.x / 32);
  const int n = a.n, H = n / 2;
  for (int p = *a.first + blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); p < end; p += nw) {
    const unsigned long long key = a.pb.keys[p];
    const int64_t loc = (int64_t)(key & ((1ull << 40) - 1));
    const int g = (int)((key >> 40) & ((1ull << a.fbits) - 1)) - a.f0;
    const int64_t ljk = loc / a.n1;
    const int li = (int)(loc - ljk * a.n1), lk = (int)(ljk / a.n2), lj = (int)(ljk - (int64_t)lk * a.n2);
    const int64_t cell = (a.woff ? a.woff[key >> (40 + a.fbits)] : 0) + li + (int64_t)n * (lj + (int64_t)n * lk);
    const int64_t row = cell / n;
    const int x = (int)(cell - row * n);
    const float2* r = a.w[g] + row * a.hp;
    const int klim = a.flim[g];
    double acc = 0.0;
#pragma unroll 4
    for (int k = l; k <= klim; k += 32) {
      const float2 v = __ldg(r + k);
      const float2 t = __ldg(a.tw + (k * x) % n);   // k x < 2^18
      const double term = (double)v.x * t.x - (double)v.y * t.y;
      acc += (k == 0 || k == H) ? term : 2.0 * term;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (l == 0) a.pb.lap[p] = (float)acc;
  }
}

// ---------------------------------------------------------------------------
// launches by size
// ---------------------------------------------------------------------------
template <int N> constexpr size_t col_smem() { return (size_t)N * kColW * sizeof(float2); }

template <int N> void prepare_n() {
  const int b = (int)col_smem<N>();
  PPB_CUDA(cudaFuncSetAttribute(col_kernel<N, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  PPB_CUDA(cudaFuncSetAttribute(col_kernel<N, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  PPB_CUDA(cudaFuncSetAttribute(mid_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
}
template <int N, int SIGN> void col_n(Launch L, const ColArgs& a, int planes) {
  const dim3 grid((unsigned)((a.fmax + kColW) / kColW * a.nout), (unsigned)planes);
  col_kernel<N, SIGN><<<grid, kColW * kLanes<N>, col_smem<N>(), L.s>>>(a);
  PPB_LAUNCHED(*L.count);
}
template <int N> constexpr unsigned row_blocks() { return (unsigned)((N * N / 2 + kPairs<N> - 1) / kPairs<N>); }

ColArgs col_args(const float2* tw, int n, int fmax) {
  ColArgs a{};
  a.tw = tw;
  a.fmax = fmax;
  a.hp_in = a.hp = fft_pitch(n);
  return a;
}
template <int N> void zcol(Launch L, ColArgs a) {   // from cuFFT's layout; plane index iy, column along z
  a.hp_in = N / 2 + 1;
  a.js_in = (int64_t)N * a.hp_in;
  a.js = (int64_t)N * a.hp;
  a.bs_in = a.hp_in;
  a.bs = a.hp;
  a.zpass = 1;
  col_n<N, 1>(L, a, a.fmax < N / 2 ? 2 * a.fmax + 1 : N);
}
template <int N, int SIGN> void ycol(Launch L, ColArgs a) {   // plane index iz, column along y
  a.js_in = a.js = a.hp;
  a.bs_in = a.bs = (int64_t)N * a.hp;
  col_n<N, SIGN>(L, a, N);
}

template <int N>
void lpt2_n(Launch L, const float2* dk, const float* delta, float2* const* w, const float2* tw, float* psi2,
            double box, bool trace) {
  const double ps = 1.0 / ((double)N * N * N);
  // z: g = -ps delta / q, f_z g (, f_z^2 g)
  ColArgs z = col_args(tw, N, N / 2);
  z.kind = 1;
  z.ps = pair_of(-ps);
  z.zero_nyq = !trace;
  z.nout = trace ? 2 : 3;
  for (int o = 0; o < z.nout; o++) z.o[o] = ColOut{dk, w[6 + o], o, N / 2};
  zcol<N>(L, z);
  // y: g, f_y g, f_y^2 g, (f_z g), f_y (f_z g) (, f_z^2 g)
  ColArgs y = col_args(tw, N, N / 2);
  y.nout = trace ? 5 : 6;
  for (int o = 0; o < y.nout; o++) y.o[o] = ColOut{w[o < 3 ? 6 : o < 5 ? 7 : 8], w[o], o < 3 ? o : o < 5 ? o - 3 : 0, N / 2};
  ycol<N, 1>(L, y);
  SrcArgs s{};
  for (int o = 0; o < y.nout; o++) s.o[o] = w[o];
  s.delta = delta;
  s.out = w[6];
  s.tw = tw;
  s.hp = fft_pitch(N);
  if (trace) src2_rows_kernel<N, true><<<row_blocks<N>(), kLanes<N> * kPairs<N>, 0, L.s>>>(s);
  else src2_rows_kernel<N, false><<<row_blocks<N>(), kLanes<N> * kPairs<N>, 0, L.s>>>(s);
  PPB_LAUNCHED(*L.count);
  ColArgs f = col_args(tw, N, N / 2);
  f.nout = 1;
  f.o[0] = ColOut{w[6], w[7], 0, N / 2};
  ycol<N, -1>(L, f);
  // psi2_c = -i k_c / k^2 src2_k: k_c / k^2 = f_c / (q dk)
  MidArgs m{w[7], w[0], w[1], tw, pair_of(ps * box / (2.0 * 3.141592653589793)), fft_pitch(N)};
  mid_kernel<N><<<dim3((unsigned)((N / 2 + kColW) / kColW), (unsigned)N), kColW * kLanes<N>, col_smem<N>(), L.s>>>(m);
  PPB_LAUNCHED(*L.count);
  ColArgs v = col_args(tw, N, N / 2);
  v.nout = 3;
  v.o[0] = ColOut{w[0], w[2], 0, N / 2};
  v.o[1] = ColOut{w[0], w[3], 1, N / 2};
  v.o[2] = ColOut{w[1], w[4], 0, N / 2};
  ycol<N, 1>(L, v);
  RowArgs x{};
  x.tw = tw;
  x.hp = fft_pitch(N);
  for (int c = 0; c < 3; c++) {
    x.in[c] = w[2 + c];
    x.out[c] = psi2 + (int64_t)c * N * N * N;
    x.pow[c] = c == 0 ? 1 : 0;
  }
  row_kernel<N><<<dim3(row_blocks<N>(), 3), kLanes<N> * kPairs<N>, 0, L.s>>>(x);
  PPB_LAUNCHED(*L.count);
}

// z and y transforms of dk with the transfer `kind` into `cnt` arrays w, for
// kind 3 with one window table (wstride floats apart) and frequency limit each
template <int N>
void zy_n(Launch L, const float2* dk, float2* const* w, int cnt, const float2* tw, int kind, double ps,
          const float* win, int64_t wstride, bool zero_nyq, const int* flim) {
  int fmax = 0;
  for (int i = 0; i < cnt; i++) fmax = flim[i] > fmax ? flim[i] : fmax;
  ColArgs z = col_args(tw, N, fmax);
  z.win = win;
  z.wstride = wstride;
  z.nout = cnt;
  z.kind = kind;
  z.ps = pair_of(ps);
  z.zero_nyq = zero_nyq;
  for (int i = 0; i < cnt; i++) z.o[i] = ColOut{dk, w[i], 0, flim[i]};
  zcol<N>(L, z);
  ColArgs y = col_args(tw, N, fmax);
  y.nout = cnt;
  for (int i = 0; i < cnt; i++) y.o[i] = ColOut{w[i], w[i], 0, flim[i]};   // in place: a block reads its columns first
  ycol<N, 1>(L, y);
}

template <int N> void rows_n(Launch L, const float2* w, float* out, const float2* tw) {
  RowArgs x{};
  x.tw = tw;
  x.hp = fft_pitch(N);
  x.in[0] = w;
  x.out[0] = out;
  row_kernel<N><<<row_blocks<N>(), kLanes<N> * kPairs<N>, 0, L.s>>>(x);
  PPB_LAUNCHED(*L.count);
}

// every multiple of 16 up to 384, the largest tile of the workloads, and the
// two larger sizes of the fused x pass (k_xpeak.cu); a size adds about 0.3 MB
// to the library and 5 s to the build, and the others take cuFFT
#define PPB_FFT_SIZES(X) \
  X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19) X(20) X(21) X(22) \
  X(23) X(24) X(28) X(32)

}  // namespace

bool fft_supported(int n) {
  if (n % 16) return false;
  switch (n / 16) {
#define X(m) case m:
    PPB_FFT_SIZES(X)
#undef X
    return true;
    default: return false;
  }
}

int fft_pitch(int n) { return (n / 2 + 1 + 3) & ~3; }
int64_t fft_work_elems(int n) { return (int64_t)n * n * fft_pitch(n); }

void fft_prepare(int n) {
  switch (n / 16) {
#define X(m) case m: prepare_n<16 * m>(); break;
    PPB_FFT_SIZES(X)
#undef X
    default: break;
  }
}

void launch_lpt2_fused(Launch L, const float2* dk, const float* delta, float2* const* w, const float2* tw, float* psi2,
                       int n, double box, bool trace) {
  switch (n / 16) {
#define X(m) case m: lpt2_n<16 * m>(L, dk, delta, w, tw, psi2, box, trace); break;
    PPB_FFT_SIZES(X)
#undef X
    default: PPB_REQUIRE(false, "fused 2LPT: unsupported grid size");
  }
}

void launch_laplacian_fused(Launch L, const float2* dk, float2* w, const float2* tw, float* out, int n, double scale,
                            bool zero_nyq) {
  const int half = n / 2;
  switch (n / 16) {
#define X(m) \
  case m: \
    zy_n<16 * m>(L, dk, &w, 1, tw, 2, scale, nullptr, 0, zero_nyq, &half); \
    rows_n<16 * m>(L, w, out, tw); \
    break;
    PPB_FFT_SIZES(X)
#undef X
    default: PPB_REQUIRE(false, "fused Laplacian: unsupported grid size");
  }
}

int twin_flim(int n, double box, double Rf) {
  // W_3 = k^2 exp(-(k Rf)^2 / 8) is largest at k Rf = sqrt(8); at 15 it is
  // 4.6e-11 of that (at 13 3.8e-8).  The single-precision forward transform
  // spreads a rounding of about 1e-7 of the field's rms amplitude over every
  // mode kept; even for a field with all its power just beyond the cut that is
  // some fifty times what the modes dropped there would add
  const double f = 15.0 * box / (6.283185307179586 * Rf);
  return f >= n / 2 ? n / 2 : (int)f + 1;
}

void launch_twin_zy(Launch L, const float2* dk, float2* const* w, int cnt, const float2* tw, int n, const float* tab,
                    int64_t tab_stride, float ps, const int* flim) {
  switch (n / 16) {
#define X(m) \
  case m: \
    zy_n<16 * m>(L, dk, w, cnt, tw, 3, ps, tab, tab_stride, false, flim); \
    break;
    PPB_FFT_SIZES(X)
#undef X
    default: PPB_REQUIRE(false, "twin transform: unsupported grid size");
  }
}

void launch_twin_rows(Launch L, float2* const* w, int cnt, const float2* tw, int n, const int* flim, int n1, int n2,
                      int fbits, int f0, const int64_t* woff, const int* first, PeakBuf pb) {
  TwinArgs a{};
  for (int i = 0; i < cnt; i++) {
    a.w[i] = w[i];
    a.flim[i] = flim[i];
  }
  a.tw = tw;
  a.n = n;
  a.hp = fft_pitch(n);
  a.n1 = n1;
  a.n2 = n2;
  a.fbits = fbits;
  a.f0 = f0;
  a.woff = woff;
  a.first = first;
  a.pb = pb;
  twin_rows_kernel<<<148 * 4, 256, 0, L.s>>>(a);
  PPB_LAUNCHED(*L.count);
}

}  // namespace ppb
