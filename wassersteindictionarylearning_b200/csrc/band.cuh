// Banded evaluation of the separable Gaussian along lines held in SMEM (the
// CUDA-core operator's inner computation, sinkhorn_band.cu).
//
// The reference contracts every line with the dense C x C factor
// G[c][k] = max(EPSILON, exp(-(c-k)^2/gamma)) (cpp/kernels.h:637-640, :669-699).
// Its entries fall off so fast that only a narrow band reaches the result's
// rounding: at gamma = 2 px^2, 19 of the 64..256 taps of a line in FP32.  A
// warp therefore sums taps c-r..c+r only, with r chosen from the data: with
// X >= max_k |x_k| over the block's lines and m = the smallest |x_c| over the
// outputs of the warp, the taps left out add at most 2 C g(r+1) X to an output
// that holds the term g(0) x_c >= m, and r is the smallest distance with
//   2 C g(r+1) X <= 2^-kTail m
// (kTail = 40 bits for FP32, 60 for FP64: 2^-16 and 2^-8 of the arithmetic's own
// rounding of that one term).  FP32 entries beyond the factor's reach are
// exactly zero, which bounds r there; FP64 entries never fall below EPSILON,
// so r is the whole line once EPSILON X could matter.  An output that is exactly
// zero in FP64 takes the whole line, and a block with a value that is not
// finite the whole line in FP64, all of the factor's reach in FP32 and then the
// zeros beyond it, eight outputs at a time: infinities, NaN and zeros meet
// as in the dense product.  A result depends on its block's lines only, never on the
// grid of the launch.
//
// Lines are held as 8-byte elements: one FP64 line, or two FP32 lines
// interleaved, whose sums advance together on the packed FP32 multiply-add
// (half the issue slots of the sums).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace wdl {
namespace band {

template <typename T>
struct Vec;
template <>
struct Vec<float> {
  using V = unsigned long long;  // two lines' values
  static constexpr int W = 2, kTail = 40, kInfExp = 255;
  __device__ static V fma(V a, V b, V c) {
    V d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
  }
  __device__ static V make(const float (&v)[2]) {
    V d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(v[0]), "f"(v[1]));
    return d;
  }
  __device__ static V dup(float x) {
    const float v[2] = {x, x};
    return make(v);
  }
  __device__ static void split(V d, float (&v)[2]) { asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(d)); }
  // Running largest and smallest magnitudes of pairs: the largest keeps a NaN.
  using M = float;
  static constexpr float kNoMin = 3.402823466e38f;
  __device__ static M up(M m, const float (&v)[2]) {
    asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(fabsf(v[0])), "f"(fabsf(v[1])));
    return m;
  }
  __device__ static M down(M m, const float (&v)[2]) {
    asm("min.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(fabsf(v[0])), "f"(fabsf(v[1])));
    return m;
  }
  __device__ static bool finite(M m) { return m <= 3.402823466e38f; }
  // magnitude bits: ordered like |x|, NaN above infinity
  __device__ static int bits(M m) { return __float_as_int(m); }
  __device__ static int expo(int b) { return b >> 23; }
};
template <>
struct Vec<double> {
  using V = double;
  static constexpr int W = 1, kTail = 60, kInfExp = 2047;
  __device__ static V fma(V a, V b, V c) { return ::fma(a, b, c); }
  __device__ static V make(const double (&v)[1]) { return v[0]; }
  __device__ static V dup(double x) { return x; }
  __device__ static void split(V d, double (&v)[1]) { v[0] = d; }
  using M = int;
  static constexpr int kNoMin = 0x7fefffff;
  __device__ static M up(M m, const double (&v)[1]) { return max(m, __double2hiint(v[0]) & 0x7fffffff); }
  __device__ static M down(M m, const double (&v)[1]) { return min(m, __double2hiint(v[0]) & 0x7fffffff); }
  __device__ static bool finite(M m) { return m < 0x7ff00000; }
  __device__ static int bits(M m) { return m; }
  __device__ static int expo(int b) { return b >> 20; }
};

// Zeros between two lines in SMEM (and before the first): taps up to this far
// outside a line need no test.
constexpr int kPad = 16;

// One axis of the factor: entries g[0..C), and the constants of the radius.
template <typename T>
struct Axis {
  const T* g;    // first row of the axis's factor: g[d] = max(EPSILON, exp(-d^2/gamma))
  int C;         // line length
  int C8;        // C rounded up to a multiple of 8 (lines are zero-padded to it)
  int G;         // C8 / 8 groups of eight outputs
  int pitch;     // elements between lines in SMEM
  int reach;     // FP32: largest distance with a non-zero entry
  int base;      // kTail + 2 + log2(C)
  int most;      // FP64: largest exponent difference at which EPSILON X stays negligible
  float k1;      // gamma ln 2
  int ext;       // the table in SMEM holds |d| < ext (and d = -ext)
  int lim[4];    // largest exponent differences served by radii 4, 8, 12, 16 (FP32: any, from the reach on)
};

// The pitch is an odd number of 16-byte units, so that eight neighbouring
// lines read at one position by 16-byte accesses fall in different banks.
__host__ __device__ inline int line_pitch(int C) { return ((C + 7) & ~7) + kPad + 2; }

// SMEM of a table and a block of lines, in 8-byte elements.
template <typename T>
__host__ __device__ inline int table_elems(const Axis<T>& ax) { return 2 * ax.ext; }
template <typename T>
__host__ __device__ inline int lines_elems(const Axis<T>& ax, int lines) { return kPad + lines * ax.pitch; }

// Factor table: g[|d|] for d = -ext .. ext - 1 (once per interleaved line).
template <typename T>
__device__ __forceinline__ const typename Vec<T>::V* load_table(const Axis<T>& ax, typename Vec<T>::V* tab, int tid,
                                                                int nthreads) {
  for (int i = tid; i < 2 * ax.ext; i += nthreads) {
    const int d = abs(i - ax.ext);
    tab[i] = Vec<T>::dup(d < ax.C ? ax.g[d] : T(0));
  }
  return tab + ax.ext;
}

__device__ __forceinline__ void st2(unsigned long long* p, unsigned long long a, unsigned long long b) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(a, b);
}
__device__ __forceinline__ void st2(double* p, double a, double b) {
  *reinterpret_cast<double2*>(p) = make_double2(a, b);
}

// Zeros around the lines of a block of lines (S: its first line).
template <typename T>
__device__ __forceinline__ void zero_pads(const Axis<T>& ax, typename Vec<T>::V* S, int lines, int tid,
                                          int nthreads) {
  using V = typename Vec<T>::V;
  constexpr int kQ = (kPad + 2) / 2;
  if (tid < kPad / 2) st2(S - kPad + 2 * tid, V(0), V(0));
  for (int i = tid; i < lines * kQ; i += nthreads) {
    const int l = i / kQ;
    st2(S + l * ax.pitch + ax.C8 + 2 * (i - l * kQ), V(0), V(0));
  }
}

// Radius, rounded up to a multiple of 4, of outputs whose smallest centre magnitude
// is `m`, in lines bounded by `x` (both as Vec::bits).  C8 - 8 reaches every
// input from every group.
template <typename T>
__device__ __forceinline__ int radius4(const Axis<T>& ax, int m, int x) {
  const int em = Vec<T>::expo(m), ex = Vec<T>::expo(x);
  const int diff = em == 0 || ex == Vec<T>::kInfExp ? 1 << 20 : ex + 1 - em;
  int r;
  if (diff <= ax.lim[2]) {
    r = diff <= ax.lim[0] ? 4 : diff <= ax.lim[1] ? 8 : 12;
  } else if (diff <= ax.lim[3]) {
    r = 16;
  } else if (ex == Vec<T>::kInfExp || (sizeof(T) == 8 && diff > ax.most)) {
    r = ax.C8;
  } else {
    const float f = ceilf(sqrtf(ax.k1 * (float)(ax.base + diff)));
    r = ((int)fminf(f, (float)(sizeof(T) == 8 ? ax.C8 : ax.reach)) + 3) & ~3;
  }
  return min(r, ax.C8 - 8);
}

__device__ __forceinline__ void ld2(unsigned long long (&v)[4], int at, const unsigned long long* p) {
  const ulonglong2 f = *reinterpret_cast<const ulonglong2*>(p);
  v[at] = f.x; v[at + 1] = f.y;
}
__device__ __forceinline__ void ld2(double (&v)[4], int at, const double* p) {
  const double2 f = *reinterpret_cast<const double2*>(p);
  v[at] = f.x; v[at + 1] = f.y;
}
template <typename V>
__device__ __forceinline__ void ld4(V (&v)[4], const V* p) {
  ld2(v, 0, p);
  ld2(v, 2, p + 2);
}
template <typename V>
__device__ __forceinline__ void st8(V* p, const V (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 8; q += 2) st2(p + q, v[q], v[q + 1]);
}

// acc[j] += sum over the four inputs x[i] at distance d = D + j - i, the table
// window lo = g[D-4..D-1], mid = g[D..D+3], hi = g[D+4..D+7].
template <typename T, typename V>
__device__ __forceinline__ void fir_block(V (&acc)[8], const V (&x)[4], const V (&lo)[4], const V (&mid)[4],
                                          const V (&hi)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int q = j - i;
      acc[j] = Vec<T>::fma(x[i], q < 0 ? lo[q + 4] : q < 4 ? mid[q] : hi[q - 4], acc[j]);
    }
}

// Outputs c0..c0+7 of one line (c0 a multiple of 8), taps within r4 (a multiple
// of 4, uniform over the warp) of each, in ascending order.  Eight outputs per
// thread: per four inputs, two 16-byte loads of the line and two (broadcast) of
// the table feed 32 multiply-adds, which leaves the arithmetic, not shared
// memory, as the limit.  GUARD: taps may lie beyond the padding.
template <typename T, bool GUARD>
__device__ __forceinline__ void fir8(const typename Vec<T>::V* line, const typename Vec<T>::V* g, int c0, int C8,
                                     int r4, typename Vec<T>::V (&acc)[8]) {
  using V = typename Vec<T>::V;
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = V(0);
  int D = r4;
  V w0[4], w1[4], w2[4], x[4];
  ld4(w1, g + D);
  ld4(w2, g + D + 4);
  const int last = -(r4 + 4);  // the block of inputs c0 + r4 + 4 .. c0 + r4 + 7
  int kb = c0 - D;
  const V* lp = line + kb;
  const V* gp = g + D - 4;
  while (true) {
    ld4(w0, gp);
    if (!GUARD || (kb >= 0 && kb < C8)) {
      ld4(x, lp);
      fir_block<T>(acc, x, w0, w1, w2);
    }
    if (D == last) break;
    ld4(w2, gp - 4);
    if (!GUARD || (kb + 4 >= 0 && kb + 4 < C8)) {
      ld4(x, lp + 4);
      fir_block<T>(acc, x, w2, w0, w1);
    }
    if (D - 4 == last) break;
    ld4(w1, gp - 8);
    if (!GUARD || (kb + 8 >= 0 && kb + 8 < C8)) {
      ld4(x, lp + 8);
      fir_block<T>(acc, x, w1, w2, w0);
    }
    if (D - 8 == last) break;
    D -= 12;
    gp -= 12;
    lp += 12;
    kb += 12;
  }
}

// The sum of a block with a value that is not finite, FP32: all of the table's
// taps, then the zeros beyond them, whose product with that value is NaN, as in
// the dense sum.  Outputs whose own inputs are all NaN, as every line's are soon
// after a scaling left the range, are NaN at once (256 x 256, 16 histograms, an
// evaluation that overflows: dense, with the factor from global memory, 50 ms;
// without this 17; with it 5.2).  Two inputs at a time in a small loop: written with
// fir8 (in line, as a call, or as a loop of its own) it cost the finite lines
// beside it 2 to 4 %.
template <typename T>
__device__ __forceinline__ void far8(const typename Vec<T>::V* line, const typename Vec<T>::V* g, const Axis<T>& ax,
                                     int c0, typename Vec<T>::V (&acc)[8]) {
  using V = typename Vec<T>::V;
  bool none = true;  // no output with a number of its own
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    acc[j] = line[c0 + j];
    T v[Vec<T>::W];
    Vec<T>::split(acc[j], v);
    none = none && (c0 + j >= ax.C || (v[0] != v[0] && v[Vec<T>::W - 1] != v[Vec<T>::W - 1]));
  }
  if (none) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = V(0);
  V z = V(0);
  const int lo = c0 + 8 - ax.ext, hi = c0 + ax.ext - 1;  // inputs whose eight entries the table holds
#pragma unroll 1
  for (int k = 0; k < ax.C8; k += 2) {
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(line + k);
    if (k >= lo && k < hi) {
      ulonglong2 w[5];  // g[c0 - k - 2 .. c0 - k + 7]
#pragma unroll
      for (int q = 0; q < 5; ++q) w[q] = *reinterpret_cast<const ulonglong2*>(g + (c0 - k - 2 + 2 * q));
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int a = j + 2, b = j + 1;  // distances c0 + j - k and c0 + j - k - 1
        acc[j] = Vec<T>::fma(x.x, (a & 1) ? w[a / 2].y : w[a / 2].x, acc[j]);
        acc[j] = Vec<T>::fma(x.y, (b & 1) ? w[b / 2].y : w[b / 2].x, acc[j]);
      }
    } else {
      z = Vec<T>::fma(x.x, V(0), z);
      z = Vec<T>::fma(x.y, V(0), z);
    }
  }
  const V one = Vec<T>::dup(T(1));
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = Vec<T>::fma(z, one, acc[j]);
}

// Division of 0 <= i < 65536 by a number that the host knows.
struct Div {
  int n;
  uint32_t inv;
  __host__ static Div by(int n) { return {n, n > 1 ? 0xffffffffu / (uint32_t)n + 1u : 0u}; }
  __device__ __forceinline__ int operator()(int i) const { return n > 1 ? (int)__umulhi((uint32_t)i, inv) : i; }
};

// Items of one pass: the eight-output groups of nl lines, lanes over the lines
// first; warp w of nw takes items 32 w .. 32 w + 31, and so on.  pre(line, c0,
// ext) loads what the epilogue needs of global memory before the sums;
// sink(line, c0, acc, ext) takes the outputs (those at c >= C are to be
// dropped).  xmag bounds the lines.
template <typename T, int NE, class Pre, class Sink>
__device__ __forceinline__ void fir_lines(const typename Vec<T>::V* lines, const typename Vec<T>::V* g,
                                          const Axis<T>& ax, Div nl, int xmag, int warp, int nw, int lane, Pre pre,
                                          Sink sink) {
  using V = typename Vec<T>::V;
  constexpr int W = Vec<T>::W;
  const int items = nl.n * ax.G;
  for (int i0 = warp * 32; i0 < items; i0 += nw * 32) {
    const int it = i0 + lane;
    const bool ok = it < items;
    const int grp = ok ? nl(it) : 0, line = ok ? it - grp * nl.n : 0;
    const int c0 = grp * 8;
    const V* lp = lines + line * ax.pitch;
    T ext[NE > 0 ? NE : 1][8][W];
    if (NE > 0 && ok) pre(line, c0, ext);
    typename Vec<T>::M m = Vec<T>::kNoMin;
    const bool whole = c0 + 8 <= ax.C;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      V x[4];
      ld4(x, lp + c0 + 4 * q);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        T v[W];
        Vec<T>::split(x[j], v);
        if (whole || c0 + 4 * q + j < ax.C) m = Vec<T>::down(m, v);
      }
    }
    const int r4 = radius4(ax, (int)__reduce_min_sync(0xffffffffu, (unsigned)(ok ? Vec<T>::bits(m) : 0x7fffffff)), xmag);
    V acc[8];
    if constexpr (sizeof(T) == 8) {  // the table holds a whole line's taps
      if (r4 <= kPad) fir8<T, false>(lp, g, c0, ax.C8, r4, acc);
      else fir8<T, true>(lp, g, c0, ax.C8, r4, acc);
    } else {
      if (r4 <= kPad && r4 + 8 <= ax.ext) fir8<T, false>(lp, g, c0, ax.C8, r4, acc);
      else if (r4 + 8 <= ax.ext) fir8<T, true>(lp, g, c0, ax.C8, r4, acc);
      else far8<T>(lp, g, ax, c0, acc);
    }
    if (ok) sink(line, c0, acc, ext);
  }
}

// Largest magnitude of a block's lines: each warp leaves its maximum, and after
// the block's next barrier every thread reads the largest.
template <typename T>
__device__ __forceinline__ void put_mag(int* slots, typename Vec<T>::M v, int warp, int lane) {
  const int m = __reduce_max_sync(0xffffffffu, Vec<T>::bits(v));
  if (lane == 0) slots[warp] = m;
}
__device__ __forceinline__ int get_mag(const int* slots, int nw, int lane) {
  return __reduce_max_sync(0xffffffffu, lane < nw ? slots[lane] : 0);
}

}  // namespace band
}  // namespace wdl
