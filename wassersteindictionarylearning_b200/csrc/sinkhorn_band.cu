// The CUDA-core Sinkhorn evaluation in the kernel domain as two kinds of
// kernels per iteration, each between two transposes of the separable operator:
//
//   rows:    x pass -> phi -> geometric mean over the atoms -> b -> x pass
//   columns: y pass -> conv_b -> a = p / conv_b             -> y pass
//
// (cpp/inverseWasserstein.h:565-593).  A rows block holds the same rows of
// all K atoms of one histogram, a columns block some columns of one image, so
// every line is whole: each pass is the banded sum of band.cuh, and what lies
// between two passes never leaves the SM.  The reverse pass (:602-673) has
// the same shape, the dictionary and weight recursions side by side:
//
//   rows:    x pass -> v, r -> n, gw (sums over the atoms) -> tmp, u -> x pass
//   columns: y pass -> c / conv_b, -p c / conv_b^2         -> y pass
//
// Volumes add a y pass before and after the (then z) columns.  Per iteration
// and image the launches move 24 bytes per pixel forward and 2 x 22 backward in
// FP32, most of it within L2; b is recomputed from bary and phi, so the
// iterate store is conv_b, phi and one barycenter per histogram.
//
// Against dense axis passes (64 x 64 tiles, all C taps) with separate
// elementwise kernels, one B200: 64 histograms of 128 x 128, K = 5, L = 100,
// gamma 1, FP32 69.4 -> 20.3 ms an evaluation; 16 of 64 x 64, K = 4, L = 25, FP32
// 2.38 -> 0.84 ms (350 -> 100 launches); one of 161 x 161, K = 5, L = 50, FP64,
// weights only 10.9 -> 2.2 ms.  The dense passes spent 128 taps where 13 reach
// the FP32 rounding; here a quarter of the instructions at 128 x 128 are the sums'
// packed multiply-adds, the rest the logarithms, divisions, staging and addresses,
// and with 80 registers and 21 warps an SM their issue slots are 51 to 59 % busy: the latency
// of dependent instructions and of the loads before each sum bounds them, and for
// few histograms each launch's chain in one block an SM (9 to 17 % busy).  Tiles that
// lie inside the image and are whole groups of eight take a form without edge tests
// (24.4 -> 21.4 ms at 128 x 128).
//
// The blocks' shapes depend on the grid, K and the type only, so a
// histogram's results are the same bits in any batch.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "band.cuh"
#include "wdl_internal.cuh"
#include "wdl_math.cuh"

namespace wdl {
namespace {

using namespace band;

constexpr int kMaxThreads = 256, kMaxWarps = kMaxThreads / 32;
constexpr size_t kSmemMost = 200 * 1024;
// Atoms of one rows block (more: band_rows_pay's first figures).
constexpr int kMaxK = 32;

template <typename T>
const T* factor_row(const wdl_ctx* ctx, int axis);
template <>
const float* factor_row<float>(const wdl_ctx* ctx, int axis) { return ctx->G32[axis]; }
template <>
const double* factor_row<double>(const wdl_ctx* ctx, int axis) { return ctx->G64[axis]; }

template <typename T>
Axis<T> make_axis(const wdl_ctx* ctx, int axis) {
  Axis<T> ax;
  ax.g = factor_row<T>(ctx, axis);
  ax.C = ctx->axis_len[axis];
  ax.C8 = (ax.C + 7) & ~7;
  ax.G = ax.C8 / 8;
  ax.pitch = line_pitch(ax.C);
  ax.reach = ctx->axis_reach[axis];
  int lg = 0;
  while ((1 << lg) < ax.C) ++lg;
  ax.base = Vec<T>::kTail + 2 + lg;
  ax.most = 830 - ax.base;  // EPSILON = 1e-250 > 2^-831
  ax.k1 = (float)std::min(ctx->gamma * 0.6931471805599453, 1e30);
  // FP64 lines may need every entry (exact zeros), FP32 ones none past the reach
  ax.ext = sizeof(T) == 8 ? ax.C8 : std::min(ax.C8, ((std::max(ax.reach, 1) + 3) & ~3) + 8);
  for (int i = 0; i < 4; ++i) {
    const double r = 4.0 * (i + 1), d = std::floor(r * r / std::max((double)ax.k1, 1e-30)) - ax.base;
    ax.lim[i] = (int)std::min(std::max(d, -1.0), sizeof(T) == 8 ? (double)ax.most : 1e6);
    // the FP32 factor is zero past its reach: a radius that covers it serves every
    // difference, and none beyond it is taken (the table holds no more)
    if (sizeof(T) == 4 && 4 * (i + 1) >= ax.reach) ax.lim[i] = 1000000;
  }
  return ax;
}

// The radius that data of a few bits' spread take, and whether it covers every line.
template <typename T>
int few_bits_radius4(const Axis<T>& ax) {
  return ((int)std::ceil(std::min(std::sqrt((double)ax.k1 * (ax.base + 2)), 16384.0)) + 3) & ~3;
}
template <typename T>
bool covers_lines(const wdl_ctx* ctx) {
  for (int a = 0; a < ctx->ndim; ++a) {
    const Axis<T> ax = make_axis<T>(ctx, a);
    if (8 + 2 * few_bits_radius4(ax) < ax.C8) return false;
  }
  return true;
}

// Lines of a block: about 160 eight-output items per pass (a power of two of
// lines per atom, at least `least`), one item per thread where that fits.
// Small blocks keep every SM busy on one histogram's 64 x 64 images; at many
// histograms several share an SM.
inline int lines_per_block(int K, int G, int least) {
  int n = least;
  while (2 * n * K * G <= 160 && n < 16) n *= 2;
  return n;
}
inline int threads_for(int items) { return std::min(std::max((items + 31) & ~31, 64), kMaxThreads); }
// Columns: at least 8 elements, 64 bytes of global memory per row of the tile.
inline int cols_per_block(int G) { return lines_per_block(1, G, 8); }

template <typename T>
size_t band_smem(const Axis<T>& ax, int blocks, int lines) {
  return (size_t)(table_elems(ax) + blocks * lines_elems(ax, lines)) * 8;
}

// ---- shared pieces ------------------------------------------------------------------
// The kernels of an evaluation depend on one another in a chain.  Each lets the
// next one start once all its own blocks run, so that the next one's first
// blocks fill the SMs that the last blocks leave idle and have their tables
// ready; wait_previous then holds them until everything the chain wrote before
// is visible.  No global memory that another kernel of the chain touches is
// read or written before it.
__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// W global rows (contiguous, src0 and src1) into one zero-padded SMEM line, by one
// warp; m takes their magnitudes.  No input: ones.  Rows of whole 16-byte units
// are read four values at a time.
template <typename T, typename TI>
__device__ __forceinline__ void fill_row(typename Vec<T>::V* dst, const TI* __restrict__ src0,
                                         const TI* __restrict__ src1, const Axis<T>& ax, int lane,
                                         typename Vec<T>::M& m) {
  constexpr int W = Vec<T>::W;
  if (W == 2 && sizeof(TI) == 4 && src0 && (ax.C & 3) == 0) {
#pragma unroll 2
    for (int x = 4 * lane; x < ax.C8; x += 128) {
      float4 f[2] = {make_float4(0, 0, 0, 0), make_float4(0, 0, 0, 0)};
      if (x < ax.C) {
        f[0] = *reinterpret_cast<const float4*>(src0 + x);
        f[1] = *reinterpret_cast<const float4*>(src1 + x);
      }
      const float a[4][2] = {{f[0].x, f[1].x}, {f[0].y, f[1].y}, {f[0].z, f[1].z}, {f[0].w, f[1].w}};
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        typename Vec<T>::V v[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          T t[W];
          t[0] = (T)a[i + h][0];
          t[W - 1] = (T)a[i + h][1];
          m = Vec<T>::up(m, t);
          v[h] = Vec<T>::make(t);
        }
        st2(dst + x + i, v[0], v[1]);
      }
    }
    return;
  }
#pragma unroll 4
  for (int x = lane; x < ax.C8; x += 32) {
    T v[W];
#pragma unroll
    for (int c = 0; c < W; ++c) {
      const TI* s = c == 0 ? src0 : src1;
      v[c] = x < ax.C ? (s ? (T)s[x] : T(1)) : T(0);
    }
    m = Vec<T>::up(m, v);
    dst[x] = Vec<T>::make(v);
  }
}

// Eight consecutive values of one of the interleaved rows to global memory; FULL:
// whole 16-byte units, all eight inside the row.
__device__ __forceinline__ void put4(float* p, const float* v) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void put4(double* p, const double* v) {
  *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
  *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
}
template <bool FULL, typename T>
__device__ __forceinline__ void store_row8(T* __restrict__ dst, int c0, int C, const T (&v)[8]) {
  if (FULL) {
    put4(dst, v);
    put4(dst + 4, v + 4);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (c0 + j < C) dst[j] = v[j];
  }
}
// Outputs of a row item to rows r, r + 1 (those below `rows`) of an image.
template <bool FULL, typename T>
__device__ __forceinline__ void store_rows(T* __restrict__ img, int r, int rows, int c0, int C,
                                           const typename Vec<T>::V (&acc)[8]) {
  T v[Vec<T>::W][8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    T t[Vec<T>::W];
    Vec<T>::split(acc[j], t);
#pragma unroll
    for (int c = 0; c < Vec<T>::W; ++c) v[c][j] = t[c];
  }
  T* d = img + (uint32_t)(r * C + c0);
#pragma unroll
  for (int c = 0; c < Vec<T>::W; ++c)
    if (FULL || r + c < rows) store_row8<FULL>(d + c * C, c0, C, v[c]);
}

template <typename T>
struct NoExt {
  __device__ void operator()(int, int, T (&)[1][8][Vec<T>::W]) const {}
};

// Lines past the last row repeat it (their results are dropped): every block
// has the same number of lines, and a repeated line changes no other's radius.
template <typename T>
__device__ __forceinline__ const T* row_at(const T* img, int r, int rows, int C) {
  return img + (uint32_t)(min(r, rows - 1) * C);
}

// ---- the operator alone: x pass over rows ---------------------------------------------
template <typename TI, typename T>
__global__ void __launch_bounds__(kMaxThreads, 3) k_rows_op(Axis<T> ax, const TI* __restrict__ in,
                                                         T* __restrict__ out, int rows, Div n) {
  using V = typename Vec<T>::V;
  constexpr int W = Vec<T>::W;
  extern __shared__ __align__(16) unsigned char smem[];
  V* tab = reinterpret_cast<V*>(smem);
  V* S = tab + table_elems(ax) + kPad;
  __shared__ int mag[kMaxWarps];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nt = blockDim.x, nw = nt >> 5;
  const int r0 = blockIdx.x * n.n * W, C = ax.C;
  const size_t base = (size_t)blockIdx.y * rows * C;
  start_next();
  const V* g = load_table(ax, tab, tid, nt);
  zero_pads(ax, S, n.n, tid, nt);
  wait_previous();
  typename Vec<T>::M m = 0;
  for (int l = warp; l < n.n; l += nw) {
    const int r = r0 + l * W;
    const TI* s0 = in ? row_at(in + base, r, rows, C) : nullptr;
    fill_row<T>(S + l * ax.pitch, s0, in ? row_at(in + base, r + 1, rows, C) : nullptr, ax, lane, m);
  }
  put_mag<T>(mag, m, warp, lane);
  __syncthreads();
  const bool full = (C & 7) == 0 && r0 + n.n * W <= rows;
  const auto run = [&](auto f) {
    fir_lines<T, 0>(S, g, ax, n, get_mag(mag, nw, lane), warp, nw, lane, NoExt<T>(),
                    [&](int l, int c0, const V(&acc)[8], const T(&)[1][8][W]) {
                      store_rows<decltype(f)::value>(out + base, r0 + l * W, rows, c0, C, acc);
                    });
  };
  if (full) run(std::true_type());
  else run(std::false_type());
}

// ---- forward rows ---------------------------------------------------------------------
// x pass of t2 -> phi (stored); bary = exp(sum_k lambda_k log phi_k) (stored);
// b = bary / phi -> x pass -> t1 (cpp/inverseWasserstein.h:575-593).  t1 null:
// the last iteration.  Lines: atom by atom, the block's row groups of each.
template <typename T>
struct FwdRows {
  const T* t2;
  const double* lam;
  T *phi, *bary, *t1;
  int* range;
  int K, rows, nchunk;
  Div nv, nl, C;  // row groups of an atom, lines of the block, row length
};

template <typename T, int KT, bool FULL>
__device__ __forceinline__ void rows_fwd(const Axis<T>& ax, const FwdRows<T>& a, int p, int r0,
                                         typename Vec<T>::V* tab, int (*mag)[kMaxWarps], double* slam) {
  using V = typename Vec<T>::V;
  constexpr int W = Vec<T>::W;
  const int K = KT > 0 ? KT : a.K;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nt = blockDim.x, nw = nt >> 5;
  const int C = ax.C, rows = a.rows, nv = a.nv.n, nl = a.nl.n;
  const uint32_t N = (uint32_t)rows * C;
  const size_t pN = (size_t)p * N;
  V* S1 = tab + table_elems(ax) + kPad;
  V* S2 = S1 + lines_elems(ax, nl);
  const V* g = load_table(ax, tab, tid, nt);
  zero_pads(ax, S1, nl, tid, nt);
  wait_previous();
  for (int k = tid; k < K; k += nt) slam[k] = a.lam[(size_t)p * K + k];
  typename Vec<T>::M m = 0;
  const T* t2 = a.t2 + pN * K;
  for (int l = warp; l < nl; l += nw) {
    const int k = a.nv(l), r = r0 + (l - k * nv) * W;
    fill_row<T>(S1 + l * ax.pitch, row_at(t2 + k * N, r, rows, C), row_at(t2 + k * N, r + 1, rows, C), ax, lane, m);
  }
  put_mag<T>(mag[0], m, warp, lane);
  __syncthreads();
  fir_lines<T, 0>(S1, g, ax, a.nl, get_mag(mag[0], nw, lane), warp, nw, lane, NoExt<T>(),
                  [&](int l, int c0, const V(&acc)[8], const T(&)[1][8][W]) { st8(S2 + l * ax.pitch + c0, acc); });
  __syncthreads();
  m = 0;
  const int kstep = nv * ax.pitch;
  for (int e = tid; e < nv * C; e += nt) {
    const int v = a.C(e), x = e - v * C, r = r0 + v * W;
    const uint32_t j = (uint32_t)(min(r, rows - 1) * C + x);
    const bool ok0 = FULL || r < rows, ok1 = FULL || r + 1 < rows;
    V* s2 = S2 + v * ax.pitch + x;
    V* s1 = S1 + v * ax.pitch + x;
    T* pp = a.phi ? a.phi + pN * K + j : nullptr;
    double s[W];
#pragma unroll
    for (int c = 0; c < W; ++c) s[c] = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      T ph[W];
      Vec<T>::split(s2[k * kstep], ph);
      const double l = slam[k];
#pragma unroll
      for (int c = 0; c < W; ++c) {
        if (pp && (c ? ok1 : ok0)) pp[k * N + c * C] = ph[c];
        s[c] += acc_safe_log<T>(ph[c]) * l;
      }
    }
    T by[W];
#pragma unroll
    for (int c = 0; c < W; ++c) {
      by[c] = exp_from<T>(s[c]);
      if (a.bary && (c ? ok1 : ok0)) (a.bary + pN)[j + c * C] = by[c];
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      T b[W];
      Vec<T>::split(s2[k * kstep], b);
#pragma unroll
      for (int c = 0; c < W; ++c) b[c] = by[c] / b[c];
      m = Vec<T>::up(m, b);
      s1[k * kstep] = Vec<T>::make(b);
    }
  }
  if (a.range && !Vec<T>::finite(m)) a.range[p] = 1;
  if (!a.t1) return;
  put_mag<T>(mag[1], m, warp, lane);
  __syncthreads();
  T* t1 = a.t1 + pN * K;
  fir_lines<T, 0>(S1, g, ax, a.nl, get_mag(mag[1], nw, lane), warp, nw, lane, NoExt<T>(),
                  [&](int l, int c0, const V(&acc)[8], const T(&)[1][8][W]) {
                    const int k = a.nv(l), r = r0 + (l - k * nv) * W;
                    store_rows<FULL>(t1 + k * N, r, rows, c0, C, acc);
                  });
}

template <typename T, int KT>
__global__ void __launch_bounds__(kMaxThreads, 3) k_rows_fwd(Axis<T> ax, FwdRows<T> a) {
  start_next();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int mag[2][kMaxWarps];
  __shared__ double slam[kMaxK];
  const int p = blockIdx.x / a.nchunk, r0 = (blockIdx.x - p * a.nchunk) * a.nv.n * Vec<T>::W;
  auto* tab = reinterpret_cast<typename Vec<T>::V*>(smem);
  if ((ax.C & 7) == 0 && r0 + a.nv.n * Vec<T>::W <= a.rows) rows_fwd<T, KT, true>(ax, a, p, r0, tab, mag, slam);
  else rows_fwd<T, KT, false>(ax, a, p, r0, tab, mag, slam);
}

// ---- reverse rows -----------------------------------------------------------------------
// Round s's end and round s-1's start (cpp/inverseWasserstein.h:604-611,
// :619-627, :637-653, :661-669): x pass of t2 = [dictionary | weights] -> v = ./
// phi, r = . b (phi and b = bary / phi of the step), n = sum_k v, gw =
// sum_k r; then tmp = (lambda n - v) b, u = (lambda gw - r) / phi, the
// weight gradient's dot products, and the x pass -> t1.  FIRST: v = r = 0, n and
// gw come from the loss.  The dot products are kept per block (dotp) over the
// rounds and added up once.  Blocks past the last rows block add the round's
// c / conv_b over the histograms into the FP64 atom gradient.
template <typename T>
struct BwdRows {
  const T *t2, *n, *gw, *phi, *bary, *lam;
  T* t1;
  double* dotp;
  int K, P, rows, nchunk, nblocks, dict, want_u;
  Div nv, nl, C;
  size_t PKN;
  const T* q;
  double* gdic;
};

template <typename T, int KT, bool FIRST, bool FULL>
__device__ __forceinline__ void rows_bwd(const Axis<T>& ax, const BwdRows<T>& a, int p, int r0,
                                         typename Vec<T>::V* tab, int (*mag)[kMaxWarps], T* slam) {
  using V = typename Vec<T>::V;
  constexpr int W = Vec<T>::W, KR = KT > 0 ? KT : 1;
  const int K = KT > 0 ? KT : a.K;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nt = blockDim.x, nw = nt >> 5;
  const int rows = a.rows, C = ax.C, nv = a.nv.n, nl = a.nl.n;
  const uint32_t N = (uint32_t)rows * C;
  const size_t pN = (size_t)p * N;
  V* S1 = tab + table_elems(ax) + kPad;                // [dictionary, weights][K * n] lines
  const int half = nl * ax.pitch;                      // from the dictionary's lines to the weights'
  V* S2 = S1 + lines_elems(ax, 2 * nl);                // the same
  double* sdot = reinterpret_cast<double*>(S2 + 2 * half);  // [warp][K]
  const int q0 = a.dict ? 0 : 1;
  // the weights' items start on the warp after the dictionary's last
  const int warp_w = a.dict ? (warp + nw - ((nl * ax.G + 31) >> 5) % nw) % nw : warp;
  const V* g = load_table(ax, tab, tid, nt);
  for (int q = q0; q < 2; ++q) zero_pads(ax, S1 + q * half, nl, tid, nt);
  wait_previous();
  for (int k = tid; k < K; k += nt) slam[k] = a.lam[(size_t)p * K + k];
  if (KT == 0)
    for (int i = tid; i < nw * K; i += nt) sdot[i] = 0;
  if (!FIRST) {
    typename Vec<T>::M m[2] = {0, 0};
    for (int l2 = (q0 ? nl : 0) + warp; l2 < 2 * nl; l2 += nw) {
      const int q = l2 >= nl ? 1 : 0, l = l2 - q * nl;
      const int k = a.nv(l), r = r0 + (l - k * nv) * W;
      const T* t2 = a.t2 + (q * a.PKN + pN * K) + k * N;
      fill_row<T>(S1 + q * half + l * ax.pitch, row_at(t2, r, rows, C), row_at(t2, r + 1, rows, C), ax, lane, m[q]);
    }
    put_mag<T>(mag[0], m[0], warp, lane);
    put_mag<T>(mag[1], m[1], warp, lane);
    __syncthreads();
    for (int q = q0; q < 2; ++q)
      fir_lines<T, 0>(S1 + q * half, g, ax, a.nl, get_mag(mag[q], nw, lane), q ? warp_w : warp, nw, lane, NoExt<T>(),
                      [&](int l, int c0, const V(&acc)[8], const T(&)[1][8][W]) {
                        st8(S2 + q * half + l * ax.pitch + c0, acc);
                      });
    __syncthreads();
  } else {
    if (!FULL)  // the lines' ends
      for (int i = tid; i < 2 * nl * 8; i += nt) {
        const int l = i >> 3, x = ax.C8 - 8 + (i & 7);
        if (x >= C) S1[l < nl ? l * ax.pitch + x : half + (l - nl) * ax.pitch + x] = 0;
      }
    __syncthreads();
  }
  typename Vec<T>::M md = 0, mw = 0;
  double dot[KR];
#pragma unroll
  for (int k = 0; k < KR; ++k) dot[k] = 0;
  const int kstep = nv * ax.pitch;
  const T* phi = a.phi + pN * K;
  const T* bary = a.bary + pN;
  for (int e0 = warp * 32; e0 < nv * C; e0 += nt) {
    const bool in = e0 + lane < nv * C;
    const int e = in ? e0 + lane : 0;
    const int v = a.C(e), x = e - v * C, r = r0 + v * W;
    const bool ok0 = in && (FULL || r < rows), ok1 = in && (FULL || r + 1 < rows);
    const uint32_t up = FULL || r + 1 < rows ? C : 0;  // from the first row to the second
    const uint32_t j = (uint32_t)((FULL ? r : min(r, rows - 1)) * C + x);
    V* s1 = S1 + v * ax.pitch + x;
    V* s2 = S2 + v * ax.pitch + x;
    T ph[KR][W], bk[KR][W], by[W], sn[W], sg[W];
#pragma unroll
    for (int c = 0; c < W; ++c) {
      by[c] = bary[j + c * up];
      if (KT > 0) {
#pragma unroll
        for (int k = 0; k < KR; ++k) ph[k][c] = phi[k * N + j + c * up];
      }
      sn[c] = FIRST && a.dict ? (a.n + pN)[j + c * up] : T(0);
      sg[c] = FIRST ? (a.gw + pN)[j + c * up] : T(0);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      T h[W], b[W], vv[W], rv[W];
#pragma unroll
      for (int c = 0; c < W; ++c) {
        h[c] = KT > 0 ? ph[KT > 0 ? k : 0][c] : phi[k * N + j + c * up];
        b[c] = by[c] / h[c];
        if (KT > 0) bk[KT > 0 ? k : 0][c] = b[c];
      }
      if (!FIRST && in) {
        if (a.dict) {
          Vec<T>::split(s2[k * kstep], vv);
#pragma unroll
          for (int c = 0; c < W; ++c) sn[c] += vv[c] /= h[c];
          s2[k * kstep] = Vec<T>::make(vv);
        }
        Vec<T>::split(s2[half + k * kstep], rv);
#pragma unroll
        for (int c = 0; c < W; ++c) sg[c] += rv[c] *= b[c];
        s2[half + k * kstep] = Vec<T>::make(rv);
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const T l = slam[k];
      T h[W], b[W], t[W], u[W];
      double acc = 0;
#pragma unroll
      for (int c = 0; c < W; ++c) {
        h[c] = KT > 0 ? ph[KT > 0 ? k : 0][c] : phi[k * N + j + c * up];
        b[c] = KT > 0 ? bk[KT > 0 ? k : 0][c] : by[c] / h[c];
        t[c] = u[c] = T(0);
        if (c ? ok1 : ok0) acc += acc_log<T>(h[c]) * (double)sg[c];
      }
      if (in && a.dict) {
        if (!FIRST) Vec<T>::split(s2[k * kstep], t);
#pragma unroll
        for (int c = 0; c < W; ++c) t[c] = (l * sn[c] - t[c]) * b[c];
        md = Vec<T>::up(md, t);
        s1[k * kstep] = Vec<T>::make(t);
      }
      if (in && a.want_u) {
        if (!FIRST) Vec<T>::split(s2[half + k * kstep], u);
#pragma unroll
        for (int c = 0; c < W; ++c) u[c] = (l * sg[c] - u[c]) / h[c];
        mw = Vec<T>::up(mw, u);
        s1[half + k * kstep] = Vec<T>::make(u);
      }
      if (KT > 0) {
        dot[KT > 0 ? k : 0] += acc;
      } else {
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
        if (lane == 0) sdot[warp * K + k] += acc;
      }
    }
  }
  if (KT > 0) {
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      double acc = dot[k];
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
      if (lane == 0) sdot[warp * K + k] = acc;
    }
  }
  put_mag<T>(mag[2], md, warp, lane);
  put_mag<T>(mag[3], mw, warp, lane);
  __syncthreads();
  const int chunk = r0 / (nv * W);
  for (int k = tid; k < K; k += nt) {
    double s = 0;
    for (int w = 0; w < nw; ++w) s += sdot[w * K + k];
    a.dotp[((size_t)p * K + k) * a.nchunk + chunk] += s;
  }
  for (int q = q0; q < (a.want_u ? 2 : 1); ++q) {
    T* t1 = a.t1 + (q * a.PKN + pN * K);
    fir_lines<T, 0>(S1 + q * half, g, ax, a.nl, get_mag(mag[2 + q], nw, lane), q ? warp_w : warp, nw, lane, NoExt<T>(),
                    [&](int l, int c0, const V(&acc)[8], const T(&)[1][8][W]) {
                      const int k = a.nv(l), r = r0 + (l - k * nv) * W;
                      store_rows<FULL>(t1 + k * N, r, rows, c0, C, acc);
                    });
  }
}

template <typename T, int KT, bool FIRST>
__global__ void __launch_bounds__(kMaxThreads, 3) k_rows_bwd(Axis<T> ax, BwdRows<T> a) {
  const int nt = blockDim.x;
  start_next();
  if ((int)blockIdx.x >= a.nblocks) {
    wait_previous();
    const size_t KN = (size_t)(KT > 0 ? KT : a.K) * a.rows * ax.C, step = (size_t)(gridDim.x - a.nblocks) * nt;
    for (size_t i = (size_t)(blockIdx.x - a.nblocks) * nt + threadIdx.x; i < KN; i += step) {
      double s = 0;
#pragma unroll 8
      for (int p = 0; p < a.P; ++p) s += (double)a.q[(size_t)p * KN + i];
      a.gdic[i] += s;
    }
    return;
  }
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int mag[4][kMaxWarps];
  __shared__ T slam[kMaxK];
  const int p = blockIdx.x / a.nchunk, r0 = (blockIdx.x - p * a.nchunk) * a.nv.n * Vec<T>::W;
  auto* tab = reinterpret_cast<typename Vec<T>::V*>(smem);
  if ((ax.C & 7) == 0 && r0 + a.nv.n * Vec<T>::W <= a.rows) rows_bwd<T, KT, FIRST, true>(ax, a, p, r0, tab, mag, slam);
  else rows_bwd<T, KT, FIRST, false>(ax, a, p, r0, tab, mag, slam);
}

// ---- columns -----------------------------------------------------------------------------
// An image viewed as [outer][C][inner], contracted along C: a block takes n
// neighbouring elements (n W inner positions) of one (image, outer).  kOp: the
// pass alone; kDiv: conv_b (stored) -> a = p / conv_b -> the pass again; kMid:
// the reverse pass's c -> c / conv_b (stored in q), -p c / conv_b^2 -> the pass
// again, or for the weight recursion's images c (-p / conv_b^2) (:612-617,
// :655-660); kMidLast: c / conv_b alone.
enum { kOp, kDiv, kMid, kMidLast };

template <typename T, typename TO>
struct Cols {
  const T* in;
  TO* out;
  const T *atoms, *cbr;  // [K][N]; conv_b read by kMid
  T *cb, *q;             // conv_b written by kDiv (or null); c / conv_b
  int* range;
  int inner, chunks, K, PK, im0;  // images im0, im0 + 1, ...
  Div n;
  size_t N;
};

// W neighbouring values of a row of the tile.  FULL: both inside, 8-byte
// accesses; else up is the distance to the second one (0 where there is none).
template <bool FULL, typename T>
__device__ __forceinline__ void get_cols(const T* __restrict__ p, int up, T (&v)[Vec<T>::W]) {
  if (Vec<T>::W == 2 && FULL) {
    const float2 f = *reinterpret_cast<const float2*>(p);
    v[0] = (T)f.x;
    v[Vec<T>::W - 1] = (T)f.y;
  } else {
#pragma unroll
    for (int c = 0; c < Vec<T>::W; ++c) v[c] = p[c * up];
  }
}
template <bool FULL, typename T, typename TO>
__device__ __forceinline__ void put_cols(TO* __restrict__ p, int up, const T (&v)[Vec<T>::W]) {
  if (Vec<T>::W == 2 && sizeof(TO) == 4 && FULL) {
    *reinterpret_cast<float2*>(p) = make_float2((float)v[0], (float)v[Vec<T>::W - 1]);
  } else {
    p[0] = (TO)v[0];
    if (Vec<T>::W == 2 && (FULL || up)) p[1] = (TO)v[Vec<T>::W - 1];
  }
}

template <typename T, typename TO, int MODE, bool FULL>
__device__ __forceinline__ void cols(const Axis<T>& ax, const Cols<T, TO>& a, int i0, uint32_t off,
                                     typename Vec<T>::V* tab, int (*mag)[kMaxWarps]) {
  using V = typename Vec<T>::V;
  constexpr int W = Vec<T>::W;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nt = blockDim.x, nw = nt >> 5;
  const int C = ax.C, nl = a.n.n;
  const uint32_t inner = a.inner;
  V* S1 = tab + table_elems(ax) + kPad;
  V* S2 = S1 + lines_elems(ax, nl);
  const int im = a.im0 + blockIdx.y;
  // columns past the last repeat it, as rows
  const auto at_col = [&](int l) { return FULL ? l * W : min(i0 + l * W, a.inner - 1) - i0; };
  const auto has_up = [&](int l) { return FULL || i0 + l * W + 1 < a.inner ? 1 : 0; };
  const auto valid = [&](int l) { return FULL || i0 + l * W < a.inner; };
  const V* g = load_table(ax, tab, tid, nt);
  zero_pads(ax, S1, nl, tid, nt);
  if (MODE == kDiv || MODE == kMid) zero_pads(ax, S2, nl, tid, nt);
  wait_previous();
  typename Vec<T>::M m = 0;
  const T* src = a.in + (size_t)im * a.N + off;
#pragma unroll 2
  for (int e = tid; e < nl * (ax.C8 / 2); e += nt) {
    const int yh = a.n(e), l = e - yh * nl, y = 2 * yh;
    const T* s = src + (uint32_t)(y * inner + at_col(l));
    V v[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      T t[W];
#pragma unroll
      for (int c = 0; c < W; ++c) t[c] = T(0);
      if (FULL || y + r < C) get_cols<FULL>(s + r * inner, has_up(l), t);
      m = Vec<T>::up(m, t);
      v[r] = Vec<T>::make(t);
    }
    st2(S1 + l * ax.pitch + y, v[0], v[1]);
  }
  put_mag<T>(mag[0], m, warp, lane);
  __syncthreads();
  const int xmag = get_mag(mag[0], nw, lane);
  TO* dst = a.out + (size_t)im * a.N + off;
  const auto store = [&](int l, int c0, const V(&acc)[8], const T(&)[1][8][W]) {
    if (!valid(l)) return;
    uint32_t i = c0 * inner + l * W;
#pragma unroll
    for (int j = 0; j < 8; ++j, i += inner) {
      T t[W];
      Vec<T>::split(acc[j], t);
      if (FULL || c0 + j < C) put_cols<FULL, T, TO>(dst + i, has_up(l), t);
    }
  };
  if constexpr (MODE == kOp) {
    fir_lines<T, 0>(S1, g, ax, a.n, xmag, warp, nw, lane, NoExt<T>(), store);
  } else {
    const int pk = im >= a.PK ? im - a.PK : im;
    const bool weights = MODE != kDiv && im >= a.PK;
    const T* at = a.atoms + (size_t)(pk % a.K) * a.N + off;
    const T* cbr = MODE == kDiv ? nullptr : a.cbr + (size_t)pk * a.N + off;
    T* cbw = (MODE == kDiv && a.cb) ? a.cb + (size_t)pk * a.N + off : nullptr;
    T* qw = (MODE != kDiv && !weights) ? a.q + (size_t)pk * a.N + off : nullptr;
    constexpr int kAt = 0, kCb = MODE == kMid ? 1 : 0, kExt = MODE == kMid ? 2 : 1;
    m = 0;
    fir_lines<T, kExt>(
        S1, g, ax, a.n, xmag, warp, nw, lane,
        [&](int l, int c0, T(&ext)[kExt][8][W]) {
          uint32_t i = c0 * inner + at_col(l);
#pragma unroll
          for (int j = 0; j < 8; ++j, i += inner) {
            if (FULL || c0 + j < C) {
              if (MODE != kMidLast) get_cols<FULL>(at + i, has_up(l), ext[kAt][j]);
              if (MODE != kDiv) get_cols<FULL>(cbr + i, has_up(l), ext[kCb][j]);
            } else {
#pragma unroll
              for (int c = 0; c < W; ++c) ext[kAt][j][c] = ext[kCb][j][c] = T(1);
            }
          }
        },
        [&](int l, int c0, const V(&acc)[8], const T(&ext)[kExt][8][W]) {
          V nx[8];
          uint32_t i = c0 * inner + l * W;
#pragma unroll
          for (int j = 0; j < 8; ++j, i += inner) {
            T c[W], w[W];
            Vec<T>::split(acc[j], c);
#pragma unroll
            for (int h = 0; h < W; ++h) w[h] = T(0);
            if (FULL || c0 + j < C) {
              if (MODE == kDiv) {
                if (cbw && valid(l)) put_cols<FULL, T, T>(cbw + i, has_up(l), c);
#pragma unroll
                for (int h = 0; h < W; ++h) w[h] = ext[kAt][j][h] / c[h];
              } else if (weights) {
#pragma unroll
                for (int h = 0; h < W; ++h) w[h] = c[h] * (-ext[kAt][j][h] / (ext[kCb][j][h] * ext[kCb][j][h]));
              } else {
                T qv[W];
#pragma unroll
                for (int h = 0; h < W; ++h) {
                  qv[h] = c[h] / ext[kCb][j][h];
                  if (MODE == kMid) w[h] = -ext[kAt][j][h] * c[h] / (ext[kCb][j][h] * ext[kCb][j][h]);
                }
                if (valid(l)) put_cols<FULL, T, T>(qw + i, has_up(l), qv);
              }
              m = Vec<T>::up(m, w);
            }
            nx[j] = Vec<T>::make(w);
          }
          if (MODE != kMidLast) st8(S2 + l * ax.pitch + c0, nx);
        });
    if (MODE == kMidLast) return;
    if (MODE == kDiv && a.range && !Vec<T>::finite(m)) a.range[im / a.K] = 1;
    put_mag<T>(mag[1], m, warp, lane);
    __syncthreads();
    fir_lines<T, 0>(S2, g, ax, a.n, get_mag(mag[1], nw, lane), warp, nw, lane, NoExt<T>(), store);
  }
}

template <typename T, typename TO, int MODE>
__global__ void __launch_bounds__(kMaxThreads, 3) k_cols(Axis<T> ax, Cols<T, TO> a) {
  start_next();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int mag[2][kMaxWarps];
  const int o = blockIdx.x / a.chunks, i0 = (blockIdx.x - o * a.chunks) * a.n.n * Vec<T>::W;
  const uint32_t off = (uint32_t)o * ax.C * a.inner + i0;  // within an image
  auto* tab = reinterpret_cast<typename Vec<T>::V*>(smem);
  const bool full = (ax.C & 7) == 0 && i0 + a.n.n * Vec<T>::W <= a.inner && (Vec<T>::W == 1 || (a.inner & 1) == 0);
  if (full) cols<T, TO, MODE, true>(ax, a, i0, off, tab, mag);
  else cols<T, TO, MODE, false>(ax, a, i0, off, tab, mag);
}

// Loss and its gradient (cpp/loss.h:19-90) over segments of kLossSeg pixels: n the loss
// gradient, gw = n bary, part the segment's share of the loss.
template <typename T>
__global__ void k_loss_seg(const T* __restrict__ bary, const double* __restrict__ obs,
                           const T* __restrict__ wgrad, T* __restrict__ n, T* __restrict__ gw,
                           double* __restrict__ part, int loss_type, size_t N) {
  __shared__ double sh[32];
  const size_t p = blockIdx.y, j0 = (size_t)blockIdx.x * kLossSeg, j1 = min(N, j0 + kLossSeg);
  double acc = 0;
  for (size_t j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
    const size_t i = p * N + j;
    const T v1 = bary[i];
    const double o = obs[i];
    const T v2 = (T)o;
    T g;
    if (loss_type == WDL_LOSS_TV) {
      const T d = v1 - v2;
      acc += 0.5 * fabs((double)v1 - o);
      g = d > T(0) ? T(0.5) : T(-0.5);
    } else if (loss_type == WDL_LOSS_QUADRATIC) {
      const double d = (double)v1 - o;
      acc += d * d;
      g = T(2) * (v1 - v2);
    } else if (loss_type == WDL_LOSS_KL) {
      const double r = (double)v1 / o;
      acc += (double)v1 * log(r > kEpsilon ? r : kEpsilon) - (double)v1 + o;
      g = safe_log<T>(v1 / v2);
    } else {  // Wasserstein: gradient precomputed by the nested Sinkhorn
      g = wgrad[i];
    }
    n[i] = g;
    gw[i] = g * v1;
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) part[p * gridDim.x + blockIdx.x] = acc;
}

// Block i < PK: dot[i] = sum of its partial dot products; the other blocks: one
// histogram's loss from its segments.
__global__ void k_band_sums(const double* __restrict__ dotp, double* __restrict__ dot, int PK, size_t nparts,
                            const double* __restrict__ lossp, double* __restrict__ loss, int nseg) {
  __shared__ double sh[32];
  const bool is_dot = (int)blockIdx.x < PK;
  const double* src = is_dot ? dotp + (size_t)blockIdx.x * nparts : lossp + (size_t)(blockIdx.x - PK) * nseg;
  const size_t n = is_dot ? nparts : (size_t)nseg;
  double s = 0;
  for (size_t i = threadIdx.x; i < n; i += blockDim.x) s += src[i];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) {
    if (is_dot) dot[blockIdx.x] = s;
    else loss[blockIdx.x - PK] = s;
  }
}

// The limit is raised to the most any call takes: it belongs to the kernel, not to
// the launch, and a smaller value set by another thread in between would refuse
// this one's.  48 KB without it hold the kernel's static arrays too.
constexpr size_t kSmemStatic = 1024;  // at least every kernel's: magnitudes, kMaxK weights
template <typename F>
int want_smem(wdl_ctx* ctx, F f, size_t bytes) {
  if (bytes + kSmemStatic > 48 * 1024)
    WDL_CUDA_TRY(ctx, cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost));
  return WDL_OK;
}

// A launch of the chain (see start_next).  Overlapped starts pay where they hide a
// tail (several waves of blocks: images272 8.55 -> 8.30 ms) or a host that issues
// the launches one by one (the operator: 26.6 -> 20.5 us on volumes); in a
// replayed graph of small launches they cost 2 us each (dict64 0.87 -> 1.08 ms).
template <typename... Args, typename... Vals>
int launch_chained(wdl_ctx* ctx, void (*kernel)(Args...), dim3 grid, int threads, size_t smem, cudaStream_t s,
                   const Vals&... vals) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  const bool waves = (size_t)grid.x * grid.y >= 4 * (size_t)ctx->sm_count;
  if (!waves) cudaStreamIsCapturing(s, &cap);
  int rc;
  if ((rc = want_smem(ctx, kernel, smem))) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = waves || cap == cudaStreamCaptureStatusNone ? 1 : 0;
  WDL_CUDA_TRY(ctx, cudaLaunchKernelEx(&cfg, kernel, (Args)vals...));
  WDL_LAUNCH_CHECK(ctx);
  return WDL_OK;
}

template <typename T, typename TO, int MODE>
int launch_cols(wdl_ctx* ctx, int axis, int outer, int inner, Cols<T, TO> a, size_t nimg, cudaStream_t s) {
  const Axis<T> ax = make_axis<T>(ctx, axis);
  const int nl = cols_per_block(ax.G), w = nl * Vec<T>::W, threads = threads_for(nl * ax.G);
  a.n = Div::by(nl);
  a.inner = inner;
  a.chunks = (inner + w - 1) / w;
  a.N = ctx->N;
  const size_t smem = band_smem(ax, MODE == kOp || MODE == kMidLast ? 1 : 2, nl);
  int rc;
  const int first = a.im0;
  for (size_t done = 0; done < nimg; done += 65535) {  // gridDim.y is limited to 65535
    const unsigned n = (unsigned)std::min<size_t>(nimg - done, 65535);
    a.im0 = first + (int)done;
    if ((rc = launch_chained(ctx, k_cols<T, TO, MODE>, dim3((unsigned)(a.chunks * outer), n), threads, smem, s, ax, a)))
      return rc;
  }
  return WDL_OK;
}

template <typename TI, typename T>
int launch_rows_op(wdl_ctx* ctx, const TI* in, T* out, size_t nimg, cudaStream_t s) {
  const Axis<T> ax = make_axis<T>(ctx, 0);
  const int rows = (int)(ctx->N / ax.C), nl = lines_per_block(1, ax.G, 1), nr = nl * Vec<T>::W;
  const size_t smem = band_smem(ax, 1, nl);
  int rc;
  for (size_t done = 0; done < nimg; done += 65535) {
    const unsigned n = (unsigned)std::min<size_t>(nimg - done, 65535);
    if ((rc = launch_chained(ctx, k_rows_op<TI, T>, dim3((unsigned)((rows + nr - 1) / nr), n), threads_for(nl * ax.G),
                             smem, s, ax, in ? in + done * ctx->N : nullptr, out + done * ctx->N, rows, Div::by(nl))))
      return rc;
  }
  return WDL_OK;
}

// The y pass of a volume (the columns of each z plane), out of place.
template <typename T, typename TO>
int plane_cols(wdl_ctx* ctx, const T* in, TO* out, size_t nimg, int im0, cudaStream_t s) {
  Cols<T, TO> a{};
  a.in = in;
  a.out = out;
  a.im0 = im0;
  return launch_cols<T, TO, kOp>(ctx, 1, ctx->D, ctx->W, a, nimg, s);
}

#define WDL_BY_K(K, CALL)    \
  switch (K) {               \
    case 1: CALL(1); break;  \
    case 2: CALL(2); break;  \
    case 3: CALL(3); break;  \
    case 4: CALL(4); break;  \
    case 5: CALL(5); break;  \
    case 6: CALL(6); break;  \
    case 7: CALL(7); break;  \
    case 8: CALL(8); break;  \
    default: CALL(0); break; \
  }

}  // namespace

// The shape of a rows launch.
template <typename T>
struct RowsShape {
  Axis<T> ax;
  int rows, n, nchunk;
  RowsShape(const wdl_ctx* ctx, int K) : ax(make_axis<T>(ctx, 0)) {
    rows = (int)(ctx->N / ax.C);
    n = lines_per_block(K, ax.G, 1);
    nchunk = (rows + n * Vec<T>::W - 1) / (n * Vec<T>::W);
  }
  // one thread per item or, where there are more, per element of the step between
  // the passes
  int threads(int items) const { return threads_for(std::max(items, n * ax.C)); }
  size_t fwd_smem(int K) const { return band_smem(ax, 2, K * n); }
  size_t bwd_smem(int K) const { return band_smem(ax, 2, 2 * K * n) + (size_t)kMaxWarps * K * sizeof(double); }
};

// Every line buffer of a call fits the SM's shared memory.
template <typename T>
bool band_fits(const wdl_ctx* ctx, int K) {
  if (K > kMaxK || ctx->N * (size_t)(K > 0 ? K : 1) >= ((size_t)1 << 31)) return false;
  for (int a = 0; a < ctx->ndim; ++a) {
    const Axis<T> ax = make_axis<T>(ctx, a);
    if (ax.C > 8192) return false;
    const size_t need = a > 0 ? band_smem(ax, K > 0 ? 2 : 1, cols_per_block(ax.G))
                        : K > 0 ? RowsShape<T>(ctx, K).bwd_smem(K)
                                : band_smem(ax, 1, lines_per_block(1, ax.G, 1));
    if (need > kSmemMost) return false;
  }
  return true;
}
// The fused rows and columns kernels of an evaluation against separate kernels around
// the operator, on sizes and the factor alone (a histogram's bits may not depend on
// the batch).  A rows block's chain of K logarithms and divisions a pixel, and its line
// buffers for K atoms, lose where there are many atoms or hardly a pixel; on
// short lines that the factor covers whole, the sums have no tap to leave out either.
// Banded rows / separate kernels / before the banded kernels, ms an evaluation, L = 6 or 8:
//   atoms x groups of eight: 8 of 64 x 64, K = 64, FP64 4.1 / 2.6 / 3.0; 8 of 32^3, K = 64
//     33.6 / 19.4 / 23.9; gamma 50, FP64: 64 of 64 x 64 K = 12 2.71 / 2.80 / 2.81, K = 16 3.85 /
//     3.57 / 3.58, FP32 K = 16 2.01 / 2.00 / 2.17, K = 20 2.64 / 2.54 / 2.62; 8 of 40^3
//     K = 8 4.40 / 4.98 / 5.10, K = 20 15.5 / 12.4 / 11.8
//   pixels: one histogram, K = 5, FP32 16 x 16 0.39 / 0.25 / 0.27, 32 x 32 0.30 / 0.31 / 0.41;
//     barycenters of 16^3, K = 8, L = 20 0.56 / 0.48 / 0.48; FP64 16 x 16 against before: 1.27 x the speed
//     with 3 atoms, 1.00 with 8, 0.89 with 16 (2.5 x for 64 histograms)
//   shared memory, one block on an SM: 24 of 128 x 128, K = 24, FP64 8.6 / 5.3 / 11.7, at gamma
//     50 12.0 / 7.9 / 11.7; few atoms on long lines want it: 2048 x 64, K = 2 0.46 / 0.68 / 6.3
template <typename T>
bool band_rows_pay(const wdl_ctx* ctx, int K) {
  const RowsShape<T> sh(ctx, K);
  const bool vol = ctx->ndim == 3;
  if (std::max({ctx->W, ctx->H, ctx->D}) > 64) return K <= 16 || sh.bwd_smem(K) <= 110 * 1024;
  if (ctx->N < (sizeof(T) == 4 ? (vol ? 4097 : 1024) : vol ? 513 : 257) &&
      (sizeof(T) == 4 || vol || K > (int)(ctx->N / 32)))
    return false;
  const int items = K * sh.ax.G;
  if (!covers_lines<T>(ctx)) return items <= (vol ? 80 : 192);
  // eight of 32^3, K = 24, gamma 50, FP32: 1.06 x the speed before; of 36^3, K = 14: 0.88 x
  const bool brief = sh.ax.G <= 4;
  if (vol) return items <= (!brief ? 64 : sizeof(T) == 4 ? 96 : 80);
  return items <= (sizeof(T) == 4 || brief ? 128 : 96);
}
template bool band_rows_pay<float>(const wdl_ctx*, int);
template bool band_rows_pay<double>(const wdl_ctx*, int);

// The banded operator inside an evaluation against the dense axis passes.  On a
// small grid a banded pass is a block or two per image, whose chain (table, lines,
// maximum, sums) outlasts a dense tile of 64 x 64.  An evaluation with the Wasserstein
// loss (101 applications for it), 8 histograms, K = 4, L = 4, banded / dense ms: FP32
// 32 x 32 1.04 / 0.79 at gamma 2, 1.23 / 0.80 at gamma 50; 24 x 64 1.25 / 0.98 and 1.44 /
// 1.00; 48 x 48 1.10 / 1.05 and 1.41 / 1.08; 56 x 56 1.06 / 1.29 and 1.52 / 1.33, where at
// gamma 50 the sums take a line's every tap; volumes of 24^3 1.81 / 1.25, of 32^3 1.83 / 1.41 and
// 2.13 / 1.45.  FP64, whose dense passes cost more: 16 x 16
// 0.90 / 0.70, 32 x 32 1.27 / 1.05, 40 x 40 1.41 / 1.42; volumes of 16^3 1.31 / 1.20,
// of 24^3 with 64 histograms 4.7 / 5.4.
template <typename T>
bool band_pays(const wdl_ctx* ctx) {
  if (ctx->ndim == 2) {
    if (std::max(ctx->W, ctx->H) > 64) return true;
    if (ctx->N <= (sizeof(T) == 4 ? 48 * 48 : 32 * 32)) return false;
    return sizeof(T) == 8 || !covers_lines<T>(ctx);
  }
  // volumes: where the sums take a line's every tap
  return std::max({ctx->W, ctx->H, ctx->D}) > (sizeof(T) == 4 ? 48 : 16) || !covers_lines<T>(ctx);
}
template bool band_pays<float>(const wdl_ctx*);
template bool band_pays<double>(const wdl_ctx*);

// FP32 band sums against the split-BF16 axis passes, on grids above 128 and volumes:
// by the taps of a group of eight outputs over data of a few bits' spread.  The
// rule knows the context only (a histogram's bits may not depend on the batch), so
// the line lies where no batch loses.  At 72 taps (gamma 25), band against axis ms an
// evaluation: 32 of 200 x 200, K = 4, L = 20 8.4 / 9.1, 48 of 200 x 128, L = 10 3.70 /
// 3.79, 32 of 272 x 272, L = 20 14.4 / 16.5, 12 of 72^3, L = 6 11.1 / 11.8, one of 272 x 272
// 1.4 / 2.5; beyond it: 200 x 128 at 80 taps 3.92 / 3.78, 200 x 200 at 88 9.3 / 9.1 and at
// 136 11.8 / 10.4, 6 of 128^3 at 128 42.5 / 32.9 (one histogram would still win).
// Lines of up to 48 values are cheap at any width: 32 of 48^3 7.5 / 8.7, 64 of 24^3
// 1.9 / 3.6; 12 of 72^3 with all taps 14.0 / 11.8.
bool band_narrow(const wdl_ctx* ctx) {
  for (int a = 0; a < ctx->ndim; ++a) {
    const Axis<float> ax = make_axis<float>(ctx, a);
    if (ax.C8 > 48 && std::sqrt((double)ax.k1 * (ax.base + 2)) > 32.0) return false;
  }
  return true;
}

template bool band_fits<float>(const wdl_ctx*, int);
template bool band_fits<double>(const wdl_ctx*, int);

// The operator: TI -> T -> TO (the conversions of the FP64 entry points ride on
// the first and last pass).  tmp (and tmp2 for volumes): nimg * N values; out
// may be in, or for volumes tmp.
template <typename TI, typename T, typename TO>
int band_conv(wdl_ctx* ctx, const TI* in, TO* out, T* tmp, T* tmp2, size_t nimg, cudaStream_t s) {
  int rc;
  if ((rc = launch_rows_op<TI, T>(ctx, in, tmp, nimg, s))) return rc;
  if (ctx->ndim == 2) {
    Cols<T, TO> a{};
    a.in = tmp;
    a.out = out;
    return launch_cols<T, TO, kOp>(ctx, 1, 1, ctx->W, a, nimg, s);
  }
  if ((rc = plane_cols<T, T>(ctx, tmp, tmp2, nimg, 0, s))) return rc;
  Cols<T, TO> a{};
  a.in = tmp2;
  a.out = out;
  return launch_cols<T, TO, kOp>(ctx, 2, 1, ctx->W * ctx->H, a, nimg, s);
}
template int band_conv<double, float, double>(wdl_ctx*, const double*, double*, float*, float*, size_t, cudaStream_t);
template int band_conv<double, double, double>(wdl_ctx*, const double*, double*, double*, double*, size_t,
                                               cudaStream_t);
template int band_conv<float, float, float>(wdl_ctx*, const float*, float*, float*, float*, size_t, cudaStream_t);

// Forward iterations (b0 null: ones).  Slots of the iterate store are PKN (conv_b,
// phi) and PN (bary) apart; a barycenter-only run passes no conv_b, no phi and
// one bary.
template <typename T>
int band_forward(wdl_ctx* ctx, const BandEval<T>& e, const T* b0, cudaStream_t s) {
  const RowsShape<T> sh(ctx, e.K);
  const size_t N = ctx->N, PK = (size_t)e.P * e.K, PKN = PK * N, PN = (size_t)e.P * N;
  const unsigned blocks = (unsigned)((size_t)e.P * sh.nchunk), threads = sh.threads(e.K * sh.n * sh.ax.G);
  const size_t smem = sh.fwd_smem(e.K);
  const bool vol = ctx->ndim == 3;
  int rc;
  PassTimer timer(ctx, s);
  if ((rc = launch_rows_op<T, T>(ctx, b0, e.t1, PK, s))) return rc;
  for (int it = 0; it < e.L; ++it) {
    Cols<T, T> c{};
    c.atoms = e.atoms;
    c.cb = e.cb ? e.cb + it * PKN : nullptr;
    c.range = e.range;
    c.K = e.K;
    c.PK = (int)PK;
    if (vol) {
      if ((rc = plane_cols<T, T>(ctx, e.t1, e.t2, PK, 0, s))) return rc;
      c.in = e.t2;
      c.out = e.t1;
      if ((rc = launch_cols<T, T, kDiv>(ctx, 2, 1, ctx->W * ctx->H, c, PK, s))) return rc;
      if ((rc = plane_cols<T, T>(ctx, e.t1, e.t2, PK, 0, s))) return rc;
    } else {
      c.in = e.t1;
      c.out = e.t2;
      if ((rc = launch_cols<T, T, kDiv>(ctx, 1, 1, ctx->W, c, PK, s))) return rc;
    }
    FwdRows<T> a{};
    a.t2 = e.t2;
    a.lam = e.lam64;
    a.phi = e.phi ? e.phi + it * PKN : nullptr;
    a.bary = e.phi ? e.bary + it * PN : it == e.L - 1 ? e.bary : nullptr;
    a.t1 = it == e.L - 1 ? nullptr : e.t1;
    a.range = e.range;
    a.K = e.K;
    a.rows = sh.rows;
    a.nchunk = sh.nchunk;
    a.nv = Div::by(sh.n);
    a.nl = Div::by(e.K * sh.n);
    a.C = Div::by(sh.ax.C);
#define WDL_ROWS_FWD(KT) rc = launch_chained(ctx, k_rows_fwd<T, KT>, dim3(blocks), (int)threads, smem, s, sh.ax, a)
    WDL_BY_K(e.K, WDL_ROWS_FWD)
#undef WDL_ROWS_FWD
    if (rc) return rc;
  }
  timer.done(2.0 * e.L * PK);
  return WDL_OK;
}
template int band_forward<float>(wdl_ctx*, const BandEval<float>&, const float*, cudaStream_t);
template int band_forward<double>(wdl_ctx*, const BandEval<double>&, const double*, cudaStream_t);

// Loss partials (loss_parts per histogram) and the reverse pass's start n, gw from
// the barycenters.
template <typename T>
int loss_segments(wdl_ctx* ctx, int P, const T* bary, const double* obs, const T* wgrad, T* n, T* gw, double* part,
                  int loss_type, cudaStream_t s) {
  const size_t N = ctx->N, seg = loss_parts(ctx);
  for (int done = 0; done < P; done += 65535) {
    const int np = std::min(P - done, 65535);
    const size_t o = (size_t)done * N;
    k_loss_seg<T><<<dim3((unsigned)seg, (unsigned)np), 256, 0, s>>>(bary + o, obs + o, wgrad ? wgrad + o : nullptr,
                                                                    n + o, gw + o, part + done * seg, loss_type, N);
    WDL_LAUNCH_CHECK(ctx);
  }
  return WDL_OK;
}
template int loss_segments<float>(wdl_ctx*, int, const float*, const double*, const float*, float*, float*, double*,
                                  int, cudaStream_t);
template int loss_segments<double>(wdl_ctx*, int, const double*, const double*, const double*, double*, double*,
                                   double*, int, cudaStream_t);

template <typename T>
size_t band_dot_parts(const wdl_ctx* ctx, int K) {
  return (size_t)RowsShape<T>(ctx, K).nchunk;
}
template size_t band_dot_parts<float>(const wdl_ctx*, int);
template size_t band_dot_parts<double>(const wdl_ctx*, int);

// Reverse pass: dot (raw weight gradient), gdic (raw atom gradient, summed over
// the histograms; cleared by the caller with dotp) when e.dict, and with a
// loss pointer the histograms' losses.
template <typename T>
int band_backward(wdl_ctx* ctx, const BandEval<T>& e, double* loss, cudaStream_t s) {
  const RowsShape<T> sh(ctx, e.K);
  const size_t N = ctx->N, PK = (size_t)e.P * e.K, KN = (size_t)e.K * N, PKN = PK * N, PN = (size_t)e.P * N;
  const unsigned blocks = (unsigned)((size_t)e.P * sh.nchunk);
  // the same threads with and without the dictionary recursion: the dot
  // products' order of summation depends on them
  const unsigned threads = sh.threads(2 * e.K * sh.n * sh.ax.G);
  const size_t smem = sh.bwd_smem(e.K);
  const bool vol = ctx->ndim == 3;
  const int im0 = e.dict ? 0 : (int)PK;
  int rc;
  PassTimer timer(ctx, s);
  BwdRows<T> a{};
  a.t2 = e.t2;
  a.n = e.n;
  a.gw = e.gw;
  a.lam = e.lam;
  a.t1 = e.t1;
  a.dotp = e.dotp;
  a.K = e.K;
  a.P = e.P;
  a.rows = sh.rows;
  a.nv = Div::by(sh.n);
  a.nl = Div::by(e.K * sh.n);
  a.C = Div::by(sh.ax.C);
  a.nchunk = sh.nchunk;
  a.nblocks = (int)blocks;
  a.dict = e.dict;
  a.PKN = PKN;
  a.q = e.q;
  a.gdic = e.gdic;
  // q of the last columns launch, added up by the next rows launch's extra blocks
  const unsigned sum_blocks = e.dict ? grid_for(KN, (int)threads, ctx->sm_count, 2) : 0;
  for (int step = e.L; step >= 1; --step) {
    a.phi = e.phi + (step - 1) * PKN;
    a.bary = e.bary + (step - 1) * PN;
    a.want_u = step > 1;
    const bool first = step == e.L;
    const unsigned grid = blocks + (first ? 0 : sum_blocks);
#define WDL_ROWS_BWD(KT)                                                                                        \
  rc = first ? launch_chained(ctx, k_rows_bwd<T, KT, true>, dim3(grid), (int)threads, smem, s, sh.ax, a)         \
             : launch_chained(ctx, k_rows_bwd<T, KT, false>, dim3(grid), (int)threads, smem, s, sh.ax, a)
    WDL_BY_K(e.K, WDL_ROWS_BWD)
#undef WDL_ROWS_BWD
    if (rc) return rc;
    if (step == 1 && !e.dict) break;
    const size_t nimg = step > 1 ? (e.dict ? 2 * PK : PK) : PK;
    Cols<T, T> c{};
    c.atoms = e.atoms;
    c.cbr = e.cb + (step - 1) * PKN;
    c.q = e.q;
    c.K = e.K;
    c.PK = (int)PK;
    c.im0 = im0;
    const int axis = vol ? 2 : 1, inner = vol ? ctx->W * ctx->H : ctx->W;
    if (vol && (rc = plane_cols<T, T>(ctx, e.t1, e.t2, nimg, im0, s))) return rc;
    c.in = vol ? e.t2 : e.t1;
    c.out = vol ? e.t1 : e.t2;
    if (step == 1) rc = launch_cols<T, T, kMidLast>(ctx, axis, 1, inner, c, nimg, s);
    else rc = launch_cols<T, T, kMid>(ctx, axis, 1, inner, c, nimg, s);
    if (rc) return rc;
    if (step == 1) break;
    if (vol && (rc = plane_cols<T, T>(ctx, e.t1, e.t2, nimg, im0, s))) return rc;
  }
  if (e.dict) {  // the last round's share
    a.nblocks = 0;
    if ((rc = launch_chained(ctx, k_rows_bwd<T, 0, true>, dim3(grid_for(KN, (int)threads, ctx->sm_count)), (int)threads,
                             (size_t)0, s, sh.ax, a)))
      return rc;
  }
  k_band_sums<<<(unsigned)(PK + (loss ? e.P : 0)), 256, 0, s>>>(e.dotp, e.dot, (int)PK, sh.nchunk, e.lossp,
                                                              loss, (int)loss_parts(ctx));
  WDL_LAUNCH_CHECK(ctx);
  timer.done(((e.dict ? 2.0 * e.L - 1 : 0.0) + 2.0 * (e.L - 1)) * PK);
  return WDL_OK;
}
template int band_backward<float>(wdl_ctx*, const BandEval<float>&, double*, cudaStream_t);
template int band_backward<double>(wdl_ctx*, const BandEval<double>&, double*, cudaStream_t);

}  // namespace wdl
