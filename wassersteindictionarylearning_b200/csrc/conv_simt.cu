// CUDA-core forms of the separable Gaussian operator (plain FP32 and FP64) and
// of the stabilised log-sum-exp operator.
//
// The reference applies the 2-D Gaussian as an x-pass into a transposed
// temporary followed by a y-pass (cpp/kernels.h:669-699) and the 3-D one as
// three such passes (:762-807).  Here every pass is the same primitive: an
// image viewed as [R][C] (C contiguous) is contracted along C with the dense
// C x C factor and written as [C][R], moving the contracted axis to the front.
// Applying it once per axis returns the image to its original layout.  Most calls
// take the banded passes of sinkhorn_band.cu instead: the dense ones serve small
// grids and lines too long for a block's shared memory.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "log_group.cuh"
#include "wdl_internal.cuh"

namespace wdl {
namespace {

// ---- dense axis pass: out[c][r] = sum_k in[r][k] * G[k][c] ----------------------
// Block tile 64 (r) x 64 (c), k-slab 16, 256 threads with a 4x4 register tile
// (thread (tr, tc) owns 4 rows and the columns 4 tc + j).  Shared memory holds
// the input slab transposed (k-major).  FP32: the thread's rows are 4 tr + i,
// read as one 16-byte vector per k (row stride TR + 4 keeps it aligned; a
// quarter-warp reads 128 contiguous bytes).  FP64: the rows are tr + 16 i,
// read as 4 scalars per k: the 16 tr of a warp read 16 consecutive doubles, one
// conflict-free wavefront, where 16-byte vectors of doubles 32 bytes apart
// would conflict two ways; row stride TR + 1 spreads the slab's stores over
// the banks.  The two tc of a warp read two broadcast 4-vectors of the factor.
constexpr int TR = 64, TC = 64, TK = 16;

template <typename T>
struct AxisRows {
  static constexpr bool kInterleaved = sizeof(T) == 8;
  static constexpr int kStride = kInterleaved ? TR + 1 : TR + 4;
  __device__ static int row(int tr, int i) { return kInterleaved ? tr + 16 * i : 4 * tr + i; }
};

template <typename T>
__global__ void __launch_bounds__(256) axis_pass_kernel(const T* __restrict__ in,
                                                        T* __restrict__ out,
                                                        const T* __restrict__ G, int R, int C,
                                                        size_t img_stride) {
  using Rw = AxisRows<T>;
  __shared__ __align__(16) T sA[TK][Rw::kStride];
  __shared__ __align__(16) T sB[TK][TC + 4];
  const int tid = threadIdx.x;
  const int tr = tid & 15, tc = tid >> 4;
  const int r0 = blockIdx.x * TR, c0 = blockIdx.y * TC;
  const T* src = in + (size_t)blockIdx.z * img_stride;
  T* dst = out + (size_t)blockIdx.z * img_stride;

  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = T(0);

  for (int k0 = 0; k0 < C; k0 += TK) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int e = tid + 256 * q;
      int rr = e >> 4, kk = e & 15;
      int r = r0 + rr, k = k0 + kk;
      sA[kk][rr] = (r < R && k < C) ? src[(size_t)r * C + k] : T(0);
      int kb = e >> 6, cc = e & 63;
      int kg = k0 + kb, c = c0 + cc;
      sB[kb][cc] = (kg < C && c < C) ? G[(size_t)kg * C + c] : T(0);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      T a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = sA[kk][Rw::row(tr, i)];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = sB[kk][tc * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    int c = c0 + tc * 4 + j;
    if (c >= C) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int r = r0 + Rw::row(tr, i);
      if (r < R) dst[(size_t)c * R + r] = acc[i][j];
    }
  }
}

template <typename T>
int axis_pass(wdl_ctx* ctx, const T* in, T* out, const T* G, int R, int C, size_t nimg,
              size_t img_stride, cudaStream_t s) {
  size_t done = 0;
  while (done < nimg) {  // gridDim.z is limited to 65535
    size_t chunk = nimg - done;
    if (chunk > 65535) chunk = 65535;
    dim3 grid((R + TR - 1) / TR, (C + TC - 1) / TC, (unsigned)chunk);
    axis_pass_kernel<T><<<grid, 256, 0, s>>>(in + done * img_stride, out + done * img_stride, G,
                                             R, C, img_stride);
    WDL_LAUNCH_CHECK(ctx);
    done += chunk;
  }
  return WDL_OK;
}

// ---- log-domain axis pass ---------------------------------------------------------
// out[c][r] = log sum_k s_k exp(-(c-k)^2/gamma + in[r][k]), the reference's
// stabilised log-sum-exp (cpp/kernels.h:1082-1091).  With signs, s_k = +-1 from
// in_sign and the sign of the sum goes to out_sign, log|sum| to out
// (cpp/kernels.h:1123-1136).  The reference takes the maximum of the exponents
// in one pass and the shifted sum in a second; here the two are one pass with
// the running maximum (a new maximum rescales the partial sum), which gives the
// same value to rounding.
//
// A block owns LR rows of one image, staged in SMEM with an odd row stride (the
// rows of a warp fall in different banks).  A thread makes four neighbouring
// outputs c0..c0+3 of one row (c0 a multiple of 4): taps go outwards from the
// centres, both sides per step, and one step at distance d needs only two new
// row values (in[c0 - d] and in[c0 + 3 + d]; the other six taps of the step are
// values the four outputs have read at earlier steps), one tap weight and one
// stop test for the four.  With X = max_k in[r][k], every tap at distance >= d
// has exponent <= -d^2/gamma + X, so the group stops at the first d where
// -d^2/gamma + X < max - kTail for each of its outputs: the taps left out add at
// most 2C e^-kTail relative to an output's largest term, below the rounding of
// its sum (kTail = 40 bits for FP32, 60 nats for FP64).  FP32 works in base 2
// (inputs scaled by log2 e once when staged; ex2 / lg2), FP64 in base e with
// exp / log.  The summation order (centre, then outwards, both sides) differs
// from the reference's k = 0..C-1; only rounding depends on it.
//
// An output's result depends only on its row and its group (fixed by c), never
// on the block shape: LR (rows per block) is chosen per shape by the autotuner
// below without changing a result.
constexpr int kLogRowsDefault = 32;

using namespace ::wdl::lse;

// Stage LR rows of one image in SMEM (row stride CP, odd, with kHalo taps of
// kNone on each side), their signs (halo signs positive), the row maxima X and
// the tap table lk[d] = -d^2/gamma (scaled).  Rows whose length and start
// allow it are read as 16-byte vectors.
template <typename T, bool SIGNED, int LR>
__device__ __forceinline__ void log_stage(const T* __restrict__ in, const uint8_t* __restrict__ in_sign,
                                          T* rows, uint8_t* sg, T* xmax, T* lk, size_t base, int r0, int nr,
                                          int C, int CP, int SP, T gamma_t) {
  using Op = LogOps<T>;
  constexpr int V = 16 / sizeof(T);  // elements per 16-byte vector
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool vec = (C % V) == 0 && (base % V) == 0 && ((uintptr_t)in & 15) == 0;
  // sign bytes four at a time (FP32 rows: SP and kHalo keep the SMEM rows 4-aligned)
  const bool vsg = SIGNED && V == 4 && vec && ((uintptr_t)in_sign & 3) == 0;
  // warp w owns rows w, w + 8, ..., so the row maxima come from shuffles
  for (int rr = warp; rr < LR; rr += 8) {
    T* rw = rows + rr * CP + kHalo;
    uint8_t* sw = sg + rr * SP + kHalo;
    for (int k = lane; k < kHalo; k += 32) {
      rw[-kHalo + k] = Op::kNone;
      rw[C + k] = Op::kNone;
      if (SIGNED) {
        sw[-kHalo + k] = 1;
        sw[C + k] = 1;
      }
    }
    T vm = Op::kFloor;
    const size_t ro = base + (size_t)(r0 + rr) * C;
    const T* ir = in + ro;
    const uint8_t* isr = SIGNED ? in_sign + ro : nullptr;
    if (vec && rr < nr) {
      for (int k = lane * V; k < C; k += 32 * V) {
        T t[V];
        if constexpr (V == 4) {
          const float4 f = *reinterpret_cast<const float4*>(ir + k);
          t[0] = f.x; t[1] = f.y; t[2] = f.z; t[3] = f.w;
        } else {
          const double2 f = *reinterpret_cast<const double2*>(ir + k);
          t[0] = f.x; t[1] = f.y;
        }
        if (SIGNED && vsg) *reinterpret_cast<uint32_t*>(sw + k) = *reinterpret_cast<const uint32_t*>(isr + k);
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const T v = t[i] * Op::kScale;
          rw[k + i] = v;
          if (SIGNED && !vsg) sw[k + i] = isr[k + i];
          vm = vmax(vm, v);
        }
      }
    } else {
      for (int k = lane; k < C; k += 32) {
        T v = Op::kFloor;
        uint8_t sv = 1;
        if (rr < nr) {
          v = ir[k] * Op::kScale;
          if (SIGNED) sv = isr[k];
        }
        rw[k] = v;
        if (SIGNED) sw[k] = sv;
        vm = vmax(vm, v);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const T w = __shfl_xor_sync(0xffffffffu, vm, o);
      vm = vmax(vm, w);
    }
    if (lane == 0) xmax[rr] = vm;
  }
  for (int d = threadIdx.x; d < C; d += blockDim.x) lk[d] = -T(d) * T(d) / gamma_t * Op::kScale;
}


// Thread t makes the groups (c0 = 4 (t / LR + i 256 / LR)) of row rr = t % LR:
// the 32 lanes of a warp read 32 rows' taps at one position (conflict-free
// with the odd stride when LR = 32) and store runs out[c][r0 + rr] of
// consecutive rows.
// SUB: also write sub_out = sub_from (period sub_k images) - out, image by
// image (img0: the launch's first image).
// SQ > 0: the images are SQ x SQ (R = C = SQ), known at compile time, so
// strides and loop bounds are constants.
template <typename T, bool SIGNED, int LR, bool SUB, int SQ>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? (SIGNED ? 4 : 5) : 2) log_axis_pass_kernel(
    const T* __restrict__ in, T* __restrict__ out, int R_, int C_, size_t img_stride, T gamma_t,
    const uint8_t* __restrict__ in_sign, uint8_t* __restrict__ out_sign,
    unsigned long long* __restrict__ exps, const T* __restrict__ sub_from, T* __restrict__ sub_out,
    int sub_k, size_t img0) {
  const int R = SQ > 0 ? SQ : R_, C = SQ > 0 ? SQ : C_;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int CP = log_cp(C), SP = log_sp(C);
  T* rows = reinterpret_cast<T*>(smem_raw);             // [LR][CP]
  T* lk = rows + LR * CP;                               // [C]: -d^2/gamma (scaled)
  T* xmax = lk + C;                                     // [LR]
  uint8_t* sg = reinterpret_cast<uint8_t*>(xmax + LR);  // [LR][SP] (SIGNED)
  const int r0 = blockIdx.x * LR;
  const size_t base = (size_t)blockIdx.y * img_stride;
  const int nr = min(LR, R - r0);
  const int lane = threadIdx.x & 31;
  log_stage<T, SIGNED, LR>(in, in_sign, rows, sg, xmax, lk, base, r0, nr, C, CP, SP, gamma_t);
  __syncthreads();
  const int G = (C + 3) >> 2;
  const bool full = (C & 3) == 0;
  T* outi = out + base;
  uint8_t* osi = SIGNED ? out_sign + base : nullptr;
  const T* sfi = SUB ? sub_from + ((img0 + blockIdx.y) % (size_t)sub_k) * img_stride : nullptr;
  T* soi = SUB ? sub_out + base : nullptr;
  unsigned n_ex = 0;  // exps evaluated by this thread (profiling only)
  // blockDim is a multiple of LR, so a thread keeps one row: rr = tid % LR,
  // groups tid / LR, tid / LR + 256 / LR, ...
  const int rr = threadIdx.x % LR;
  const T* row = rows + rr * CP + kHalo;
  const uint8_t* sgn = sg + rr * SP + kHalo;
  const T X = xmax[rr];
  for (int gi = threadIdx.x / LR; gi < G && rr < nr; gi += 256 / LR) {
    const int c0 = 4 * gi;
    T v[4];
    bool pos[4];
    const int o = c0 * R + r0 + rr;  // offset in the image (R * C < 2^31, checked at launch)
    if (full) {
      n_ex += 4u * log_group<T, SIGNED, true>(row, sgn, lk, X, c0, C, v, pos);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        outi[o + j * R] = v[j];
        if (SIGNED) osi[o + j * R] = pos[j] ? 1 : 0;
        if (SUB) soi[o + j * R] = sfi[o + j * R] - v[j];
      }
    } else {
      const int nv = min(4, C - c0);
      n_ex += (unsigned)nv * log_group<T, SIGNED, false>(row, sgn, lk, X, c0, C, v, pos);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j < nv) {
          outi[o + j * R] = v[j];
          if (SIGNED) osi[o + j * R] = pos[j] ? 1 : 0;
          if (SUB) soi[o + j * R] = sfi[o + j * R] - v[j];
        }
      }
    }
  }
  if (exps) {
    unsigned long long v = n_ex;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) atomicAdd(exps, v);
  }
}

// The pass with one output per thread (log_lane): eight rows and four positions
// per warp, the groups of a row spread over the warps and over gridDim.z blocks.
// For launches that leave the GPU mostly idle, where a pass takes as long as one
// thread's chain of taps: a group of four is 8 exponentials a tap on one warp of
// 32 rows, here 2 on one of 8 rows.  Two 61 x 84 histograms, K = 3, FP64: the unsigned
// pass 17 us (its best rows per block) -> 6.8 us, the signed pair 20 -> 7.9 us.
constexpr int kLaneRows = 8;
template <typename T, bool SIGNED, bool SUB>
__global__ void __launch_bounds__(256, 2) log_lane_pass_kernel(
    const T* __restrict__ in, T* __restrict__ out, int R, int C, size_t img_stride, T gamma_t,
    const uint8_t* __restrict__ in_sign, uint8_t* __restrict__ out_sign,
    unsigned long long* __restrict__ exps, const T* __restrict__ sub_from, T* __restrict__ sub_out,
    int sub_k, size_t img0) {
  constexpr int LR = kLaneRows;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int CP = log_cp(C), SP = log_sp(C);
  T* rows = reinterpret_cast<T*>(smem_raw);             // laid out as log_axis_pass_kernel's
  T* lk = rows + LR * CP;
  T* xmax = lk + C;
  uint8_t* sg = reinterpret_cast<uint8_t*>(xmax + LR);
  const int r0 = blockIdx.x * LR;
  const size_t base = (size_t)blockIdx.y * img_stride;
  const int nr = min(LR, R - r0);
  log_stage<T, SIGNED, LR>(in, in_sign, rows, sg, xmax, lk, base, r0, nr, C, CP, SP, gamma_t);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rr = lane & 7, q = lane >> 3;
  const T* row = rows + rr * CP + kHalo;
  const uint8_t* sgn = sg + rr * SP + kHalo;
  const T X = xmax[rr];
  const int G = (C + 3) >> 2;
  unsigned n_ex = 0;
  for (int gi = blockIdx.z * 8 + warp; gi < G; gi += 8 * gridDim.z) {  // uniform over the warp
    const int c0 = 4 * gi, c = c0 + q;
    T v;
    bool pos;
    const int n = log_lane<T, SIGNED>(row, sgn, lk, X, c0, c, C, rr < nr, &v, &pos);
    if (rr < nr && c < C) {
      const size_t o = base + (size_t)(c * R + r0 + rr);
      out[o] = v;
      if (SIGNED) out_sign[o] = pos ? 1 : 0;
      if (SUB) sub_out[o] = sub_from[((img0 + blockIdx.y) % (size_t)sub_k) * img_stride + (size_t)(c * R + r0 + rr)] - v;
      n_ex += (unsigned)n;
    }
  }
  if (exps) {
    unsigned long long v = n_ex;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) atomicAdd(exps, v);
  }
}

template <typename T>
size_t log_axis_smem(int LR, int C) {
  return ((size_t)LR * log_cp(C) + C + LR) * sizeof(T) + (size_t)LR * log_sp(C) + 16;
}

// The grid side compiled as a constant (the log-domain dictionary-learning
// configuration's 256 x 256); other shapes take the general kernel.
constexpr int kLogSquare = 256;

template <typename T, int LR>
int log_axis_launch(wdl_ctx* ctx, const T* in, T* out, int R, int C, size_t nimg, size_t img_stride,
                    const uint8_t* in_sign, uint8_t* out_sign, cudaStream_t s, const T* sub_from,
                    T* sub_out, int sub_k) {
  const size_t smem = log_axis_smem<T>(LR, C);
  if ((size_t)R * C >= (size_t)1 << 31)
    return set_error(ctx, WDL_ERR_UNSUPPORTED, "log-domain operator: image of 2^31 values or more");
  const T gamma_t = T(ctx->gamma);
  unsigned long long* exps = ctx->profiling ? ctx->d_taps : nullptr;
  size_t done = 0;
  while (done < nimg) {
    size_t chunk = nimg - done;
    if (chunk > 65535) chunk = 65535;
    dim3 grid((R + LR - 1) / LR, (unsigned)chunk);
    size_t off = done * img_stride;
    const bool sq = R == kLogSquare && C == kLogSquare;
    if (in_sign) {
      auto k = sq ? log_axis_pass_kernel<T, true, LR, false, kLogSquare> : log_axis_pass_kernel<T, true, LR, false, 0>;
      if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      k<<<grid, 256, smem, s>>>(in + off, out + off, R, C, img_stride, gamma_t, in_sign + off,
                                out_sign + off, exps, nullptr, nullptr, 1, done);
    } else if (sub_from) {
      auto k = sq ? log_axis_pass_kernel<T, false, LR, true, kLogSquare> : log_axis_pass_kernel<T, false, LR, true, 0>;
      if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      k<<<grid, 256, smem, s>>>(in + off, out + off, R, C, img_stride, gamma_t, nullptr, nullptr, exps,
                                sub_from, sub_out + off, sub_k, done);
    } else {
      auto k = sq ? log_axis_pass_kernel<T, false, LR, false, kLogSquare> : log_axis_pass_kernel<T, false, LR, false, 0>;
      if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      k<<<grid, 256, smem, s>>>(in + off, out + off, R, C, img_stride, gamma_t, nullptr, nullptr, exps,
                                nullptr, nullptr, 1, done);
    }
    WDL_LAUNCH_CHECK(ctx);
    done += chunk;
  }
  return WDL_OK;
}

// Blocks of the one-output-per-thread form before its rows are split over gridDim.z.
inline size_t lane_blocks(int R, size_t nimg) { return (size_t)((R + kLaneRows - 1) / kLaneRows) * nimg; }
// It is a candidate while those are at most four per SM: from there on the group of four
// has threads enough, and its taps, weights and stop tests serve four outputs.
inline bool lane_candidate(const wdl_ctx* ctx, int R, int C, size_t nimg, size_t smem) {
  return lane_blocks(R, nimg) <= 4 * (size_t)ctx->sm_count && (size_t)R * C < ((size_t)1 << 31) && smem <= 200 * 1024;
}

template <typename T>
int log_lane_launch(wdl_ctx* ctx, const T* in, T* out, int R, int C, size_t nimg, size_t img_stride,
                    const uint8_t* in_sign, uint8_t* out_sign, cudaStream_t s, const T* sub_from,
                    T* sub_out, int sub_k) {
  const size_t smem = log_axis_smem<T>(kLaneRows, C), blocks = lane_blocks(R, nimg);
  unsigned long long* exps = ctx->profiling ? ctx->d_taps : nullptr;
  // split a row's groups over blocks until each warp has one or the grid is four blocks per SM
  const int G = (C + 3) / 4;
  const size_t z = std::max<size_t>(1, std::min<size_t>((G + 7) / 8, 4 * (size_t)ctx->sm_count / blocks));
  const dim3 grid((unsigned)((R + kLaneRows - 1) / kLaneRows), (unsigned)nimg, (unsigned)z);
  auto k = in_sign    ? log_lane_pass_kernel<T, true, false>
           : sub_from ? log_lane_pass_kernel<T, false, true>
                      : log_lane_pass_kernel<T, false, false>;
  if (smem > 48 * 1024)
    WDL_CUDA_TRY(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  k<<<grid, 256, smem, s>>>(in, out, R, C, img_stride, T(ctx->gamma), in_sign, out_sign, exps, sub_from, sub_out,
                            sub_k, 0);
  WDL_LAUNCH_CHECK(ctx);
  return WDL_OK;
}

template <typename T>
int log_axis_dispatch(wdl_ctx* ctx, int LR, bool lanes, const T* in, T* out, int R, int C, size_t nimg,
                      size_t img_stride, const uint8_t* in_sign, uint8_t* out_sign, cudaStream_t s,
                      const T* sub_from, T* sub_out, int sub_k) {
  if (lanes)
    return log_lane_launch<T>(ctx, in, out, R, C, nimg, img_stride, in_sign, out_sign, s, sub_from, sub_out, sub_k);
  // choice: rows per block
  switch (LR) {
    case 8:
      return log_axis_launch<T, 8>(ctx, in, out, R, C, nimg, img_stride, in_sign, out_sign, s, sub_from,
                                   sub_out, sub_k);
    case 16:
      return log_axis_launch<T, 16>(ctx, in, out, R, C, nimg, img_stride, in_sign, out_sign, s, sub_from,
                                    sub_out, sub_k);
    default:
      return log_axis_launch<T, 32>(ctx, in, out, R, C, nimg, img_stride, in_sign, out_sign, s, sub_from,
                                    sub_out, sub_k);
  }
}

// Autotuner: the first call of a shape (rows, row length, image count, type,
// signed) outside a graph capture runs every candidate (rows per block, and the
// one-output-per-thread form where the grid is small) on the
// call's own data (once untimed, once timed with CUDA events on the call's
// stream) and keeps the fastest for later calls of that shape.  WDL_AUTOTUNE=0
// keeps the default.
template <typename T>
int log_axis_pass(wdl_ctx* ctx, const T* in, T* out, int R, int C, size_t nimg, size_t img_stride,
                  const uint8_t* in_sign, uint8_t* out_sign, cudaStream_t s, const T* sub_from = nullptr,
                  T* sub_out = nullptr, int sub_k = 1) {
  const long long key[6] = {1, R, C, (long long)nimg, (long long)sizeof(T), in_sign ? 1 : 0};
  for (const auto& e : ctx->tuned)
    if (!std::memcmp(e.key, key, sizeof(key)))
      return log_axis_dispatch<T>(ctx, e.choice, e.lanes, in, out, R, C, nimg, img_stride, in_sign, out_sign, s, sub_from, sub_out, sub_k);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(s, &cap);
  if (!autotune_enabled() || !ctx->autotune || cap != cudaStreamCaptureStatusNone || ctx->profiling)
    return log_axis_dispatch<T>(ctx, kLogRowsDefault, false, in, out, R, C, nimg, img_stride, in_sign, out_sign, s, sub_from, sub_out, sub_k);
  const struct { int rows; bool lanes; } cand[4] = {{8, false}, {16, false}, {32, false}, {kLaneRows, true}};
  int best = kLogRowsDefault;
  bool best_lanes = false;
  float best_ms = 1e30f;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  WDL_CUDA_TRY(ctx, cudaEventCreate(&e0));
  WDL_CUDA_TRY(ctx, cudaEventCreate(&e1));
  int rc = WDL_OK;
  for (const auto& c : cand) {
    if (log_axis_smem<T>(c.rows, C) > 200 * 1024) continue;
    if (c.lanes && !lane_candidate(ctx, R, C, nimg, log_axis_smem<T>(c.rows, C))) continue;
    // an untimed run first: the first launch of a variant also loads it
    if ((rc = log_axis_dispatch<T>(ctx, c.rows, c.lanes, in, out, R, C, nimg, img_stride, in_sign, out_sign, s, sub_from, sub_out, sub_k))) break;
    cudaEventRecord(e0, s);
    if ((rc = log_axis_dispatch<T>(ctx, c.rows, c.lanes, in, out, R, C, nimg, img_stride, in_sign, out_sign, s, sub_from, sub_out, sub_k))) break;
    cudaEventRecord(e1, s);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best_ms) {
      best_ms = ms;
      best = c.rows;
      best_lanes = c.lanes;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  wdl_ctx::TuneEntry t;
  std::memcpy(t.key, key, sizeof(key));
  t.choice = best;
  t.lanes = best_lanes;
  t.ms = best_ms;
  ctx->tuned.push_back(t);
  // the candidates computed identical outputs; the last one's stands
  return WDL_OK;
}

template <typename T>
const T* factor(const wdl_ctx* ctx, int axis);
template <>
const float* factor<float>(const wdl_ctx* ctx, int axis) { return ctx->G32[axis]; }
template <>
const double* factor<double>(const wdl_ctx* ctx, int axis) { return ctx->G64[axis]; }

struct ConvTimer {
  wdl_ctx* ctx;
  cudaStream_t s;
  size_t nimg;
  bool count_exps;
  ConvTimer(wdl_ctx* c, cudaStream_t st, size_t n, bool exps = false)
      : ctx(c), s(st), nimg(n), count_exps(exps && c->profiling) {
    if (!ctx->profiling) return;
    if (count_exps) {
      if (!ctx->d_taps && cudaMalloc(&ctx->d_taps, sizeof(unsigned long long)) != cudaSuccess) {
        ctx->d_taps = nullptr;
        count_exps = false;
      }
      if (count_exps) cudaMemsetAsync(ctx->d_taps, 0, sizeof(unsigned long long), s);
    }
    cudaEventRecord(ctx->ev_a, s);
  }
  void done() {
    if (!ctx->profiling) return;
    cudaEventRecord(ctx->ev_b, s);
    cudaEventSynchronize(ctx->ev_b);
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev_a, ctx->ev_b);
    ctx->conv_ms += ms;
    ctx->conv_launches += 1;
    ctx->conv_images += (double)nimg;
    if (count_exps) {
      unsigned long long h = 0;
      if (cudaMemcpy(&h, ctx->d_taps, sizeof(h), cudaMemcpyDeviceToHost) == cudaSuccess)
        ctx->log_exps += (double)h;
    }
  }
};

template <typename T>
int conv_stack_simt(wdl_ctx* ctx, const T* in, T* out, T* tmp, size_t nimg, cudaStream_t s) {
  // The operator between other kernels of an evaluation: the banded passes, but on
  // small grids the dense ones (band_pays).
  const int W = ctx->W, H = ctx->H, D = ctx->D;
  const size_t N = ctx->N;
  ConvTimer timer(ctx, s, nimg);
  int rc;
  if (band_fits<T>(ctx, 0) && band_pays<T>(ctx)) {
    rc = ctx->ndim == 2 ? band_conv<T, T, T>(ctx, in, out, tmp, nullptr, nimg, s)
                        : band_conv<T, T, T>(ctx, in, out, out, tmp, nimg, s);
    if (rc) return rc;
    timer.done();
    return WDL_OK;
  }
  if (ctx->ndim == 2) {
    if ((rc = axis_pass<T>(ctx, in, tmp, factor<T>(ctx, 0), H, W, nimg, N, s))) return rc;
    if ((rc = axis_pass<T>(ctx, tmp, out, factor<T>(ctx, 1), W, H, nimg, N, s))) return rc;
  } else {
    if ((rc = axis_pass<T>(ctx, in, out, factor<T>(ctx, 0), D * H, W, nimg, N, s))) return rc;
    if ((rc = axis_pass<T>(ctx, out, tmp, factor<T>(ctx, 1), W * D, H, nimg, N, s))) return rc;
    if ((rc = axis_pass<T>(ctx, tmp, out, factor<T>(ctx, 2), H * W, D, nimg, N, s))) return rc;
  }
  timer.done();
  return WDL_OK;
}

template <typename T>
int log_conv_stack_simt(wdl_ctx* ctx, const T* in, T* out, T* tmp, size_t nimg,
                        const uint8_t* in_sign, uint8_t* out_sign, uint8_t* tmp_sign,
                        cudaStream_t s, const T* sub_from, T* sub_out, size_t sub_period) {
  if (ctx->ndim != 2)
    return set_error(ctx, WDL_ERR_UNSUPPORTED, "log-domain operator is 2-D only (as the reference)");
  const int W = ctx->W, H = ctx->H;
  const size_t N = ctx->N;
  ConvTimer timer(ctx, s, nimg, true);
  int rc;
  if ((rc = log_axis_pass<T>(ctx, in, tmp, H, W, nimg, N, in_sign, in_sign ? tmp_sign : nullptr, s)))
    return rc;
  if (sub_from && (in_sign || sub_period == 0 || sub_period % N))
    return set_error(ctx, WDL_ERR_INVALID_ARG, "log_conv_stack: subtraction needs an unsigned operand and whole images");
  if ((rc = log_axis_pass<T>(ctx, tmp, out, W, H, nimg, N, in_sign ? tmp_sign : nullptr, out_sign, s,
                             sub_from, sub_out, sub_from ? (int)(sub_period / N) : 1)))
    return rc;
  timer.done();
  return WDL_OK;
}

}  // namespace

int conv_stack_f64(wdl_ctx* ctx, const double* in, double* out, double* tmp, size_t nimg,
                   cudaStream_t s) {
  return conv_stack_simt<double>(ctx, in, out, tmp, nimg, s);
}

int conv_stack_simt_f32(wdl_ctx* ctx, const float* in, float* out, float* tmp, size_t nimg,
                        cudaStream_t s) {
  return conv_stack_simt<float>(ctx, in, out, tmp, nimg, s);
}

int log_conv_stack_f32(wdl_ctx* ctx, const float* in, float* out, float* tmp, size_t nimg,
                       const uint8_t* in_sign, uint8_t* out_sign, uint8_t* tmp_sign,
                       cudaStream_t s, const float* sub_from, float* sub_out, size_t sub_period) {
  return log_conv_stack_simt<float>(ctx, in, out, tmp, nimg, in_sign, out_sign, tmp_sign, s, sub_from,
                                    sub_out, sub_period);
}

int log_conv_stack_f64(wdl_ctx* ctx, const double* in, double* out, double* tmp, size_t nimg,
                       const uint8_t* in_sign, uint8_t* out_sign, uint8_t* tmp_sign,
                       cudaStream_t s, const double* sub_from, double* sub_out, size_t sub_period) {
  return log_conv_stack_simt<double>(ctx, in, out, tmp, nimg, in_sign, out_sign, tmp_sign, s, sub_from,
                                     sub_out, sub_period);
}

}  // namespace wdl
