// finpar/OptionPricing.fut (entry main, f32) behind the C API the Futhark
// compiler generates for it (include/op.h): Sobol quasi-random paths through
// an inverse Gaussian, a Brownian bridge and a Black-Scholes model, priced
// under one of three contracts and averaged per model.
//
// op_paths_kernel<C> is specialised on the contract C, which fixes a path's
// shape (dates x underlyings: contract 1 is 1 x 1, contract 2 is 5 x 3,
// contract 3 is 367 x 3, the reference's size coercions at :294-298), so
// every loop over a path has a constant trip count and the paths of contracts
// 1 and 2 stay in registers.  A thread prices a contiguous range of paths:
// the first path's Sobol point is assembled from the set bits of its Gray
// code (:13-33); each following path n differs from n - 1 in one Gray-code
// bit, so its point is the previous one XOR one direction vector per
// dimension.  Contract 1's Gaussian is computed on the fly, contract 2's ahead of
// the Brownian bridge recursion, the correlated prices date by date with a running
// product (the scan of :217), and the payoff is decided as the dates go by,
// so a path holds only its Sobol integers and the bridge values.  Each
// thread accumulates its payoffs per model in f64, each CTA adds its threads'
// sums in a fixed tree order, and op_reduce_kernel adds the CTAs' sums, again
// in a fixed order, and divides by num_mc_it in f32.
//
// Arithmetic: this file is compiled with --fmad=false, so every f32
// operation is rounded on its own as in the reference (and the CPU oracle);
// division and square root are IEEE; f32.exp and f32.log are the f32
// rounding of CUDA's f64 exp and log.  The kernel is compute-bound (about
// 1e5 operations per path of contract 3, mostly the inverse Gaussian and the
// exponentials).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "op.h"
#include "exact_math.cuh"
#include "fut_api.cuh"

namespace {

template <int C>
struct OpShape;
// kMinCtas: the thread-per-path kernel's CTAs per SM the register budget is
// sized for (contract 2's 15-dimension paths want the registers of one)
template <>
struct OpShape<1> {
  static constexpr int D = 1, U = 1, kMinCtas = 4;
};
template <>
struct OpShape<2> {
  static constexpr int D = 5, U = 3, kMinCtas = 3;
};
template <>
struct OpShape<3> {  // priced by op_paths_warp_kernel
  static constexpr int D = 367, U = 3;
};

constexpr int kOpThreads = 128;  // thread-per-path CTAs: contract 2 fits three per SM
constexpr int kOpModels = 4;  // models priced per launch (accumulators in registers)

struct OpDev {
  int num_mc_it, num_bits, num_models, num_discts;
  const int32_t* dir_vs;
  const float *md_cs, *md_vols, *md_drifts, *md_sts, *md_detvals, *md_discts;
  const int32_t* bb_inds;
  const float* bb_data;
  float* pay_out;  // reference order: every path's payoff, [path][model]; null otherwise
};

__device__ __forceinline__ float f32exp(float x) { return (float)exp((double)x); }
__device__ __forceinline__ float f32log(float x) { return (float)log((double)x); }

// Wichura's AS241 coefficient tables (:59-118), as the reference's f32 literals
__constant__ float kSmallA[8] = {3.387132872796366608f, 133.14166789178437745f, 1971.5909503065514427f,
                                 13731.693765509461125f, 45921.953931549871457f, 67265.770927008700853f,
                                 33430.575583588128105f, 2509.0809287301226727f};
__constant__ float kSmallB[8] = {1.0f, 42.313330701600911252f, 687.1870074920579083f, 5394.1960214247511077f,
                                 21213.794301586595867f, 39307.89580009271061f, 28729.085735721942674f,
                                 5226.495278852854561f};
__constant__ float kInterA[8] = {1.42343711074968357734f, 4.6303378461565452959f, 5.7694972214606914055f,
                                 3.64784832476320460504f, 1.27045825245236838258f, 0.24178072517745061177f,
                                 0.0227238449892691845833f, 7.7454501427834140764e-4f};
__constant__ float kInterB[8] = {1.0f, 2.05319162663775882187f, 1.6763848301838038494f, 0.68976733498510000455f,
                                 0.14810397642748007459f, 0.0151986665636164571966f, 5.475938084995344946e-4f,
                                 1.05075007164441684324e-9f};
__constant__ float kTailA[8] = {6.6579046435011037772f, 5.4637849111641143699f, 1.7848265399172913358f,
                                0.29656057182850489123f, 0.026532189526576123093f, 0.0012426609473880784386f,
                                2.71155556874348757815e-5f, 2.01033439929228813265e-7f};
__constant__ float kTailB[8] = {1.0f, 0.59983220655588793769f, 0.13692988092273580531f, 0.0148753612908506148525f,
                                7.868691311456132591e-4f, 1.8463183175100546818e-5f, 1.4215117583164458887e-7f,
                                2.04426310338993978564e-5f};

// :52-57.  near_div's range holds at every argument the Gaussian has: both
// polynomials lie between 0.5 and 2^10 there (central branch: x in 0 .. 0.181;
// tails: x in -0.24 .. 3.4 and 0 ..), and a NaN or infinite argument (a Sobol
// integer of 0 or 2^B) gives NaN either way.
__device__ __forceinline__ float poly_appr(float x, const float* a, const float* b) {
  const float num = x * (x * (x * (x * (x * (x * (x * a[7] + a[6]) + a[5]) + a[4]) + a[3]) + a[2]) + a[1]) + a[0];
  const float den = x * (x * (x * (x * (x * (x * (x * b[7] + b[6]) + b[5]) + b[4]) + b[3]) + b[2]) + b[1]) + b[0];
  return near_div(num, den, near_rcp(den));
}

// :120-136, split at its branch: gauss_central for |p - 0.5| <= 0.425,
// gauss_tail otherwise
__device__ __forceinline__ bool gauss_is_central(float dp) {
  return fabsf(dp) <= 0.425f;
}
__device__ __forceinline__ float gauss_central(float dp) {
  return dp * poly_appr(0.180625f - dp * dp, kSmallA, kSmallB);
}
__device__ __forceinline__ float gauss_tail(float dp) {
  const float pp = dp < 0.0f ? dp + 0.5f : 0.5f - dp;
  const float r = near_sqrt(-f32log(pp));  // 1.6 .. 4.8, or infinite or NaN: then so is x
  const float x = r <= 5.0f ? poly_appr(r - 1.6f, kInterA, kInterB) : poly_appr(r - 5.0f, kTailA, kTailB);
  return dp < 0.0f ? 0.0f - x : x;
}
__device__ __forceinline__ float ugaussian_el(float p) {
  const float dp = p - 0.5f;
  return gauss_is_central(dp) ? gauss_central(dp) : gauss_tail(dp);
}

// :234-240
__device__ __forceinline__ float fmin_payoff(const float* xs) {
  const float a = xs[0] / 3758.05f, b = xs[1] / 11840.0f, c = xs[2] / 1200.0f;
  return a < b ? (a < c ? a : c) : (b < c ? b : c);
}

// bb_inds selects dates of the path: bi[0] always, and from i = 1 on
// bi[i], ri[i] in 1 .. D and li[i] in 0 .. D (0: no left point).  Kernels
// that find otherwise price nothing and return NaN instead of reading
// outside the path (the entry point rejects such inputs before launching).
template <int D>
__device__ bool bridge_indices_valid(const int32_t* ind) {
  bool ok = ind[0] >= 1 && ind[0] <= D;
  for (int i = 1; i < D; i++)
    ok = ok && ind[i] >= 1 && ind[i] <= D && ind[D + i] >= 0 && ind[D + i] <= D && ind[2 * D + i] >= 1 &&
         ind[2 * D + i] <= D;
  return ok;
}

// Bound by its instructions, the Gaussians' above all.  With 15 dimensions
// (contract 2) a path's Gaussians come first, the central branch in every lane and
// the tail arguments, 15 % of them, queued by the warp and evaluated 32 at a time: on
// the fly nearly every Gaussian has some lane in its tail, with an f64 logarithm.
// 1M paths 219 -> 130 us, 131072 45 -> 32, 16384 18.7 -> 14.5.  Contract 1 keeps the
// branch: its one Gaussian per path queued took 115 us for 8.4M paths against 108,
// and with eight paths per lane at a time 103, but 50 against 36 for 2M.
template <int C>
__global__ void __launch_bounds__(kOpThreads, OpShape<C>::kMinCtas) op_paths_kernel(OpDev a, int m0, double* __restrict__ partial) {
  constexpr int D = OpShape<C>::D, U = OpShape<C>::U, K = D * U;
  constexpr bool kQueue = K > 1;
  constexpr int kQueued = kQueue ? K * 32 : 1;
  // a warp's Gaussians, [dimension][lane], its queue of tail arguments and where
  // their Gaussians go
  __shared__ float s_z[kOpThreads / 32][kQueued], s_q[kOpThreads / 32][kQueued];
  __shared__ uint16_t s_to[kOpThreads / 32][kQueued];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* const z = s_z[warp];
  __shared__ int32_t s_ind[3 * D];  // bb_inds: bi, li, ri
  __shared__ float s_dat[3 * D];    // bb_data: sd, lw, rw
  __shared__ int s_ok;
  for (int i = threadIdx.x; i < 3 * D; i += blockDim.x) {
    s_ind[i] = a.bb_inds[i];
    s_dat[i] = a.bb_data[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) s_ok = bridge_indices_valid<D>(s_ind);
  __syncthreads();
  const bool ok = s_ok;
  const int64_t T = (int64_t)gridDim.x * blockDim.x;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t N = ok ? a.num_mc_it : 0;
  const int64_t lo = N * t / T, hi = N * (t + 1) / T;
  const int B = a.num_bits;
  const uint32_t bits = B >= 32 ? 0xffffffffu : ((1u << B) - 1u);
  const float scale = ldexpf(1.0f, -B);  // x / 2 ** num_bits is x * 2 ** -num_bits, both exact
  const int nm = min(kOpModels, a.num_models - m0);
  double acc[kOpModels];
#pragma unroll
  for (int mm = 0; mm < kOpModels; mm++) acc[mm] = 0.0;
  int32_t xs[K];  // the path's Sobol integers, dimension k = date * U + underlying
  float bb[K];    // the Brownian bridge, [date][underlying]
  for (int k = 0; k < K; k++) xs[k] = 0;
  // queued: the lanes of a warp stay together, one path longer for some of them
  const int64_t last = kQueue ? lo + __reduce_max_sync(0xffffffffu, (int)(hi - lo)) : hi;
  for (int64_t it = lo; it < last; it++) {
    const bool on = it < hi;
    const int32_t n = (int32_t)(it + 1);
    if (on && it == lo) {  // from the Gray code's set bits (:13-33)
      for (uint32_t g = (uint32_t)((n >> 1) ^ n) & bits; g != 0u; g &= g - 1u) {
        const int i = __ffs((int)g) - 1;
        for (int k = 0; k < K; k++) xs[k] ^= a.dir_vs[(int64_t)k * B + i];
      }
    } else if (on) {  // Gray code of n = that of n - 1 with bit ctz(n) flipped
      const int c = __ffs(n) - 1;
      if (c < B)
        for (int k = 0; k < K; k++) xs[k] ^= a.dir_vs[(int64_t)k * B + c];
    }
    if constexpr (kQueue) {
      int nq = 0;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const float dp = (float)xs[k] * scale - 0.5f;
        const bool tail = on && !gauss_is_central(dp);
        z[k * 32 + lane] = gauss_central(dp);
        const unsigned ball = __ballot_sync(0xffffffffu, tail);
        if (tail) {
          const int at = nq + __popc(ball & ((1u << lane) - 1u));
          s_q[warp][at] = dp;
          s_to[warp][at] = (uint16_t)(k * 32 + lane);
        }
        nq += __popc(ball);
      }
      __syncwarp();
      for (int e = lane; e < nq; e += 32) z[s_to[warp][e]] = gauss_tail(s_q[warp][e]);
      __syncwarp();
      if (!on) continue;  // only ever in the last round
    }
    auto gauss = [&](int k) { return kQueue ? z[k * 32 + lane] : ugaussian_el((float)xs[k] * scale); };
    // Brownian bridge per underlying (:142-175)
    for (int k = 0; k < K; k++) bb[k] = 0.0f;
    for (int u = 0; u < U; u++) {
      bb[(s_ind[0] - 1) * U + u] = s_dat[0] * gauss(u);
      for (int i = 1; i < D; i++) {
        const int j = s_ind[D + i] - 1, kk = s_ind[2 * D + i] - 1, l = s_ind[i] - 1;
        const float wk = bb[kk * U + u];
        const float zi = gauss(i * U + u);
        const float tmp = s_dat[2 * D + i] * wk + s_dat[i] * zi;
        bb[l * U + u] = j == -1 ? tmp : tmp + s_dat[D + i] * bb[j * U + u];
      }
      for (int ii = 1; ii < D; ii++) {
        const int i = D - ii;
        bb[i * U + u] = bb[i * U + u] - bb[(i - 1) * U + u];
      }
    }
    // per model: correlation (:188-199), prices (:201-228), payoff (:242-301)
#pragma unroll
    for (int mm = 0; mm < kOpModels; mm++) {
      if (mm >= nm) break;
      const int m = m0 + mm;
      const float* cm = a.md_cs + (int64_t)m * U * U;
      const float* vol = a.md_vols + (int64_t)m * K;
      const float* dr = a.md_drifts + (int64_t)m * K;
      const float* st = a.md_sts + (int64_t)m * U;
      const float* disc = a.md_discts + (int64_t)m * a.num_discts;
      float sc[U];
#pragma unroll
      for (int u = 0; u < U; u++) sc[u] = 1.0f;
      float pay = 0.0f, amount = 0.0f;
      int date = 0;
      bool decided = false, cond = false;
      for (int d = 0; d < D; d++) {
        float price[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          float noise = 0.0f;
#pragma unroll
          for (int i = 0; i <= u; i++) noise = noise + bb[d * U + i] * cm[u * U + i];
          const float cv = dr[d * U + u] + noise * vol[d * U + u];
          sc[u] = sc[u] * f32exp(cv);
          price[u] = st[u] * sc[u];
        }
        if constexpr (C == 1) {
          const float amt = (price[0] - 4000.0f) * a.md_detvals[m];
          pay = (0.0f < amt ? amt : 0.0f) * disc[0];
        } else if constexpr (C == 2) {
          if (!decided) {
            if (d < 4) {
              if (1.0f <= fmin_payoff(price)) {
                date = d;
                amount = d == 0 ? 1150.0f : d == 1 ? 1300.0f : d == 2 ? 1450.0f : 1600.0f;
                decided = true;
              }
            } else {
              const float x50 = fmin_payoff(price);
              date = 4;
              amount = 1.0f <= x50 ? 1750.0f : (0.75f < x50 ? 1000.0f : x50 * 1000.0f);
              decided = true;
            }
          }
          if (d == D - 1) pay = amount * disc[date];
        } else {
          cond = cond || (price[0] <= 2630.6349999999998f || price[1] <= 8288.0f || price[2] <= 840.0f);
          if (d == D - 1) {
            const float price1 = 100.0f * disc[0];
            const bool goto40 = cond && (price[0] < 3758.05f || price[1] < 11840.0f || price[2] < 1200.0f);
            const float amt = goto40 ? 1000.0f * fmin_payoff(price) : 1000.0f;
            pay = price1 + amt * disc[1];
          }
        }
      }
      acc[mm] += (double)pay;
      if (a.pay_out) a.pay_out[it * a.num_models + m0 + mm] = pay;
    }
  }
  // per-CTA sums in a fixed tree order: partial[mm][blockIdx.x]
  __shared__ double red[kOpThreads];
#pragma unroll
  for (int mm = 0; mm < kOpModels; mm++) {
    if (mm >= nm) break;
    red[threadIdx.x] = ok ? acc[mm] : __longlong_as_double(0x7ff8000000000000LL);
    __syncthreads();
    for (int w = kOpThreads / 2; w > 0; w >>= 1) {
      if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
      __syncthreads();
    }
    if (threadIdx.x == 0) partial[(int64_t)mm * gridDim.x + blockIdx.x] = red[0];
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Warp per path (contract 3: 367 dates x 3 underlyings)
// ---------------------------------------------------------------------------
// A warp prices a contiguous range of paths, its lanes sharing each path's
// dimensions k = lane, lane + 32, ...: the Sobol integers (kept from path to
// path), the Gaussians, the differences, the exponentials and the payoff's
// date test run across the lanes on [date][underlying] arrays in shared
// memory.  The bridge recursion (:150-165) runs level by level on the CTA's
// schedule (op_bridge_schedule): the steps of one level touch disjoint
// positions and read only values of earlier levels, so each step computes
// exactly what it computes in the sequential loop.  The running product of
// the prices (the scan of :217) stays sequential per underlying, in the
// reference's order.
constexpr int kWarpPathWarps = 7;

// Thread 0 of a CTA: level[i] of every bridge step i = 1 .. D-1 -- one more
// than the levels of the last writes of the positions it reads or writes and
// of the reads of the position it writes -- and the steps sorted by level:
// order[start[v] .. start[v + 1]) are the steps of level v, v = 1 .. nlev.
// lw, lr, level: [D] scratch; start: [D + 2].  False if an index leaves the
// path.
template <int D>
__device__ bool op_bridge_schedule(const int32_t* ind, int* lw, int* lr, int* level, int* order, int* start,
                                   int& nlev) {
  if (!bridge_indices_valid<D>(ind)) return false;
  for (int p = 0; p < D; p++) lw[p] = lr[p] = -1;
  lw[ind[0] - 1] = 0;  // step 0 writes bi[0]
  int maxl = 0;
  for (int i = 1; i < D; i++) {
    const int j = ind[D + i] - 1, k = ind[2 * D + i] - 1, l = ind[i] - 1;
    int lev = max(max(lw[k], lw[l]), lr[l]) + 1;
    if (j >= 0) lev = max(lev, lw[j] + 1);
    lev = max(lev, 1);
    level[i] = lev;
    lw[l] = lev;
    lr[k] = max(lr[k], lev);
    if (j >= 0) lr[j] = max(lr[j], lev);
    maxl = max(maxl, lev);
  }
  for (int v = 0; v <= maxl + 1; v++) start[v] = 0;
  for (int i = 1; i < D; i++) start[level[i] + 1]++;
  for (int v = 1; v <= maxl + 1; v++) start[v] += start[v - 1];
  for (int v = 0; v <= maxl; v++) lw[v] = start[v];  // insertion cursors
  for (int i = 1; i < D; i++) order[lw[level[i]]++] = i;
  nlev = maxl;
  return true;
}

template <int C>
struct OpWarpSmem {
  static constexpr int D = OpShape<C>::D, KP = (OpShape<C>::D * OpShape<C>::U + 31) / 32 * 32;
  static constexpr int kFixed = (8 * D + 2 + 3) & ~3;  // bb_inds, bb_data, order, start
  static constexpr int kWarp = 3 * KP;                 // Sobol integers, two path arrays
  static constexpr int kWords = kFixed + kWarpPathWarps * kWarp;
  static_assert(3 * D <= kWarp, "the schedule's scratch fits a warp's arrays");
};

// dirT[i][k] = dir_vs[k][i]: the direction numbers of bit i of every
// dimension, contiguous for the warp's lanes.
__global__ void op_transpose_dirs_kernel(const int32_t* __restrict__ dir_vs, int K, int B,
                                         int32_t* __restrict__ dirT) {
  const int64_t n = (int64_t)K * B;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = q / K, k = q - i * K;
    dirT[q] = dir_vs[k * B + i];
  }
}

// *taken != 0: op_paths_block_kernel has priced the paths.
template <int C>
__global__ void __launch_bounds__(kWarpPathWarps * 32, 2) op_paths_warp_kernel(OpDev a, const int32_t* __restrict__ dirT,
                                                                            int m0, double* __restrict__ partial,
                                                                            const int* __restrict__ taken) {
  if (*taken) return;
  using L = OpWarpSmem<C>;
  constexpr int D = OpShape<C>::D, U = OpShape<C>::U, K = D * U, KP = L::KP;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ float op_dyn[];
  int32_t* s_ind = reinterpret_cast<int32_t*>(op_dyn);  // bb_inds: bi, li, ri
  float* s_dat = op_dyn + 3 * D;                         // bb_data: sd, lw, rw
  int* s_order = reinterpret_cast<int*>(op_dyn + 6 * D);
  int* s_start = s_order + D;  // D + 2
  __shared__ int s_ok, s_nlev;
  __shared__ double red[kWarpPathWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* wbase = op_dyn + L::kFixed + warp * L::kWarp;
  int32_t* sX = reinterpret_cast<int32_t*>(wbase);  // Sobol integers [K]
  float* sG = wbase + KP;                           // Gaussians, then the bridge's differences
  float* sB = wbase + 2 * KP;                       // the bridge, then exponentials and prices
  for (int i = threadIdx.x; i < 3 * D; i += blockDim.x) {
    s_ind[i] = a.bb_inds[i];
    s_dat[i] = a.bb_data[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {  // scratch: warp 0's arrays, not in use yet
    int* scr = reinterpret_cast<int*>(op_dyn + L::kFixed);
    int nl = 0;
    s_ok = op_bridge_schedule<D>(s_ind, scr, scr + D, scr + 2 * D, s_order, s_start, nl);
    s_nlev = nl;
  }
  __syncthreads();
  const bool ok = s_ok;
  const int nlev = s_nlev;
  const int64_t W = (int64_t)gridDim.x * kWarpPathWarps;
  const int64_t w = (int64_t)blockIdx.x * kWarpPathWarps + warp;
  const int64_t N = ok ? a.num_mc_it : 0;
  const int64_t lo = N * w / W, hi = N * (w + 1) / W;
  const int B = a.num_bits;
  const uint32_t bits = B >= 32 ? 0xffffffffu : ((1u << B) - 1u);
  const float scale = ldexpf(1.0f, -B);
  const int nm = min(kOpModels, a.num_models - m0);
  double acc[kOpModels];
#pragma unroll
  for (int mm = 0; mm < kOpModels; mm++) acc[mm] = 0.0;
  for (int64_t it = lo; it < hi; it++) {
    const int32_t n = (int32_t)(it + 1);
    const uint32_t gray = (uint32_t)((n >> 1) ^ n) & bits;
    const int c = __ffs(n) - 1;  // the Gray-code bit path n flips
    if (it == lo) {  // Sobol point (:13-33) from the Gray code's set bits
      for (int k = lane; k < K; k += 32) sX[k] = 0;
      for (uint32_t g = gray; g != 0u; g &= g - 1u) {
        const int32_t* row = dirT + (int64_t)(__ffs((int)g) - 1) * K;
        for (int k = lane; k < K; k += 32) sX[k] ^= row[k];
      }
    } else if (c < B) {  // or from the previous path's point
      const int32_t* row = dirT + (int64_t)c * K;
#pragma unroll 4
      for (int k = lane; k < K; k += 32) sX[k] ^= row[k];
    }
    // Gaussians (:120-136) in two passes, so neither branch runs on a
    // partly idle warp: the central branch for every dimension, queueing
    // (in sB, free until the bridge) the dimensions that need the tail
    // branch; then the queue, densely
    int32_t* queue = reinterpret_cast<int32_t*>(sB);
    int nq = 0;
    for (int k0 = 0; k0 < K; k0 += 32) {
      const int k = k0 + lane;
      bool tail = false;
      if (k < K) {
        const float dp = (float)sX[k] * scale - 0.5f;
        if (gauss_is_central(dp)) sG[k] = gauss_central(dp);
        else tail = true;
      }
      const unsigned ball = __ballot_sync(kAll, tail);
      if (tail) queue[nq + __popc(ball & ((1u << lane) - 1u))] = k;
      nq += __popc(ball);
    }
    __syncwarp();
    for (int q = lane; q < nq; q += 32) {
      const int k = queue[q];
      sG[k] = gauss_tail((float)sX[k] * scale - 0.5f);
    }
    __syncwarp();
    for (int k = lane; k < K; k += 32) sB[k] = 0.0f;
    __syncwarp();
    if (lane < U) sB[(s_ind[0] - 1) * U + lane] = s_dat[0] * sG[lane];
    __syncwarp();
    for (int v = 1; v <= nlev; v++) {  // the bridge (:150-165), a level at a time
      // no step of a level reads a position another step of it writes, so a
      // batch of steps loads everything before it stores
      const int s0 = s_start[v], cnt = (s_start[v + 1] - s0) * U;
      constexpr int kBatch = 4;
      for (int p0 = lane; p0 < cnt; p0 += 32 * kBatch) {
        float val[kBatch];
        int dst[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
          const int p = p0 + 32 * q;
          dst[q] = -1;
          if (p < cnt) {
            const int i = s_order[s0 + p / U], u = p % U;
            const int j = s_ind[D + i] - 1, kk = s_ind[2 * D + i] - 1;
            const float tmp = s_dat[2 * D + i] * sB[kk * U + u] + s_dat[i] * sG[i * U + u];
            val[q] = j == -1 ? tmp : tmp + s_dat[D + i] * sB[j * U + u];
            dst[q] = (s_ind[i] - 1) * U + u;
          }
        }
#pragma unroll
        for (int q = 0; q < kBatch; q++)
          if (dst[q] >= 0) sB[dst[q]] = val[q];
      }
      __syncwarp();
    }
    for (int k = lane; k < K; k += 32)  // differences of consecutive dates (:167-175)
      sG[k] = k >= U ? sB[k] - sB[k - U] : sB[k];
    __syncwarp();
#pragma unroll
    for (int mm = 0; mm < kOpModels; mm++) {
      if (mm >= nm) break;
      const int m = m0 + mm;
      const float* cm = a.md_cs + (int64_t)m * U * U;
      const float* vol = a.md_vols + (int64_t)m * K;
      const float* dr = a.md_drifts + (int64_t)m * K;
      const float* disc = a.md_discts + (int64_t)m * a.num_discts;
      for (int k = lane; k < K; k += 32) {  // exp(drift + correlated noise * vol) (:188-215)
        const int d = k / U, u = k - d * U;
        float noise = 0.0f;
        for (int i = 0; i <= u; i++) noise = noise + sG[d * U + i] * cm[u * U + i];
        sB[k] = f32exp(dr[k] + noise * vol[k]);
      }
      __syncwarp();
      if (lane < U) {  // running product and prices (:216-218)
        const float st = a.md_sts[(int64_t)m * U + lane];
        float sc = 1.0f;
        constexpr int kBlk = 8;
        for (int d0 = 0; d0 < D; d0 += kBlk) {
          float e[kBlk];
#pragma unroll
          for (int q = 0; q < kBlk; q++) e[q] = d0 + q < D ? sB[(d0 + q) * U + lane] : 1.0f;
#pragma unroll
          for (int q = 0; q < kBlk; q++) {
            if (d0 + q < D) {
              sc = sc * e[q];
              sB[(d0 + q) * U + lane] = st * sc;
            }
          }
        }
      }
      __syncwarp();
      float pay = 0.0f;
      if constexpr (C == 3) {  // :266-292
        bool hit = false;
        for (int d = lane; d < D; d += 32) {
          const float* x = sB + d * 3;
          hit = hit || (x[0] <= 2630.6349999999998f || x[1] <= 8288.0f || x[2] <= 840.0f);
        }
        const bool cond = __any_sync(kAll, hit);
        if (lane == 0) {
          const float* last = sB + (D - 1) * 3;
          const float price1 = 100.0f * disc[0];
          const bool goto40 = cond && (last[0] < 3758.05f || last[1] < 11840.0f || last[2] < 1200.0f);
          const float amt = goto40 ? 1000.0f * fmin_payoff(last) : 1000.0f;
          pay = price1 + amt * disc[1];
        }
      }
      if (lane == 0) {
        acc[mm] += (double)pay;
        if (a.pay_out) a.pay_out[it * a.num_models + m0 + mm] = pay;
      }
      __syncwarp();  // sB is rewritten by the next model or path
    }
  }
#pragma unroll
  for (int mm = 0; mm < kOpModels; mm++) {  // the CTA's sum, warps in order
    if (mm >= nm) break;
    if (lane == 0) red[warp] = ok ? acc[mm] : __longlong_as_double(0x7ff8000000000000LL);
    __syncthreads();
    if (threadIdx.x == 0) {
      double sum = 0.0;
      for (int q = 0; q < kWarpPathWarps; q++) sum += red[q];
      partial[(int64_t)mm * gridDim.x + blockIdx.x] = sum;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// CTA per 32 paths (contract 3), for a bridge in which every step fills a date of
// its own from dates filled before -- what a Brownian bridge is; other index
// patterns are left to op_paths_warp_kernel.
// ---------------------------------------------------------------------------
// The bridge is then done in place: the Gaussian of step i waits in the slot of
// the date that step i fills, so one [date][underlying][path] array holds the
// paths (145 KB of shared memory), and every phase runs with all 32 lanes busy:
//   Gaussians   lane = dimension, a warp walking 8 paths of 32 dimensions: the
//               next path's Sobol integer is one XOR (Gray code); tail arguments
//               are queued per warp and evaluated 32 at a time
//   bridge      lane = path, the steps of a level spread over the warps
//   prices      lane = path: all warps but the last compute the exponentials
//               of a chunk of dates, while the last multiplies up and tests the
//               chunk before it, date by date
// A warp per path with its lanes over the dimensions spent 13 K warp instructions
// per path, a third of them on steps with few lanes busy (the bridge's levels, the
// product on 3 lanes); this spends 7 K, half in the Gaussians and a third in the
// exponentials, and is bound by issuing them.  131072 paths: 2531 us there, 1183
// here; 2048: 144 and 64; 20 warps, the most with 87 registers each (16 1236, 24
// 1188, 32 with spills 1283).
constexpr int kBlkWarps = 20, kBlkThreads = 32 * kBlkWarps;
constexpr int kBlkRuns = 8;    // paths of a Gaussian item
constexpr int kBlkDates = 57;  // dates of a chunk: three per computing warp

struct OpBlk {
  static constexpr int D = OpShape<3>::D, U = OpShape<3>::U, K = D * U;
  static constexpr int PS = 33;                                 // stride of a slot's 32 paths
  static constexpr int oB = 0;                                  // [K][PS] Gaussians, then the bridge
  static constexpr int oE = oB + (K * PS + 3) / 4 * 4;          // [2][kBlkDates][U][32] exponentials
  static constexpr int oBase = oE + 2 * kBlkDates * U * 32;     // [K] Sobol integers of the block's path 0
  static constexpr int oStep = oBase + (K + 3) / 4 * 4;         // [D] of l, k, j, sd | rw, lw: steps by level
  static constexpr int oStep2 = oStep + 4 * D;
  static constexpr int oStart = oStep2 + (2 * D + 3) / 4 * 4;   // [D + 2]
  static constexpr int oSlot = oStart + D + 2;                  // [D] date of step i
  static constexpr int oQueue = oSlot + D;                      // [kBlkWarps][64] arguments, then slots
  static constexpr int kWords = oQueue + kBlkWarps * 128;
  // the schedule's scratch, in B's place
  static constexpr int oWriter = oB, oLevel = oB + D, oCount = oB + 2 * D;
};

// Levels of the bridge's steps -- one more than those of the steps that filled the
// dates it reads -- and the steps sorted by level; false if a step fills a date
// twice or reads one not filled before it.  All threads of the CTA.
__device__ bool op_block_schedule(const int32_t* __restrict__ ind, const float* __restrict__ dat, float* sm,
                                  int& nlev) {
  using L = OpBlk;
  constexpr int D = L::D;
  const int i = threadIdx.x;
  static_assert(D <= kBlkThreads, "a thread per step");
  int* writer = reinterpret_cast<int*>(sm) + L::oWriter;
  int* level = reinterpret_cast<int*>(sm) + L::oLevel;
  int* count = reinterpret_cast<int*>(sm) + L::oCount;
  int* start = reinterpret_cast<int*>(sm) + L::oStart;
  int* slot = reinterpret_cast<int*>(sm) + L::oSlot;
  const bool step = i < D;
  const int l = step ? ind[i] - 1 : 0, j = step && i > 0 ? ind[D + i] - 1 : -1, k = step && i > 0 ? ind[2 * D + i] - 1 : 0;
  bool good = l >= 0 && l < D && j >= -1 && j < D && k >= 0 && k < D;
  if (step) writer[i] = D;
  __syncthreads();
  if (step && good && atomicMin(&writer[l], i) != D) good = false;
  if (step) {
    level[i] = 0;
    count[i] = 0;
    slot[i] = l;
  }
  if (!__syncthreads_and(good)) return false;
  // every date has its one writer: D steps, no date twice
  const int wk = step && i > 0 ? writer[k] : -1, wj = j >= 0 ? writer[j] : -1;
  if (!__syncthreads_and(!(step && i > 0) || (wk < i && wj < i))) return false;
  int lev = 0;
  for (bool moved = true; moved;) {  // as many rounds as there are levels
    int now = lev;
    if (step && i > 0) now = max(level[wk], wj >= 0 ? level[wj] : 0) + 1;
    moved = __syncthreads_or(now != lev);
    lev = now;
    if (step) level[i] = lev;
    __syncthreads();
  }
  int rank = 0;
  if (step && i > 0) rank = atomicAdd(&count[lev], 1);
  __syncthreads();
  if (i == 0) {
    int at = 0, v = 1;
    start[0] = start[1] = 0;
    for (; v < D && count[v] > 0; v++) start[v + 1] = at += count[v];
    start[D + 1] = v - 1;
  }
  __syncthreads();
  nlev = start[D + 1];
  if (step && i > 0) {
    const int at = start[lev] + rank;
    int* s4 = reinterpret_cast<int*>(sm) + L::oStep + 4 * at;
    s4[0] = l * L::U * L::PS;
    s4[1] = k * L::U * L::PS;
    s4[2] = j < 0 ? -1 : j * L::U * L::PS;
    sm[L::oStep + 4 * at + 3] = dat[i];
    sm[L::oStep2 + 2 * at] = dat[2 * D + i];
    sm[L::oStep2 + 2 * at + 1] = dat[D + i];
  }
  __syncthreads();
  return true;
}

// partial: [models of the launch][slots], this kernel's sums first, zeros after;
// *taken: whether this kernel priced the paths.
__global__ void __launch_bounds__(kBlkThreads, 1) op_paths_block_kernel(OpDev a, const int32_t* __restrict__ dirT,
                                                                       int m0, double* __restrict__ partial, int slots,
                                                                       int* __restrict__ taken) {
  using L = OpBlk;
  constexpr int D = L::D, U = L::U, K = L::K, PS = L::PS;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(16) float op_dyn[];
  float* const B_ = op_dyn + L::oB;
  int32_t* const base = reinterpret_cast<int32_t*>(op_dyn) + L::oBase;
  const int* const start = reinterpret_cast<const int*>(op_dyn) + L::oStart;
  const int* const slot = reinterpret_cast<const int*>(op_dyn) + L::oSlot;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* const qarg = op_dyn + L::oQueue + warp * 128;
  int* const qslot = reinterpret_cast<int*>(qarg) + 64;
  int nlev;
  const bool mine = op_block_schedule(a.bb_inds, a.bb_data, op_dyn, nlev);
  if (blockIdx.x == 0 && tid == 0) *taken = mine;
  if (!mine) return;
  const float sd0 = a.bb_data[0];
  const int first = slot[0] * U * PS;  // step 0 fills the first date
  const int bits = a.num_bits;
  const uint32_t mask = bits >= 32 ? 0xffffffffu : (1u << bits) - 1u;
  const float scale = ldexpf(1.0f, -bits);
  const int nm = min(kOpModels, a.num_models - m0);
  // block q holds the paths n = 32 q .. 32 q + 31 (of 1 .. num_mc_it)
  const int64_t nblk = (int64_t)a.num_mc_it / 32 + 1;
  const int64_t lo = nblk * blockIdx.x / gridDim.x, hi = nblk * (blockIdx.x + 1) / gridDim.x;
  double acc[kOpModels];
#pragma unroll
  for (int mm = 0; mm < kOpModels; mm++) acc[mm] = 0.0;
  for (int k = tid; k < K; k += kBlkThreads) base[k] = 0;
  uint32_t gray = 0;  // the Gray code whose directions base holds
  for (int64_t q = lo; q < hi; q++) {
    const uint32_t n0 = (uint32_t)(32 * q), g0 = ((n0 >> 1) ^ n0) & mask;
    for (int k = tid; k < K; k += kBlkThreads) {
      int32_t x = base[k];
      for (uint32_t f = g0 ^ gray; f != 0u; f &= f - 1u) x ^= dirT[(int64_t)(__ffs((int)f) - 1) * K + k];
      base[k] = x;
    }
    gray = g0;
    __syncthreads();
    // -- Gaussians (:120-136) of the Sobol points (:13-33) --
    int nq = 0;  // queued tail arguments
    auto flush = [&](int n) {
      __syncwarp();
      float g = 0.0f;
      int to = 0;
      if (lane < n) {
        g = gauss_tail(qarg[lane]);
        to = qslot[lane];
      }
      const float more = qarg[32 + lane];
      const int more_to = qslot[32 + lane];
      if (lane < n) B_[to] = g;
      __syncwarp();
      qarg[lane] = more;
      qslot[lane] = more_to;
      __syncwarp();
    };
    constexpr int kGroups = (K + 31) / 32, kParts = 32 / kBlkRuns;
    for (int it = warp; it < kGroups * kParts; it += kBlkWarps) {
      const int k = (it / kParts) * 32 + lane, r0 = (it % kParts) * kBlkRuns;
      const bool on = k < K;
      const int kk = on ? k : K - 1;
      const int to = (slot[kk / U] * U + kk % U) * PS + r0;
      int32_t v[5];
#pragma unroll
      for (int c = 0; c < 5; c++) v[c] = c < bits ? dirT[(int64_t)c * K + kk] : 0;
      int32_t x = base[kk];
      const int rg = r0 ^ (r0 >> 1);  // bits 2 .. 4
#pragma unroll
      for (int c = 2; c < 5; c++)
        if ((rg >> c) & 1) x ^= v[c];
#pragma unroll
      for (int t = 0; t < kBlkRuns; t++) {
        if (t > 0) x ^= v[(t & 1) ? 0 : (t & 2) ? 1 : 2];
        const float dp = (float)x * scale - 0.5f;
        const bool tail = on && !gauss_is_central(dp);
        const float g = gauss_central(dp);
        if (on && !tail) B_[to + t] = g;
        const unsigned ball = __ballot_sync(kAll, tail);
        if (tail) {
          const int at = nq + __popc(ball & ((1u << lane) - 1u));
          qarg[at] = dp;
          qslot[at] = to + t;
        }
        nq += __popc(ball);
        if (nq >= 32) {
          flush(32);
          nq -= 32;
        }
      }
    }
    flush(nq);
    __syncthreads();
    // -- bridge (:142-165) in place, a level at a time --
    if (warp < U) B_[first + warp * PS + lane] = sd0 * B_[first + warp * PS + lane];
    __syncthreads();
    for (int v = 1; v <= nlev; v++) {
      const int s0 = start[v], cnt = (start[v + 1] - s0) * U;
      for (int e = warp; e < cnt; e += kBlkWarps) {
        const int at = s0 + e / U, u = (e % U) * PS + lane;
        const float4 w4 = *reinterpret_cast<const float4*>(op_dyn + L::oStep + 4 * at);
        const float2 w2 = *reinterpret_cast<const float2*>(op_dyn + L::oStep2 + 2 * at);
        const int l = __float_as_int(w4.x), kk = __float_as_int(w4.y), j = __float_as_int(w4.z);
        float val = w2.x * B_[kk + u] + w4.w * B_[l + u];
        if (j >= 0) val = val + w2.y * B_[j + u];
        B_[l + u] = val;
      }
      __syncthreads();
    }
    // -- per model: exponentials (:188-215), prices and payoff (:216-292) --
    const int64_t n = 32 * q + lane;
    const bool path = n >= 1 && n <= a.num_mc_it;
#pragma unroll
    for (int mm = 0; mm < kOpModels; mm++) {
      if (mm >= nm) break;
      const int m = m0 + mm;
      const float* vol = a.md_vols + (int64_t)m * K;
      const float* dr = a.md_drifts + (int64_t)m * K;
      const float* st = a.md_sts + (int64_t)m * U;
      float cm[U][U];
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int i = 0; i <= u; i++) cm[u][i] = a.md_cs[((int64_t)m * U + u) * U + i];
      float sc[U], price[U];
      bool hit = false;
#pragma unroll
      for (int u = 0; u < U; u++) sc[u] = 1.0f;
      constexpr int kChunks = (D + kBlkDates - 1) / kBlkDates;
      for (int c = 0; c <= kChunks; c++) {
        if (warp < kBlkWarps - 1) {
          float* const E = op_dyn + L::oE + (c & 1) * kBlkDates * U * 32;
          const int d1 = min(D, (c + 1) * kBlkDates);
          for (int d = c * kBlkDates + warp; d < d1; d += kBlkWarps - 1) {
            float inc[U];  // differences of consecutive dates (:167-175)
#pragma unroll
            for (int u = 0; u < U; u++) {
              const float b = B_[(d * U + u) * PS + lane];
              inc[u] = d > 0 ? b - B_[((d - 1) * U + u) * PS + lane] : b;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
              float noise = 0.0f;
#pragma unroll
              for (int i = 0; i <= u; i++) noise = noise + inc[i] * cm[u][i];
              E[((d - c * kBlkDates) * U + u) * 32 + lane] = f32exp(dr[d * U + u] + noise * vol[d * U + u]);
            }
          }
        } else if (c > 0) {
          const float* const E = op_dyn + L::oE + ((c - 1) & 1) * kBlkDates * U * 32;
          const float s0 = st[0], s1 = st[1], s2 = st[2];
          const int nd = min(kBlkDates, D - (c - 1) * kBlkDates);
#pragma unroll 4
          for (int d = 0; d < nd; d++) {
#pragma unroll
            for (int u = 0; u < U; u++) sc[u] = sc[u] * E[(d * U + u) * 32 + lane];
            price[0] = s0 * sc[0];
            price[1] = s1 * sc[1];
            price[2] = s2 * sc[2];
            hit = hit || (price[0] <= 2630.6349999999998f || price[1] <= 8288.0f || price[2] <= 840.0f);
          }
        }
        __syncthreads();
      }
      if (warp == kBlkWarps - 1 && path) {
        const float* disc = a.md_discts + (int64_t)m * a.num_discts;
        const float price1 = 100.0f * disc[0];
        const bool goto40 = hit && (price[0] < 3758.05f || price[1] < 11840.0f || price[2] < 1200.0f);
        const float amt = goto40 ? 1000.0f * fmin_payoff(price) : 1000.0f;
        const float pay = price1 + amt * disc[1];
        acc[mm] += (double)pay;
        if (a.pay_out) a.pay_out[(n - 1) * a.num_models + m] = pay;
      }
    }
  }
  if (warp == kBlkWarps - 1) {
#pragma unroll
    for (int mm = 0; mm < kOpModels; mm++) {  // the CTA's sum, in a fixed order
      if (mm >= nm) break;
      double sum = acc[mm];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(kAll, sum, o);
      double* const out = partial + (int64_t)mm * slots;
      for (int b = blockIdx.x + lane * gridDim.x; b < slots; b += 32 * gridDim.x) out[b] = lane == 0 && b == blockIdx.x ? sum : 0.0;
    }
  }
}

// out[m0 + mm] = (f32)(sum of partial[mm][0 .. T)) / (f32)num_mc_it, one CTA
// per model, the same order on every run (T: the paths kernel's CTAs).
constexpr int kOpReduceThreads = 256;
__global__ void __launch_bounds__(kOpReduceThreads) op_reduce_kernel(const double* __restrict__ partial, int64_t T,
                                                                     int m0, int num_mc_it, float* __restrict__ out) {
  __shared__ double red[kOpReduceThreads];
  const int mm = blockIdx.x;
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < T; i += kOpReduceThreads) s += partial[(int64_t)mm * T + i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = kOpReduceThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[m0 + mm] = (float)red[0] / (float)num_mc_it;
}

// ---------------------------------------------------------------------------
// The reference's own order of the sum over paths (finpar/OptionPricing.fut:321
// as its golden outputs were produced): an f32 running sum in path order,
// s_k = fl(s_{k-1} + p_k).  Computed exactly, in parallel, from one fact: while
// s stays in one binade [2^e, 2^(e+1)) -- f32 grid spacing u = 2^(e-23) -- and
// 0 <= p_k < 2^e, fl(s + p_k) = s + u * t_k, where t_k is p_k / u rounded to the
// nearest integer, and on a tie to the one that makes s / u even.  So payoffs
// act on s / u as integer additions that depend on s through its parity alone,
// and a run of them as a pair of additions, one per parity; such pairs compose.
//
//   op_seq_maps_kernel  a warp per block of kSeqBlock payoffs: the block's pair
//                       for the exponent that the mean payoff (already known
//                       from the f64 sum) predicts, or the two it lies between;
//   op_seq_reduce_kernel  (maps null: no pairs) one CTA per model: composes the blocks' pairs from the
//                       running sum on, up to the first block in which the sum
//                       leaves its binade; that block's payoffs are added one
//                       after the other in f32, as the sequential loop does (and
//                       so is every block holding a payoff that is not a finite
//                       nonnegative normal number below 2^e).
//
// The sum leaves its binade about once per doubling of the paths: for 8.4 M
// payoffs 15 blocks are walked and 8 steps composed, one after the other, and
// that chain's latency (4 us each: the pairs' and payoffs' loads from L2, two
// scans, 256 additions) bounds the second kernel; the first is bound by its
// instructions.  One CTA walking all payoffs 16384 at a time, as before, took
// 7 us per step, 4.01 ms in all; now 26 + 105 us.
// ---------------------------------------------------------------------------
constexpr int kSeqBlock = 256;    // payoffs per block: 8 per lane of a warp
constexpr int kSeqThreads = 1024;
constexpr int kSeqPer = 4;        // blocks per thread and step of the composition
constexpr int kSeqMaps = 2;       // exponents a block's pair is made for, at most
constexpr uint32_t kSeqLim = 1u << 24;   // s / u reaching 2^24 leaves the binade
constexpr uint32_t kSeqNone = 1u << 30;  // no pair: larger than any sum in the binade

// What a run of payoffs adds to s / u, by the parity of s / u before it.
struct SeqPair {
  uint32_t a0, a1;
};
__device__ __forceinline__ uint32_t seq_cap(uint32_t v) { return min(v, kSeqNone); }
// f, then g
__device__ __forceinline__ SeqPair seq_then(SeqPair f, SeqPair g) {
  return {seq_cap(f.a0 + ((f.a0 & 1u) ? g.a1 : g.a0)), seq_cap(f.a1 + ((f.a1 & 1u) ? g.a0 : g.a1))};
}
// The run a followed by payoff p, for sums in binade e; false when p needs a
// step of its own in f32.
__device__ __forceinline__ bool seq_add(SeqPair& a, float p, int e) {
  const uint32_t b = __float_as_uint(p);
  if (b == 0u) return true;  // +0
  const int be = (int)(b >> 23);  // sign and exponent: above 0xfe is negative, infinite or NaN
  const int d = e - (be - 127);   // p in [2^(e-d), 2^(e-d+1))
  if (be == 0 || be > 0xfe || d < 1) return false;
  const uint32_t m = (b & 0x7fffffu) | 0x800000u;
  const int sh = min(d, 26);  // beyond that p is less than half a unit, as at 26
  const uint32_t t = m >> sh, rem = m & ((1u << sh) - 1u), half = 1u << (sh - 1);
  const bool tie = rem == half;
  const uint32_t up = rem > half;
  a.a0 = seq_cap(a.a0 + t + (tie ? ((a.a0 + t) & 1u) : up));
  a.a1 = seq_cap(a.a1 + t + (tie ? ((a.a1 + t + 1u) & 1u) : up));
  return true;
}

// The exponents block b's pairs are made for: those of the sum that the mean
// payoff predicts before the block, give or take a quarter.
__device__ __forceinline__ int seq_exponent(float s) { return (int)((__float_as_uint(s) >> 23) & 0xffu) - 127; }
__device__ __forceinline__ void seq_exponents(float mean, int64_t b, int& lo, int& hi) {
  const float s = mean * (float)(b * kSeqBlock);
  lo = seq_exponent(s * 0.8f);
  hi = seq_exponent(s * 1.25f);
}

// The pair of a block's payoffs for binade e, in every lane of the warp.
__device__ __forceinline__ SeqPair seq_block_pair(const float (&v)[kSeqBlock / 32], int n, int e) {
  constexpr int PL = kSeqBlock / 32;
  const int lane = threadIdx.x & 31;
  SeqPair a{0u, 0u};
  bool ok = true;
#pragma unroll
  for (int j = 0; j < PL; j++)
    if (lane * PL + j < n) ok = ok && seq_add(a, v[j], e);
  if (!ok) a = {kSeqNone, kSeqNone};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {  // lanes in order: lane l holds lanes l .. l + 2 o - 1
    const SeqPair g{__shfl_down_sync(0xffffffffu, a.a0, o), __shfl_down_sync(0xffffffffu, a.a1, o)};
    if ((lane & (2 * o - 1)) == 0) a = seq_then(a, g);
  }
  return {__shfl_sync(0xffffffffu, a.a0, 0), __shfl_sync(0xffffffffu, a.a1, 0)};
}
// A block's payoffs, consecutive ones per lane; true when all are +0.
__device__ __forceinline__ bool seq_load_block(const float* __restrict__ p, int num_models, int64_t b, int n,
                                               float (&v)[kSeqBlock / 32]) {
  constexpr int PL = kSeqBlock / 32;
  static_assert(PL % 4 == 0, "16-byte loads");
  const int lane = threadIdx.x & 31;
  const float* q = p + (b * kSeqBlock + lane * PL) * num_models;
  uint32_t any = 0;
  if (num_models == 1 && n == kSeqBlock && ((uintptr_t)q & 15) == 0) {
#pragma unroll
    for (int j = 0; j < PL; j += 4) {
      const float4 t = *reinterpret_cast<const float4*>(q + j);
      v[j] = t.x;
      v[j + 1] = t.y;
      v[j + 2] = t.z;
      v[j + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < PL; j++) v[j] = lane * PL + j < n ? q[(int64_t)j * num_models] : 0.0f;
  }
#pragma unroll
  for (int j = 0; j < PL; j++) any |= __float_as_uint(v[j]);
  return __all_sync(0xffffffffu, any == 0u);
}

// maps[mm][kSeqMaps][block].  A block of zeros has (0, 0) for every exponent,
// written with kSeqZeros as the second number, so that it is known as one.
constexpr uint32_t kSeqZeros = 0x80000000u;
__global__ void __launch_bounds__(256) op_seq_maps_kernel(const float* __restrict__ pay, int64_t N, int num_models,
                                                          int m0, const float* __restrict__ mean,
                                                          SeqPair* __restrict__ maps) {
  const int lane = threadIdx.x & 31, mm = blockIdx.y;
  const int64_t blocks = (N + kSeqBlock - 1) / kSeqBlock;
  const int64_t b = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (b >= blocks) return;
  const int n = (int)min((int64_t)kSeqBlock, N - b * kSeqBlock);
  float v[kSeqBlock / 32];
  const bool zeros = seq_load_block(pay + m0 + mm, num_models, b, n, v);
  int lo, hi;
  seq_exponents(mean[m0 + mm], b, lo, hi);
  for (int e = lo; e <= hi; e++) {
    SeqPair a{0u, kSeqZeros};
    if (!zeros) a = seq_block_pair(v, n, e);
    if (lane == 0) maps[((int64_t)mm * kSeqMaps + (e - lo)) * blocks + b] = a;
  }
}

__global__ void __launch_bounds__(kSeqThreads) op_seq_reduce_kernel(const float* __restrict__ pay, int64_t N,
                                                                    int num_models, int m0, int num_mc_it,
                                                                    const SeqPair* __restrict__ maps,
                                                                    float* __restrict__ out) {
  constexpr int NW = kSeqThreads / 32;
  const int mm = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* p = pay + m0 + mm;  // path k at p[k * num_models]
  const int64_t blocks = (N + kSeqBlock - 1) / kSeqBlock;
  const float mean = out[m0 + mm];
  const SeqPair* mp = maps + (int64_t)mm * blocks * kSeqMaps;
  __shared__ __align__(16) float s_pay[kSeqBlock];
  __shared__ SeqPair s_warp[NW];
  __shared__ uint32_t s_base;
  __shared__ int s_stop;
  __shared__ float s_sum;
  if (mean != mean) return;  // so is this sum; or the paths kernel priced nothing (bad bridge)
  float s = 0.0f;
  int64_t b = 0;
  while (b < blocks) {
    const uint32_t sb = __float_as_uint(s);
    const bool zero = sb == 0u;                                      // only blocks of zeros have a pair
    const bool normal = (sb >> 23) - 1u < 0xfeu;                      // positive and normal
    const int e = normal ? (int)(sb >> 23) - 127 : 0;
    int done = 0;  // blocks composed
    if (maps && (zero || normal)) {
      const uint32_t S0 = zero ? 0u : (sb & 0x7fffffu) | 0x800000u;  // s / u
      // the pairs of blocks b + kSeqPer * tid ..; where the prediction missed
      // the exponent (other: this far) a warp makes the pair from the payoffs
      SeqPair f[kSeqPer];
      bool known = true;
#pragma unroll
      for (int q = 0; q < kSeqPer; q++) {
        const int64_t bb = b + (int64_t)tid * kSeqPer + q;
        f[q] = {kSeqNone, kSeqNone};
        if (bb < blocks) {
          int lo, hi;
          seq_exponents(mean, bb, lo, hi);
          const bool made = normal && e >= lo && e <= hi;
          const SeqPair g = mp[(made ? e - lo : 0) * blocks + bb];
          if (g.a1 == kSeqZeros) f[q] = {0u, 0u};
          else if (made) f[q] = g;
          else if (normal) known = false;
        }
      }
      if (tid == 0) s_stop = kSeqThreads * kSeqPer;
      // the first blocks unknown: made here, one per warp
      const bool miss = __syncthreads_or(tid * kSeqPer < NW && !known);
      if (miss) {
        const int64_t bb = b + warp;
        SeqPair a{kSeqNone, kSeqNone};
        if (bb < blocks) {
          const int n = (int)min((int64_t)kSeqBlock, N - bb * kSeqBlock);
          float v[kSeqBlock / 32];
          const bool zeros = seq_load_block(p, num_models, bb, n, v);
          a = zeros ? SeqPair{0u, 0u} : seq_block_pair(v, n, e);
        }
        if (lane == 0) s_warp[warp] = a;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kSeqPer; q++)
          f[q] = tid * kSeqPer + q < NW ? s_warp[tid * kSeqPer + q] : SeqPair{kSeqNone, kSeqNone};
        __syncthreads();
      }
      SeqPair mine = f[0];
#pragma unroll
      for (int q = 1; q < kSeqPer; q++) mine = seq_then(mine, f[q]);
      SeqPair x = mine;  // inclusive scan over the warp
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const SeqPair y{__shfl_up_sync(0xffffffffu, x.a0, o), __shfl_up_sync(0xffffffffu, x.a1, o)};
        if (lane >= o) x = seq_then(y, x);
      }
      if (lane == 31) s_warp[warp] = x;
      SeqPair before{__shfl_up_sync(0xffffffffu, x.a0, 1), __shfl_up_sync(0xffffffffu, x.a1, 1)};
      if (lane == 0) before = {0u, 0u};
      __syncthreads();
      if (warp == 0) {
        SeqPair y = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const SeqPair g{__shfl_up_sync(0xffffffffu, y.a0, o), __shfl_up_sync(0xffffffffu, y.a1, o)};
          if (lane >= o) y = seq_then(g, y);
        }
        s_warp[lane] = y;
      }
      __syncthreads();
      if (warp > 0) before = seq_then(s_warp[warp - 1], before);
      uint32_t run = S0 + ((S0 & 1u) ? before.a1 : before.a0);  // s / u before this thread's blocks
      const uint32_t start = run;
      int cross = kSeqThreads * kSeqPer;
#pragma unroll
      for (int q = 0; q < kSeqPer; q++) {
        const uint32_t nx = run + ((run & 1u) ? f[q].a1 : f[q].a0);
        if (cross == kSeqThreads * kSeqPer) {
          if (nx >= kSeqLim) cross = tid * kSeqPer + q; else run = nx;
        }
      }
      if (cross < kSeqThreads * kSeqPer) atomicMin(&s_stop, cross);
      __syncthreads();
      done = s_stop;
      // s / u there, from the thread whose blocks hold the stop (or the last one)
      const int owner = min(done / kSeqPer, kSeqThreads - 1);
      if (tid == owner) s_base = done == owner * kSeqPer ? start : run;
      __syncthreads();
      if (!zero) s = ldexpf((float)s_base, e - 23);  // exact: s_base < 2^24
      b += done;
    }
    if (b < blocks && done < kSeqThreads * kSeqPer) {  // block b, payoff by payoff
      const int n = (int)min((int64_t)kSeqBlock, N - b * kSeqBlock);
      __syncthreads();
      for (int k = tid; k < kSeqBlock; k += kSeqThreads) s_pay[k] = k < n ? p[(b * kSeqBlock + k) * num_models] : 0.0f;
      __syncthreads();
      if (tid == 0) {
        float v = s;
        if (n == kSeqBlock) {
#pragma unroll 8
          for (int k = 0; k < kSeqBlock; k += 4) {
            const float4 q = *reinterpret_cast<const float4*>(s_pay + k);
            v = (((v + q.x) + q.y) + q.z) + q.w;
          }
        } else {
          for (int k = 0; k < n; k++) v = v + s_pay[k];
        }
        s_sum = v;
      }
      __syncthreads();
      s = s_sum;
      b++;
    }
  }
  if (tid == 0) out[m0 + mm] = s / (float)num_mc_it;
}

constexpr size_t kWarpSmem3 = sizeof(float) * OpWarpSmem<3>::kWords;
constexpr size_t kBlkSmem = sizeof(float) * OpBlk::kWords;
static_assert(kBlkSmem <= 227 * 1024, "one CTA per SM");

// CTAs of the paths kernel for `paths` paths of contract c: eight 128-thread
// CTAs per SM (thread per path), or two 7-warp CTAs per SM (warp per path,
// contract 3); fewer when there are fewer paths.
int64_t op_ctas(const futhark_context* ctx, int c, int64_t paths) {
  const int64_t per = c == 3 ? kWarpPathWarps : kOpThreads;  // paths a CTA takes at once
  const int64_t want = (int64_t)ctx->num_sms * (c == 3 ? 2 : 8);
  return std::max<int64_t>(1, std::min(want, (paths + per - 1) / per));
}
constexpr int kOpMaxCtasPerSm = 8;

// Shapes and sizes of one pricing (lock held); the message names the failure.
int op_validate(futhark_context* ctx, const op_args* q) {
  const int c = q->contract_number;
  if (q->num_models < 0 || q->num_und < 0 || q->num_dates < 0 || q->num_discts < 0 || q->num_bits < 0)
    return set_error(ctx, FUTHARK_PROGRAM_ERROR, "option pricing: negative dimension");
  if (q->num_mc_it < 0)  // iota of a negative length (:315)
    return set_error(ctx, FUTHARK_PROGRAM_ERROR, "option pricing: negative num_mc_it");
  if (q->num_bits > 32)
    return set_error(ctx, FUTHARK_PROGRAM_ERROR, "option pricing: num_bits above 32 is not supported");
  const int need_d[4] = {0, 1, 5, 367}, need_u[4] = {0, 1, 3, 3}, need_disc[4] = {0, 1, 5, 2};
  if (c >= 1 && c <= 3 && q->num_models > 0) {
    if (q->num_dates != need_d[c] || q->num_und != need_u[c])
      return set_error(ctx, FUTHARK_PROGRAM_ERROR,
                       "option pricing: contract " + std::to_string(c) + " needs [" + std::to_string(need_d[c]) +
                           "][" + std::to_string(need_u[c]) + "] paths (size coercion failed)");
    if (q->num_discts < need_disc[c])
      return set_error(ctx, FUTHARK_PROGRAM_ERROR, "option pricing: too few discount factors for the contract");
  }
  return 0;
}

// Scratch: the CTAs' partial sums, then (contract 3) the transposed
// direction numbers.
size_t partial_bytes(const futhark_context* ctx) {
  return (sizeof(double) * (size_t)kOpModels * (size_t)ctx->num_sms * kOpMaxCtasPerSm + 255) & ~(size_t)255;
}
size_t dirs_bytes(const op_args* q) {
  const size_t dirs = q->contract_number == 3
                          ? sizeof(int32_t) * (size_t)std::max(0, q->num_dates) * std::max(0, q->num_und) *
                                std::max(0, q->num_bits)
                          : 0;
  return (dirs + 255) & ~(size_t)255;
}
// (reference order) every path's payoff, [path][model]
size_t payoff_bytes(const futhark_context* ctx, const op_args* q) {
  if (ctx->reduce_order != 1) return 0;
  return sizeof(float) * (size_t)std::max(0, q->num_mc_it) * (size_t)std::max(0, q->num_models);
}
// (reference order) the block pairs of one launch's models
size_t maps_bytes(const futhark_context* ctx, const op_args* q) {
  if (ctx->reduce_order != 1 || q->num_mc_it <= 0) return 0;
  const size_t blocks = ((size_t)q->num_mc_it + kSeqBlock - 1) / kSeqBlock;
  return sizeof(SeqPair) * kSeqMaps * blocks * (size_t)std::min(kOpModels, std::max(0, q->num_models));
}
size_t scratch_for(const futhark_context* ctx, const op_args* q) {
  return partial_bytes(ctx) + dirs_bytes(q) + maps_bytes(ctx, q) + payoff_bytes(ctx, q) + 256;
}

// Enqueues one pricing (lock held, device set, shapes valid, scratch large enough).
int op_launch(futhark_context* ctx, const op_args* q, float* out, void* scratch) {
  if (q->num_models == 0) return 0;
  const int c = q->contract_number;
  const bool priced = c >= 1 && c <= 3 && q->num_mc_it > 0;
  float* pay_out = priced && ctx->reduce_order == 1
                       ? reinterpret_cast<float*>(static_cast<char*>(scratch) + partial_bytes(ctx) + dirs_bytes(q) +
                                                  maps_bytes(ctx, q))
                       : nullptr;
  SeqPair* maps = reinterpret_cast<SeqPair*>(static_cast<char*>(scratch) + partial_bytes(ctx) + dirs_bytes(q));
  OpDev a{q->num_mc_it, q->num_bits, q->num_models, q->num_discts, q->dir_vs, q->md_cs, q->md_vols, q->md_drifts,
          q->md_sts, q->md_detvals, q->md_discts, q->bb_inds, q->bb_data, pay_out};
  double* partial = static_cast<double*>(scratch);
  const int64_t T = priced ? op_ctas(ctx, c, q->num_mc_it) : 0;  // CTAs, one partial each
  int32_t* dirT = reinterpret_cast<int32_t*>(static_cast<char*>(scratch) + partial_bytes(ctx));
  if (priced && c == 3) {
    cudaError_t e = cudaFuncSetAttribute((const void*)op_paths_warp_kernel<3>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWarpSmem3);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute((const void*)op_paths_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kBlkSmem);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "option pricing attributes");
    const int64_t kb = (int64_t)q->num_dates * q->num_und * q->num_bits;
    op_transpose_dirs_kernel<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((kb + 255) / 256, 1024)), 256, 0,
                               ctx->stream>>>(q->dir_vs, q->num_dates * q->num_und, q->num_bits, dirT);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(ctx, e, "option pricing transpose launch");
  }
  for (int m0 = 0; m0 < q->num_models; m0 += kOpModels) {
    const int nm = std::min(kOpModels, q->num_models - m0);
    if (priced) {
      cudaError_t e_;
      if (c == 1) op_paths_kernel<1><<<(unsigned)T, kOpThreads, 0, ctx->stream>>>(a, m0, partial);
      else if (c == 2) op_paths_kernel<2><<<(unsigned)T, kOpThreads, 0, ctx->stream>>>(a, m0, partial);
      else {
        // where the partial sums end: contract 3 has at most two of eight CTAs per SM
        int* taken = reinterpret_cast<int*>(static_cast<char*>(scratch) + partial_bytes(ctx) - 256);
        const int64_t nblk = (int64_t)q->num_mc_it / 32 + 1;
        op_paths_block_kernel<<<(unsigned)std::min<int64_t>(ctx->num_sms, std::min(T, nblk)), kBlkThreads, kBlkSmem,
                                ctx->stream>>>(a, dirT, m0, partial, (int)T, taken);
        if ((e_ = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, e_, "option pricing launch");
        op_paths_warp_kernel<3><<<(unsigned)T, kWarpPathWarps * 32, kWarpSmem3, ctx->stream>>>(a, dirT, m0, partial,
                                                                                              taken);
      }
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(ctx, e, "option pricing launch");
    }
    // other contracts price every path at 0 (:302); no paths gives 0 / 0
    op_reduce_kernel<<<nm, kOpReduceThreads, 0, ctx->stream>>>(partial, T, m0, q->num_mc_it, out);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(ctx, e, "option pricing reduction launch");
    if (pay_out) {  // the reference's order replaces the f64 one (NaN stays NaN)
      const int64_t blocks = ((int64_t)q->num_mc_it + kSeqBlock - 1) / kSeqBlock;
      // a single block is walked: its pair would only cost a launch (one path 18.9 us with it, 15 without)
      if (blocks == 1) {
        maps = nullptr;
      } else {
        op_seq_maps_kernel<<<dim3((unsigned)((blocks + 7) / 8), nm), 256, 0, ctx->stream>>>(
            pay_out, q->num_mc_it, q->num_models, m0, out, maps);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, e, "option pricing ordered reduction launch");
      }
      op_seq_reduce_kernel<<<nm, kSeqThreads, 0, ctx->stream>>>(pay_out, q->num_mc_it, q->num_models, m0,
                                                                 q->num_mc_it, maps, out);
      e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(ctx, e, "option pricing ordered reduction launch");
    }
  }
  return 0;
}

}  // namespace

extern "C" {

FUT_ARRAY_API(f32_1d, float, 1, int64_t dim0)
FUT_ARRAY_API(f32_2d, float, 2, int64_t dim0, int64_t dim1)
FUT_ARRAY_API(f32_3d, float, 3, int64_t dim0, int64_t dim1, int64_t dim2)
FUT_ARRAY_API(i32_2d, int32_t, 2, int64_t dim0, int64_t dim1)

int futhark_entry_main(struct futhark_context* ctx, struct futhark_f32_1d** out0, int32_t contract_number,
                       int32_t num_mc_it, const struct futhark_i32_2d* dir_vs, const struct futhark_f32_3d* md_cs,
                       const struct futhark_f32_3d* md_vols, const struct futhark_f32_3d* md_drifts,
                       const struct futhark_f32_2d* md_sts, const struct futhark_f32_2d* md_detvals,
                       const struct futhark_f32_2d* md_discts, const struct futhark_i32_2d* bb_inds,
                       const struct futhark_f32_2d* bb_data) {
  std::lock_guard<std::mutex> g(ctx->mu);
  if (!ctx->ok) return set_error(ctx, FUTHARK_PROGRAM_ERROR, "context has no usable CUDA device");
  if (!out0 || !dir_vs || !md_cs || !md_vols || !md_drifts || !md_sts || !md_detvals || !md_discts || !bb_inds ||
      !bb_data)
    return set_error(ctx, FUTHARK_PROGRAM_ERROR, "null array");
  const int64_t M = md_vols->shape[0], D = md_vols->shape[1], U = md_vols->shape[2];
  const int64_t B = dir_vs->shape[1], ND = md_discts->shape[1];
  // the entry point's size parameters (OptionPricing.fut:304-314)
  const bool sizes_ok = dir_vs->shape[0] == D * U && md_cs->shape[0] == M && md_cs->shape[1] == U &&
                        md_cs->shape[2] == U && md_drifts->shape[0] == M && md_drifts->shape[1] == D &&
                        md_drifts->shape[2] == U && md_sts->shape[0] == M && md_sts->shape[1] == U &&
                        md_detvals->shape[0] == M && md_detvals->shape[1] == 1 && md_discts->shape[0] == M &&
                        bb_inds->shape[0] == 3 && bb_inds->shape[1] == D && bb_data->shape[0] == 3 &&
                        bb_data->shape[1] == D;
  if (!sizes_ok) return set_error(ctx, FUTHARK_PROGRAM_ERROR, "option pricing: input sizes do not match");
  if (M > INT32_MAX || D > INT32_MAX || U > INT32_MAX || B > INT32_MAX || ND > INT32_MAX)
    return set_error(ctx, FUTHARK_PROGRAM_ERROR, "option pricing: dimension too large");
  op_args q{contract_number, num_mc_it, (int32_t)B, (int32_t)M, (int32_t)U, (int32_t)D, (int32_t)ND,
            dir_vs->data, md_cs->data, md_vols->data, md_drifts->data, md_sts->data, md_detvals->data,
            md_discts->data, bb_inds->data, bb_data->data};
  int rc = op_validate(ctx, &q);
  if (rc) return rc;
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "option pricing");
  // the bridge's indices select dates (:155-169, unchecked in the reference)
  if (contract_number >= 1 && contract_number <= 3 && M > 0 && D > 0) {
    std::vector<int32_t> ind(3 * D);
    e = cudaMemcpyAsync(ind.data(), bb_inds->data, sizeof(int32_t) * ind.size(), cudaMemcpyDeviceToHost,
                        ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "option pricing: reading bb_inds");
    // bi[i] for every i; li[i] (0: no left point) and ri[i] from i = 1 on
    bool in_range = ind[0] >= 1 && ind[0] <= D;
    for (int64_t i = 1; i < D; i++)
      in_range = in_range && ind[i] >= 1 && ind[i] <= D && ind[D + i] >= 0 && ind[D + i] <= D &&
                 ind[2 * D + i] >= 1 && ind[2 * D + i] <= D;
    if (!in_range)
      return set_error(ctx, FUTHARK_PROGRAM_ERROR, "option pricing: bb_inds selects a date outside the path");
  }
  const int64_t d1[1] = {M};
  futhark_f32_1d* out = alloc_array<futhark_f32_1d>(d1, 1);
  if (!out || !ensure_scratch(ctx, scratch_for(ctx, &q))) {
    drop_array(out);
    return set_error(ctx, FUTHARK_OUT_OF_MEMORY, "out of device memory");
  }
  rc = op_launch(ctx, &q, out->data, ctx->scratch);
  if (!rc) {
    e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) rc = cuda_fail(ctx, e, "option pricing");
  }
  if (rc) {
    drop_array(out);
    return rc;
  }
  *out0 = out;
  return 0;
}

size_t op_scratch_bytes(struct futhark_context* ctx, const struct op_args* args) {
  if (!ctx || !args || !ctx->ok) return 0;
  return scratch_for(ctx, args);
}
int op_price_f32(struct futhark_context* ctx, const struct op_args* args, float* out, void* scratch) {
  std::lock_guard<std::mutex> g(ctx->mu);
  if (!ctx->ok) return set_error(ctx, FUTHARK_PROGRAM_ERROR, "context has no usable CUDA device");
  if (!args || (!out && args->num_models > 0)) return set_error(ctx, FUTHARK_PROGRAM_ERROR, "null argument");
  int rc = op_validate(ctx, args);
  if (rc) return rc;
  if (((uintptr_t)scratch & 255) != 0)
    return set_error(ctx, FUTHARK_PROGRAM_ERROR, "option pricing: scratch is not on a 256-byte boundary");
  const cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "option pricing");
  return op_launch(ctx, args, out, scratch);
}
int op_check(struct futhark_context* ctx) {
  std::lock_guard<std::mutex> g(ctx->mu);
  if (!ctx->ok) return set_error(ctx, FUTHARK_PROGRAM_ERROR, "context has no usable CUDA device");
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(ctx, e, "option pricing");
}
void* op_context_stream(struct futhark_context* ctx) { return ctx && ctx->ok ? (void*)ctx->stream : nullptr; }
int op_context_set_reduction_order(struct futhark_context* ctx, int32_t order) {
  if (!ctx) return FUTHARK_PROGRAM_ERROR;
  std::lock_guard<std::mutex> g(ctx->mu);
  if (order != OP_ORDER_F64 && order != OP_ORDER_SEQUENTIAL_F32)
    return set_error(ctx, FUTHARK_PROGRAM_ERROR, "option pricing: unknown reduction order");
  ctx->reduce_order = order;
  return 0;
}

}  // extern "C"
