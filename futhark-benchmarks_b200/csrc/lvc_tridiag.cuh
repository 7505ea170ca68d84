// Batched tridiagonal solvers: the tridagNested* entry points of
// misc/ocean-sim/tridiag-test.fut:14-26 (f32, one system per row of
// [rows][m] arrays).
//
//   FORM 0  tridagSeq (misc/ocean-sim/tridiag.fut:81-95): normalised Thomas.
//   FORM 1  tridagPar (misc/ocean-sim/tridiag.fut:4-79): the three scans --
//           4-tuple matrix scan for the pivots, two linear-function scans --
//           folded left to right.
//
// Two kernels, one lane per system in each: lvc_tridag_row_kernel holds the rows
// of a warp's systems in shared memory (m up to about 3600, and up to about 1600
// whatever the number of rows); lvc_tridag_kernel (any m) reads rows in place.
// Each recurrence runs in the reference's operation
// order with every product, sum and quotient explicitly rounded (no fused
// multiply-add), so a system's solution is bit for bit the one the CPU
// restatement of the same fold gives.  The work is a handful of operations per
// element against 20 bytes of HBM traffic (four inputs, one output): HBM is the
// floor, and the latency of the sequential recurrence what stands above it.
// lvc_tridag_kernel keeps its per-row scratch (the pivots of FORM 1, the
// normalised super-diagonal of FORM 0) in a global [element][row] buffer --
// consecutive threads at consecutive addresses -- and the right-hand side of the
// backward pass in the output row itself.
#pragma once

#include <cstdint>

#include "exact_math.cuh"
#include "lvc_line.cuh"  // mbarrier and bulk-copy helpers

namespace lvc {

// Raised by a bounded wait that gave up (lvc_wait_selftest_kernel below);
// reset and read by the host after each solve and self-test.
__device__ int lvc_tridag_err;

constexpr int kTriThreads = 128;  // threads (systems) per CTA of lvc_tridag_kernel

// Self-test of the bounded wait that the rollback kernels' bulk-copy and
// cluster waits use (mbar_wait): one warp waits on a fresh mbarrier for at
// most `polls` polls.  With arrive == 0 nothing ever completes its phase (no
// copy targets it and no thread arrives), so the wait runs out and the kernel
// raises lvc_tridag_err, which the host reports as a timed-out wait; with
// arrive != 0 lane 0 arrives first and the wait succeeds.  No asynchronous
// operation is in flight either way, so the CTA may exit at once.
__global__ void lvc_wait_selftest_kernel(int polls, int arrive) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncwarp();
  if (arrive && threadIdx.x == 0)
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&bar)) : "memory");
  const bool ok = mbar_wait(&bar, 0, polls);
  if (!ok && threadIdx.x == 0) atomicExch(&lvc_tridag_err, 1);
}

__device__ __forceinline__ float tri_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float tri_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float tri_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float tri_div(float a, float b) { return __fdiv_rn(a, b); }
// 1 / x correctly rounded: the same value as tri_div(1.0f, x), cheaper
__device__ __forceinline__ float tri_rcp(float x) { return __frcp_rn(x); }
template <int FORM>
__global__ void __launch_bounds__(kTriThreads) lvc_tridag_kernel(int64_t rows, int m, const float* __restrict__ a,
                                                                const float* __restrict__ b,
                                                                const float* __restrict__ c,
                                                                const float* __restrict__ y,
                                                                float* __restrict__ out,
                                                                float* __restrict__ gscratch) {
  const int64_t r = (int64_t)blockIdx.x * kTriThreads + threadIdx.x;
  if (r >= rows) return;  // no barrier below: threads are independent
  const float* ar = a + r * m;
  const float* br = b + r * m;
  const float* cr = c + r * m;
  const float* yr = y + r * m;
  float* o = out + r * m;
  float* scr = gscratch + r;
  const int64_t sstride = rows;  // element i of this row's scratch at scr[i * sstride]

  if constexpr (FORM == 0) {
    // forward: cp_i = c_i / (b_i - a_i cp_{i-1}), yp_i = (y_i - a_i yp_{i-1}) / (...)  (:82-91)
    float cp = tri_div(cr[0], br[0]);
    float yp = tri_div(yr[0], br[0]);
    scr[0] = cp;
    o[0] = yp;
    for (int i = 1; i < m; i++) {
      const float ai = ar[i];
      const float nf = tri_rcp(tri_sub(br[i], tri_mul(ai, cp)));
      cp = tri_mul(cr[i], nf);
      yp = tri_mul(tri_sub(yr[i], tri_mul(ai, yp)), nf);
      scr[i * sstride] = cp;
      o[i] = yp;
    }
    // backward: x_i = yp_i - cp_i x_{i+1}  (:92-95)
    float x = yp;
    for (int i = m - 2; i >= 0; i--) {
      x = tri_sub(o[i], tri_mul(scr[i * sstride], x));
      o[i] = x;
    }
  } else {
    // Recurrence 1 (:9-33): b'_i from the scan of (b_i, -a_i c_{i-1}, 1, 0)
    const float b0 = br[0];
    float s0 = 1.0f, s1 = 0.0f, s2 = 0.0f, s3 = 1.0f;
    for (int i = 0; i < m; i++) {
      float m0 = 1.0f, m1 = 0.0f, m2 = 0.0f, m3 = 1.0f;
      if (0 < i) {
        m0 = br[i];
        m1 = tri_sub(0.0f, tri_mul(ar[i], cr[i - 1]));
        m2 = 1.0f;
        m3 = 0.0f;
      }
      const float value = tri_rcp(tri_mul(s0, m0));
      const float n0 = tri_mul(tri_add(tri_mul(m0, s0), tri_mul(m1, s2)), value);
      const float n1 = tri_mul(tri_add(tri_mul(m0, s1), tri_mul(m1, s3)), value);
      const float n2 = tri_mul(tri_add(tri_mul(m2, s0), tri_mul(m3, s2)), value);
      const float n3 = tri_mul(tri_add(tri_mul(m2, s1), tri_mul(m3, s3)), value);
      s0 = n0;
      s1 = n1;
      s2 = n2;
      s3 = n3;
      scr[i * sstride] = tri_div(tri_add(tri_mul(s0, b0), s1), tri_add(tri_mul(s2, b0), s3));
    }
    // Recurrence 2 (:38-56): y'_i = y_i - (a_i / b'_{i-1}) y'_{i-1}, into the output row
    const float y0 = yr[0];
    float c0 = 0.0f, c1 = 1.0f;
    for (int i = 0; i < m; i++) {
      float l0 = 0.0f, l1 = 1.0f;
      if (0 < i) {
        l0 = yr[i];
        l1 = tri_sub(0.0f, tri_div(ar[i], scr[(i - 1) * sstride]));
      }
      const float n0 = tri_add(l0, tri_mul(l1, c0));
      const float n1 = tri_mul(c1, l1);
      c0 = n0;
      c1 = n1;
      o[i] = tri_add(c0, tri_mul(c1, y0));
    }
    // Recurrence 3 (:61-79): backward, over the reversed index
    const float yn = tri_div(o[m - 1], scr[(int64_t)(m - 1) * sstride]);
    c0 = 0.0f;
    c1 = 1.0f;
    for (int k = 0; k < m; k++) {
      const int i = m - k - 1;
      float l0 = 0.0f, l1 = 1.0f;
      if (0 < k) {
        const float bi = scr[i * sstride];
        l0 = tri_div(o[i], bi);
        l1 = tri_sub(0.0f, tri_div(cr[i], bi));
      }
      const float n0 = tri_add(l0, tri_mul(l1, c0));
      const float n1 = tri_mul(c1, l1);
      c0 = n0;
      c1 = n1;
      o[i] = tri_add(c0, tri_mul(c1, yn));
    }
  }
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------------------
// Whole-row kernel: a warp holds `tile` systems' rows of all four inputs in shared
// memory, solves them in place, a lane per system, and stores the solutions from
// there.  Rows come and go as one contiguous block per array (bulk copies), so the
// copies cost the warp nothing, and nothing of the input is read twice.
//
// What bounds it: shared memory holds about 120 systems of 115 elements per SM, so
// a batch runs in rounds, each a copy in (HBM) and a chain of 115 elements: at 43
// cycles of dependent operations per element forward and 9 backward (near_rcp; 78
// and 9 with __frcp_rn), 67 and 18 measured.  57600 x 115, FORM 0 34 us and FORM 1
// 49, where the copies alone take 22.6; 40000 x 100 17 and 27; 100 x 115, a
// round's latency, 8.3 and 12.4 with the launch.  Kernels that streamed windows of
// rows through shared memory with the intermediates in tensor memory took 40, 68,
// 37, 64, 24.7 and 55: their copies were of rows of 8 or 20 floats, and at eight
// warps per SM each element's chain stood in the open.
// ---------------------------------------------------------------------------
constexpr int kTriRowWin = 8;  // elements per register window

// Elements k .. k + VW - 1 of a shared-memory row, to and from registers k .. of
// a window.
template <int VW>
__device__ __forceinline__ void tri_row_load(const float* p, int k, float (&v)[kTriRowWin]) {
  if constexpr (VW == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p + k);
    v[k] = t.x;
    v[k + 1] = t.y;
    v[k + 2] = t.z;
    v[k + 3] = t.w;
  } else if constexpr (VW == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p + k);
    v[k] = t.x;
    v[k + 1] = t.y;
  } else {
    v[k] = p[k];
  }
}
template <int VW>
__device__ __forceinline__ void tri_row_store(float* p, int k, const float (&v)[kTriRowWin]) {
  if constexpr (VW == 4) *reinterpret_cast<float4*>(p + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
  else if constexpr (VW == 2) *reinterpret_cast<float2*>(p + k) = make_float2(v[k], v[k + 1]);
  else p[k] = v[k];
}

// Forward state of one system.  FORM 0: cp, yp.  FORM 1: the 4-tuple scan s,
// b_0, c_{i-1}, the linear scan (c0, c1), y_0, b'_{i-1} with its reciprocal, and
// the last quotient y'_{m-1} / b'_{m-1}, which starts the backward fold.
struct TriRow {
  float cp = 0.0f, yp = 0.0f;
  float s0 = 1.0f, s1 = 0.0f, s2 = 0.0f, s3 = 1.0f, b0 = 0.0f, cprev = 0.0f;
  float y0 = 0.0f, c0 = 0.0f, c1 = 1.0f, bp = 1.0f, rb = 1.0f, yn = 0.0f;
};

// Element i of a forward pass, whatever the values: the two intermediates that
// the backward pass folds replace c_i and y_i.
template <int FORM>
__device__ __forceinline__ void tri_row_element(TriRow& f, int i, int m, float ai, float bi, float& ci, float& yi) {
  if constexpr (FORM == 0) {
    // cp_i = c_i / (b_i - a_i cp_{i-1}), yp_i = (y_i - a_i yp_{i-1}) / (...)  (:82-91)
    if (i == 0) {
      f.cp = tri_div(ci, bi);
      f.yp = tri_div(yi, bi);
    } else {
      const float nf = tri_rcp(tri_sub(bi, tri_mul(ai, f.cp)));
      f.cp = tri_mul(ci, nf);
      f.yp = tri_mul(tri_sub(yi, tri_mul(ai, f.yp)), nf);
    }
    ci = f.cp;
    yi = f.yp;
  } else {
    // recurrence 1 (:9-33): b'_i from the 4-tuple scan of (b_i, -a_i c_{i-1}, 1, 0)
    float m0 = 1.0f, m1 = 0.0f, m2 = 0.0f, m3 = 1.0f;
    if (i == 0) {
      f.b0 = bi;
      f.y0 = yi;
    } else {
      m0 = bi;
      m1 = tri_sub(0.0f, tri_mul(ai, f.cprev));
      m2 = 1.0f;
      m3 = 0.0f;
    }
    f.cprev = ci;
    const float value = tri_rcp(tri_mul(f.s0, m0));
    const float n0 = tri_mul(tri_add(tri_mul(m0, f.s0), tri_mul(m1, f.s2)), value);
    const float n1 = tri_mul(tri_add(tri_mul(m0, f.s1), tri_mul(m1, f.s3)), value);
    const float n2 = tri_mul(tri_add(tri_mul(m2, f.s0), tri_mul(m3, f.s2)), value);
    const float n3 = tri_mul(tri_add(tri_mul(m2, f.s1), tri_mul(m3, f.s3)), value);
    f.s0 = n0;
    f.s1 = n1;
    f.s2 = n2;
    f.s3 = n3;
    const float bp = tri_div(tri_add(tri_mul(f.s0, f.b0), f.s1), tri_add(tri_mul(f.s2, f.b0), f.s3));  // b'_i
    // recurrence 2 (:38-56): y'_i from the scan of (y_i, -a_i / b'_{i-1})
    float l0 = 0.0f, l1 = 1.0f;
    if (i > 0) {
      l0 = yi;
      l1 = tri_sub(0.0f, tri_div(ai, f.bp));
    }
    const float e0 = tri_add(l0, tri_mul(l1, f.c0));
    f.c1 = tri_mul(f.c1, l1);
    f.c0 = e0;
    const float yp = tri_add(f.c0, tri_mul(f.c1, f.y0));  // y'_i
    f.bp = bp;
    f.rb = tri_rcp(bp);
    // recurrence 3's elements (:61-79), the last one's first component its start
    const float q = tri_div(yp, bp);
    if (i < m - 1) {
      yi = q;
      ci = tri_sub(0.0f, tri_div(ci, bp));
    } else {
      f.yn = q;
    }
  }
}

// The same for i > 0 with near_rcp and near_div, exact while `in` holds.
// FORM 1: c_i is not wanted at i == m - 1, and f.yn is y_i's new value there.  y' is
// left in yp, and in ymin the least but zeros, which `in` does not see from below.
template <int FORM>
__device__ __forceinline__ void tri_row_step(TriRow& f, RangeCheck& in, float a, float b, float& c, float& y,
                                             float& yp, float& ymin) {
  if constexpr (FORM == 0) {
    const float d = tri_sub(b, tri_mul(a, f.cp));
    in.divisor(d);
    const float nf = near_rcp(d);
    c = f.cp = tri_mul(c, nf);
    y = f.yp = tri_mul(tri_sub(y, tri_mul(a, f.yp)), nf);
  } else {
    const float m1 = tri_sub(0.0f, tri_mul(a, f.cprev));
    const float p = tri_mul(f.s0, b);
    const float value = near_rcp(p);
    const float n0 = tri_mul(tri_add(p, tri_mul(m1, f.s2)), value);
    const float n1 = tri_mul(tri_add(tri_mul(b, f.s1), tri_mul(m1, f.s3)), value);
    const float n2 = tri_mul(f.s0, value);  // s0 + 0 * s2 is s0: p is in range, so s0 is not zero and s2 finite
    const float n3 = tri_mul(tri_add(f.s1, tri_mul(0.0f, f.s3)), value);
    f.s0 = n0;
    f.s1 = n1;
    f.s2 = n2;
    f.s3 = n3;
    const float num = tri_add(tri_mul(n0, f.b0), n1), den = tri_add(tri_mul(n2, f.b0), n3);
    const float bp = near_div(num, den, near_rcp(den));
    const float rb = near_rcp(bp);
    const float l1 = tri_sub(0.0f, near_div(a, f.bp, f.rb));
    f.c0 = tri_add(y, tri_mul(l1, f.c0));
    f.c1 = tri_mul(f.c1, l1);
    yp = tri_add(f.c0, tri_mul(f.c1, f.y0));
    in.divisor(p);
    in.large(num);  // infinite where m1 s2 or m1 s3 overflows: bp is then too, not the NaN that near_div makes of it
    in.divisor(den);
    in.divisor(bp);
    in.dividend(a);
    in.dividend(c);
    in.large(yp);
    ymin = fminf(ymin, yp == 0.0f ? 1.0f : fabsf(yp));
    f.cprev = c;
    f.bp = bp;
    f.rb = rb;
    y = yp == 0.0f ? tri_mul(yp, rb) : near_div(yp, bp, rb);
    c = tri_sub(0.0f, near_div(c, bp, rb));
  }
}

template <int FORM>
__device__ __forceinline__ bool tri_row_ok(const RangeCheck& in) {
  return FORM == 0 ? in.reciprocals_ok() : in.ok();
}

// The forward pass for any values, an element at a time: by the fast divisions where
// they hold for it, by exact ones where not; returns yp or yn, which the backward fold
// starts from.  A batch waits for a tile that comes here, and in most rows that do a
// pivot or two is out of range: with one singular row 57600 x 115 take 67 us (FORM 1)
// and 40 (FORM 0), by exact division throughout 74 and 42, without it 49 and 36.  Out of
// line: in line ordinary systems of some lengths take 1 to 3 % longer (50000 x 50 21.5
// us against 20.7).
template <int FORM>
static __device__ __noinline__ float tri_row_again(int m, const float* pa, const float* pb, float* pc, float* py) {
  TriRow f;
#pragma unroll 1
  for (int i = 0; i < m; i++) {
    const float a = pa[i], b = pb[i];
    float c = pc[i], y = py[i];
    RangeCheck in;
    if constexpr (FORM == 1) {
      in.divisor(f.bp);  // this element divides by it,
      in.large(f.s2);    // and takes s2 to be finite
    }
    bool fast = i > 0 && tri_row_ok<FORM>(in);
    if (fast) {
      TriRow g = f;
      float cg = FORM == 1 && i == m - 1 ? 1.0f : c, yg = y, yp = 0.0f, ymin = 1.0f;
      tri_row_step<FORM>(g, in, a, b, cg, yg, yp, ymin);
      fast = tri_row_ok<FORM>(in);
      if (fast) {
        f = g;
        c = cg;
        if (ymin <= 0x1p-80f) yg = tri_div(yp, g.bp);
        if (FORM == 1 && i == m - 1) f.yn = yg;
        y = yg;
      }
    }
    if (!fast) tri_row_element<FORM>(f, i, m, a, b, c, y);
    pc[i] = c;
    py[i] = y;
  }
  return FORM == 0 ? f.yp : f.yn;
}

// y'/b' of elements first - 1 (y, b) and first .. first + n - 1 but a row's first, by
// exact division.  Out of line, for rows in which y' fade out.
static __device__ __noinline__ void tri_row_quotients(float* py, int first, int n, float y, float b, float4 y0, float4 y4,
                                                      float4 b0, float4 b4) {
  const float ys[kTriRowWin] = {y0.x, y0.y, y0.z, y0.w, y4.x, y4.y, y4.z, y4.w};
  const float bs[kTriRowWin] = {b0.x, b0.y, b0.z, b0.w, b4.x, b4.y, b4.z, b4.w};
  if (first > 0) py[first - 1] = tri_div(y, b);
#pragma unroll
  for (int k = 0; k < kTriRowWin; k++)
    if (k < n && first + k > 0) py[first + k] = tri_div(ys[k], bs[k]);
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void bulk_s2g(void* dst, const void* src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}

// Row stride of the staged rows and the width of their accesses: odd m reads
// element by element and even m in pairs from rows as they lie in memory (a
// stride of an odd number of accesses: no bank conflicts); for m % 4 == 0 rows
// are read in fours, padded to an odd number of them.
__host__ __device__ __forceinline__ int tri_row_vw(int64_t m) { return m % 4 == 0 ? 4 : m % 2 == 0 ? 2 : 1; }
__host__ __device__ __forceinline__ int64_t tri_row_ld(int64_t m) { return m % 4 == 0 && (m / 4) % 2 == 0 ? m + 4 : m; }
__host__ __device__ __forceinline__ int64_t tri_row_smem(int64_t m, int sys) {
  return 16 + 16 * sys * tri_row_ld(m) + 4 * kTriRowWin;  // windows are read past a row's end
}

// bulk_in, bulk_out: the four inputs, the output start on 16-byte boundaries.
template <int FORM, int VW>
__global__ void __launch_bounds__(32) lvc_tridag_row_kernel(int64_t rows, int m, int tile, const float* __restrict__ a,
                                                            const float* __restrict__ b, const float* __restrict__ c,
                                                            const float* __restrict__ y, float* __restrict__ out,
                                                            bool bulk_in, bool bulk_out) {
  extern __shared__ __align__(16) unsigned char tri_raw[];
  uint64_t* const bar = reinterpret_cast<uint64_t*>(tri_raw);
  float* const S = reinterpret_cast<float*>(tri_raw + 16);  // [a, b, c, y][tile][ld]
  const int lane = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * tile;
  const int nr = (int)(rows - r0 < tile ? rows - r0 : tile);
  const int ld = (int)tri_row_ld(m), n = nr * m, A = tile * ld;
  const auto src = [&](int q) { return (q == 0 ? a : q == 1 ? b : q == 2 ? c : y) + r0 * m; };
  if (bulk_in && ld == m) {
    if (lane == 0) {
      mbar_init(bar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      mbar_expect_tx(bar, 16u * (unsigned)(n & ~3));
      if (n >= 4)
        for (int q = 0; q < 4; q++) bulk_g2s(S + q * A, src(q), 4u * (unsigned)(n & ~3), bar);
    }
    __syncwarp();
    if (lane < 4)  // what is left of the last system's row
      for (int e = n & ~3; e < n; e++) S[lane * A + e] = src(lane)[e];
    if (!mbar_wait(bar, 0)) {
      if (lane == 0) atomicExch(&lvc_tridag_err, 1);
      mbar_wait(bar, 0);  // for what is still in flight, once more with a limit
    }
  } else if (bulk_in) {  // padded rows: a bulk copy each would take the copy engine 54 cycles
    const int m4 = m / 4;
#pragma unroll 4
    for (int e = lane; e < nr * m4; e += 32) {
      const int row = e / m4, to = row * ld + 4 * (e - row * m4);
#pragma unroll
      for (int q = 0; q < 4; q++) cp_async16(S + q * A + to, src(q) + 4 * e);
    }
    cp_async_commit();
    cp_async_wait<0>();
  } else {  // off the 16-byte grid: four bytes at a time, asynchronous too (57600 x 115: 54 and 59
            // us, through registers 96 and 165)
#pragma unroll 4
    for (int e = lane; e < n; e += 32) {
      const int to = ld == m ? e : e / m * ld + e % m;
#pragma unroll
      for (int q = 0; q < 4; q++) cp_async4(S + q * A + to, src(q) + e);
    }
    cp_async_commit();
    cp_async_wait<0>();
  }
  __syncwarp();
  const bool act = lane < nr;
  const int sys = act ? lane : 0;
  float* const pa = S + sys * ld;
  const float* const pb = pa + A;
  float* const pc = pa + 2 * A;
  float* const py = pa + 3 * A;

  // forward: the intermediates replace c and y.  The registers hold a window of
  // eight elements; as soon as one is done it is stored and its register
  // refilled from the next window, so a load is eight elements ahead of its use
  // and no load or store waits between two elements of the chain.
  TriRow f;
  RangeCheck in;
  if (act) {
    float ymin = 1.0f;
    float va[kTriRowWin], vb[kTriRowWin], vc[kTriRowWin], vy[kTriRowWin];
#pragma unroll
    for (int k = 0; k < kTriRowWin; k += VW) {
      tri_row_load<VW>(pa, k, va);
      tri_row_load<VW>(pb, k, vb);
      tri_row_load<VW>(pc, k, vc);
      tri_row_load<VW>(py, k, vy);
    }
    tri_row_element<FORM>(f, 0, m, va[0], vb[0], vc[0], vy[0]);
    if constexpr (FORM == 1) in.divisor(f.bp);
    // element 0 is done: step(k) of window 0 starts at 1
    const int full = m / kTriRowWin;
    const float *qa = pa, *qb = pb;
    float *qc = pc, *qy = py;
    // FORM 1: quotients y'/b' whose y' have faded out of near_div's range are off the
    // chain and taken again, a window's when the last element of it has been issued
    // (which goes with the next window: its y' is not awaited).  57600 x 115 with y of
    // 1e-30: 76 us, against 182 where such tiles take the exact pass below -- as they do
    // with m = 4 k + 2, where the test makes ordinary systems 2 to 3 % slower (50000 x 50
    // 20.8 and 21.5 us; otherwise they take the same time).
    constexpr bool kLate = FORM == 1 && VW != 2;
    float yq[kTriRowWin] = {}, bq[kTriRowWin] = {}, ylast = 0.0f, blast = 1.0f;
    auto small_quotients = [&](int first, int n) {  // elements first - 1 .. first + n - 1
      tri_row_quotients(py, first, n, ylast, blast, make_float4(yq[0], yq[1], yq[2], yq[3]),
                        make_float4(yq[4], yq[5], yq[6], yq[7]), make_float4(bq[0], bq[1], bq[2], bq[3]),
                        make_float4(bq[4], bq[5], bq[6], bq[7]));
    };
    for (int w = 0; w < full; w++) {
      float seen = 1.0f;
#pragma unroll
      for (int k = 0; k < kTriRowWin; k++) {
        if (kLate && k == kTriRowWin - 1) {
          seen = ymin;
          ymin = 1.0f;
        }
        if (k > 0 || w > 0) tri_row_step<FORM>(f, in, va[k], vb[k], vc[k], vy[k], yq[k], ymin);
        bq[k] = f.bp;
        if (k % VW == VW - 1) {
          tri_row_store<VW>(qc, k - (VW - 1), vc);
          tri_row_store<VW>(qy, k - (VW - 1), vy);
          tri_row_load<VW>(qa + kTriRowWin, k - (VW - 1), va);
          tri_row_load<VW>(qb + kTriRowWin, k - (VW - 1), vb);
          tri_row_load<VW>(qc + kTriRowWin, k - (VW - 1), vc);
          tri_row_load<VW>(qy + kTriRowWin, k - (VW - 1), vy);
        }
      }
      if (kLate && seen <= 0x1p-80f) small_quotients(w * kTriRowWin, kTriRowWin - 1);
      ylast = yq[kTriRowWin - 1];
      blast = bq[kTriRowWin - 1];
      qa += kTriRowWin;
      qb += kTriRowWin;
      qc += kTriRowWin;
      qy += kTriRowWin;
    }
#pragma unroll
    for (int k = 0; k < kTriRowWin; k++) {
      if (full * kTriRowWin + k < m) {
        if (FORM == 1 && full * kTriRowWin + k == m - 1) vc[k] = 1.0f;
        if (k > 0 || full > 0) tri_row_step<FORM>(f, in, va[k], vb[k], vc[k], vy[k], yq[k], ymin);
        bq[k] = f.bp;
        qc[k] = vc[k];
        qy[k] = vy[k];
      }
    }
    if (kLate && ymin <= 0x1p-80f) small_quotients(full * kTriRowWin, m - full * kTriRowWin);
    if (!kLate && ymin <= 0x1p-80f) in.divisor(0.0f);  // out of range
    if constexpr (FORM == 1) {
      if (m > 1) f.yn = py[m - 1];
    }
  }
  float start = FORM == 0 ? f.yp : f.yn;  // of the backward fold
  if (__any_sync(0xffffffffu, !tri_row_ok<FORM>(in))) {  // again, c and y copied in once more
    for (int q = 2; q < 4; q++)
#pragma unroll 8
      for (int e = lane; e < n; e += 32) S[q * A + (ld == m ? e : e / m * ld + e % m)] = src(q)[e];
    __syncwarp();
    if constexpr (FORM == 1 && VW == 4) {
      // exact division throughout: beside the other, ordinary systems take up to 3 %
      // longer here (8000 x 200 23.7 us against 23.0)
      f = TriRow();
      if (act) {
#pragma unroll 1
        for (int i = 0; i < m; i++) tri_row_element<FORM>(f, i, m, pa[i], pb[i], pc[i], py[i]);
      }
      start = f.yn;
    } else {
      if (act) start = tri_row_again<FORM>(m, pa, pb, pc, py);
    }
  }

  // backward, the solution in place of y, the same way from the end
  float x = start, c0 = 0.0f, c1 = 1.0f;
  auto back = [&](float p, float q) {  // p, q: the intermediates in c's and y's places
    if constexpr (FORM == 0) {
      x = tri_sub(q, tri_mul(p, x));  // x_i = yp_i - cp_i x_{i+1}  (:92-95)
      return x;
    } else {
      c0 = tri_add(q, tri_mul(p, c0));
      c1 = tri_mul(c1, p);
      return tri_add(c0, tri_mul(c1, start));
    }
  };
  if (act) {
    const int wb = (m - 1) / kTriRowWin;  // whole windows before m - 1
    // element m - 1 (FORM 1: the fold's start, l0 = 0, l1 = 1), then the others of its window
    float yl = start;
    if constexpr (FORM == 1) {
      c0 = tri_add(0.0f, tri_mul(1.0f, c0));
      yl = tri_add(c0, tri_mul(c1, start));
    }
    py[m - 1] = yl;
    for (int i = m - 2; i >= wb * kTriRowWin; i--) py[i] = back(pc[i], py[i]);
    if (wb > 0) {
      float vc[kTriRowWin], vy[kTriRowWin], vx[kTriRowWin];
      const float* qc = pc + (wb - 1) * kTriRowWin;
      float* qy = py + (wb - 1) * kTriRowWin;
#pragma unroll
      for (int k = 0; k < kTriRowWin; k += VW) {
        tri_row_load<VW>(qc, k, vc);
        tri_row_load<VW>(qy, k, vy);
      }
      for (int w = wb - 1; w >= 0; w--) {
        const int next = w > 0 ? -kTriRowWin : 0;  // the first window's registers are refilled from itself
#pragma unroll
        for (int k = kTriRowWin - 1; k >= 0; k--) {
          vx[k] = back(vc[k], vy[k]);
          if (k % VW == 0) {
            tri_row_load<VW>(qc + next, k, vc);
            tri_row_load<VW>(qy + next, k, vy);
            tri_row_store<VW>(qy, k, vx);
          }
        }
        qc -= kTriRowWin;
        qy -= kTriRowWin;
      }
    }
  }
  __syncwarp();

  float* const dst = out + r0 * m;
  const float* const sol = S + 3 * A;
  if (bulk_out && ld == m) {
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncwarp();
    if (lane == 0 && n >= 4) bulk_s2g(dst, sol, 4u * (unsigned)(n & ~3));
    if (lane < (n & 3)) dst[(n & ~3) + lane] = sol[(n & ~3) + lane];
    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
    asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
  } else if (bulk_out) {
    const int m4 = m / 4;
#pragma unroll 4
    for (int e = lane; e < nr * m4; e += 32) {
      const int row = e / m4;
      __stcs(reinterpret_cast<float4*>(dst) + e, *reinterpret_cast<const float4*>(sol + row * ld + 4 * (e - row * m4)));
    }
  } else {
    for (int e = lane; e < n; e += 32) dst[e] = sol[ld == m ? e : e / m * ld + e % m];
  }
}

}  // namespace lvc
