// Tall paired kernel (f64): the paired kernel's arithmetic on twice the grid per
// CTA, so that a grid takes half the CTAs of a cluster, or none.
//
// The paired kernel keeps two grid-sized buffers on chip, the grid and the step's
// X pivots, which the implicit-Y right-hand side then replaces.  Here there is one:
//   * the pivots sit in tensor memory -- 256 KB per SM, read back by the thread
//     that stored them (tcgen05.st / .ld), so they are laid out in HBM as the
//     threads load them ([row group][column pair][row]) and come in, in four
//     batches, while the previous step's Y sweep runs;
//   * the right-hand side replaces the grid in place.  A row of the X sweep needs
//     the rows above and below as they were: inside a warp's 32 rows the lanes read
//     them before any writes; across row groups they read copies of the groups'
//     first and last rows, kept when the rows were stored.
// The X sweep takes the CTA's rows in two rounds of the paired kernel's three
// passes (each row is a system of its own), the Y sweep two units per warp.
//
// A step of a CTA's 16384 cells takes 12.0 us alone, 14.1 us in a cluster of two
// and 15.5 us of four, against 5.6 us for 8192 cells in the paired kernel and 7.2,
// 7.4 and 7.7 us in its clusters of two, four and eight: for a grid that the
// paired kernel holds in one CTA it is 7 % slower per cell, and from there on it
// wins what the exchanges and the clusters' packing cost (15 clusters of eight fit
// on the chip, 32 of four).  At 64 strikes of 256 x 256 30.7 us a step against
// 37.2, at 400 of 128 x 128 35.3 against 41.4, of 128 x 256 82.4 against 91.5.
// FP64 arithmetic of dependent chains is the bound, as in the paired kernel.
// Loading the first batch of pivots during the X sweep instead of the Y sweep: 12.3,
// 14.3 and 15.2 us.  Four warps on half the rows, two CTAs to an SM: 23.5 us a step
// at 400 strikes of 128 x 64 against the paired kernel's 16.5.
#pragma once

#include "lvc_pair.cuh"

namespace lvc {

constexpr int kTallRounds = 2, kTallWarps = 8;

struct TallLayout {
  int LD, Ycs, CHx, RG, G, CG, CHy;
  int bar, barF, barB, taddr, A, top, bot, w0, w1, w2, gx, ex, tab0, tab1, tabh, xf, xb, yf, yb, inF, totF, inB, totB,
      zin, xin, total;
};

// A CTA holding Ycs = 2 * 8 / (X / 32) row groups of 32 rows of a grid of X = 64, 128
// or 256 columns that C CTAs share; byte offsets.
LVC_HD TallLayout tall_layout(int X, int Ycs, int C) {
  constexpr int NW = kTallWarps;
  TallLayout L;
  auto up = [](int n) { return (n + 15) / 16 * 16; };
  auto line = [](int n) { return (n + 127) / 128 * 128; };
  L.LD = pair_ld(X);
  L.Ycs = Ycs;
  L.CHx = X / kLineK;
  L.RG = X >= 64 ? NW / (X / 32) : 0;  // row groups per round
  L.G = Ycs / 32;
  L.CG = X / 64;       // column groups of a Y unit
  L.CHy = Ycs / kLineK;
  int o = 0;
  L.bar = o; o += 8;    // bulk copy of the step's table
  L.barF = o; o += 8;   // cluster: forward chunk maps of the lower ranks have landed
  L.barB = o; o += 8;   // cluster: backward chunk maps of the higher ranks have landed
  L.taddr = o; o += 8;  // tensor memory
  o = line(o);
  L.A = o; o += up((Ycs + 2) * L.LD * 8);  // rows -1 .. Ycs
  // copies of each row group's first and last rows, in the banks of the rows they
  // stand for (one lane of a warp reads them among 31 rows of A)
  o = line(o);
  L.bot = o; o += L.G * X * 8;
  L.top = o + 16; o += 16 + L.G * X * 8;
  o = up(o);
  L.w0 = o; o += up(X * 8);
  L.w1 = o; o += up(X * 8);
  L.w2 = o; o += up(X * 8);
  L.gx = o; o += up(3 * Ycs * 8);  // [3][Ycs] row constants, planar
  L.ex = o; o += up(Ycs * 8);      // [Ycs] e_j of the step, planar
  L.tab0 = o; o += up(8 * Ycs * 8);
  L.tab1 = o; o += up(8 * Ycs * 8);
  L.tabh = o; o += 2 * 64;
  L.xf = o; o += up(NW * 64 * 8);  // [warp][lane] (a, b) of the warps' forward chunk maps
  L.xb = o; o += up(NW * 64 * 8);
  L.yf = o; o += up(L.CG * L.CHy * 64 * 8);
  L.yb = o; o += up(L.CG * L.CHy * 64 * 8);
  const int Cc = C > 1 ? C : 0;
  L.inF = o; o += up(Cc * X * 8);
  L.totF = o; o += up(Cc * 8);
  L.inB = o; o += up(Cc * X * 8);
  L.totB = o; o += up(Cc * 8);
  L.zin = o; o += Cc ? up(X * 8) : 0;
  L.xin = o; o += Cc ? up(X * 8) : 0;
  L.total = o;
  return L;
}

// ---- tensor memory: one lane of a warp's quarter per thread ----
// All of these are .sync.aligned: the lanes of a warp arrive together.  After a branch
// or a loop that lanes leave differently a barrier sees to that.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, int ncols) {  // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(dst)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {  // whole warp
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, int ncols) {  // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// Two pairs of doubles (8 columns) to and from this thread's lane (whole warp).
__device__ __forceinline__ void tmem_st2(uint32_t t, double2 a, double2 b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(t),
               "r"(__double2loint(a.x)), "r"(__double2hiint(a.x)), "r"(__double2loint(a.y)), "r"(__double2hiint(a.y)),
               "r"(__double2loint(b.x)), "r"(__double2hiint(b.x)), "r"(__double2loint(b.y)), "r"(__double2hiint(b.y))
               : "memory");
}
// both units' two pairs, and the wait for them, in one statement: no use of the
// values can be scheduled before they have arrived
__device__ __forceinline__ void tmem_ld2x2(uint32_t t0, uint32_t t1, double2 (&a)[2], double2 (&b)[2]) {
  int r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(t0), "r"(t1)
      : "memory");
#pragma unroll
  for (int k = 0; k < 2; k++) {
    a[k] = make_double2(__hiloint2double(r[4 * k + 1], r[4 * k]), __hiloint2double(r[4 * k + 3], r[4 * k + 2]));
    b[k] = make_double2(__hiloint2double(r[8 + 4 * k + 1], r[8 + 4 * k]),
                        __hiloint2double(r[8 + 4 * k + 3], r[8 + 4 * k + 2]));
  }
}

__global__ void __launch_bounds__(32 * kTallWarps, 1) lvc_line_tall_kernel(RollbackArgs<double, double> args) {
  constexpr int K = kLineK, R = kTallRounds;
  constexpr int NW = kTallWarps, NT = 32 * NW;
  constexpr int kCols = NW / 4 * R * 4 * K;  // tensor-memory columns: 2 units x K doubles per round and thread
  static_assert(kCols == 256, "an allocation is a power of two, half the SM's");
  using V = P2<double>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int C = args.C;
  const bool clustered = C > 1;
  int rank = 0;
  if (clustered) rank = (int)cg::this_cluster().block_rank();
  const int cid = blockIdx.x / C, ncl = gridDim.x / C;
  unsigned sc = 0, phase = 0;
  unsigned phF = 0, phB = 0;  // parities of the cluster barriers (one completion per use)
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
  uint64_t* barF = bar + 1;
  uint64_t* barB = bar + 2;
  uint32_t* s_taddr = reinterpret_cast<uint32_t*>(smem + 24);
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_init(barF, 1);
    mbar_init(barB, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncwarp();
  if (warp == 0) {
    tmem_alloc(s_taddr, kCols);
    tmem_relinquish();
  }
  tmem_fence_before_sync();
  __syncthreads();
  tmem_fence_after_sync();
  // this thread's lane, its warp's columns: [round][unit][K doubles]
  const uint32_t tmem = *s_taddr + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(warp / 4 * R * 4 * K);

  for (int it = cid; it < args.n_items; it += ncl) {
    const Item item = args.items[it];
    const CalibDev c = args.calibs[item.calib];
    const int X = c.numX, Y = c.numY, T = c.numT;
    const int Ycs = c.Ycs;
    const int r0 = rank * Ycs;
    const TallLayout Ls = tall_layout(X, Ycs, C);
    // uniform over the cluster (every CTA of a cluster sees the same item)
    if (c.kind != kKindTall || c.C != C || c.ld != Ls.LD || Ls.total > args.smem_elems * 8 || X % 64 || X > 32 * NW ||
        Ls.RG * (X / 32) != NW || Ycs != R * Ls.RG * 32 || Ycs * C != Y) {
      if (tid == 0) atomicExch(args.err, 5);
      continue;
    }
    const int LD = Ls.LD;
    double* A = reinterpret_cast<double*>(smem + Ls.A);  // row r of the block at A + (r + 1) * LD
    double* sTop = reinterpret_cast<double*>(smem + Ls.top);  // [G][X]: each row group's first row
    double* sBot = reinterpret_cast<double*>(smem + Ls.bot);  // and its last
    double* sW0 = reinterpret_cast<double*>(smem + Ls.w0);
    double* sW1 = reinterpret_cast<double*>(smem + Ls.w1);
    double* sW2 = reinterpret_cast<double*>(smem + Ls.w2);
    double* sGx = reinterpret_cast<double*>(smem + Ls.gx);
    double* sE = reinterpret_cast<double*>(smem + Ls.ex);
    double* const sT0 = reinterpret_cast<double*>(smem + Ls.tab0);
    double* const sT1 = reinterpret_cast<double*>(smem + Ls.tab1);
    double* xf = reinterpret_cast<double*>(smem + Ls.xf);
    double* xb = reinterpret_cast<double*>(smem + Ls.xb);
    double* yf = reinterpret_cast<double*>(smem + Ls.yf);
    double* yb = reinterpret_cast<double*>(smem + Ls.yb);
    double* inF = reinterpret_cast<double*>(smem + Ls.inF);
    double* totF = reinterpret_cast<double*>(smem + Ls.totF);
    double* inB = reinterpret_cast<double*>(smem + Ls.inB);
    double* totB = reinterpret_cast<double*>(smem + Ls.totB);
    double* const sTh = reinterpret_cast<double*>(smem + Ls.tabh);
    double* s_zin = reinterpret_cast<double*>(smem + Ls.zin);
    double* s_xin = reinterpret_cast<double*>(smem + Ls.xin);
    const double* tabc = args.tabs + c.tab;
    const TabLayout Lt = tab_layout(X, Y, T, c.Xp, kKindLine);
    const double strike = 0.001 * (double)item.strike;  // strikes (:247)
    const int steps = T > 1 ? T - 1 : 0;
    const double* piv = args.piv + c.piv;
    // cluster pushes as in the paired kernel
    const bool has_prev = clustered && rank > 0, has_next = clustered && rank < C - 1;
    const unsigned fold_bytes_F = (unsigned)(rank * (X + 1) * 8);
    const unsigned fold_bytes_B = clustered ? (unsigned)((C - 1 - rank) * (X + 1) * 8) : 0u;

    if (clustered) cg::this_cluster().sync(); else __syncthreads();
    // setPayoff (:46-47) on the block and the halo rows (zero at the global
    // boundary and in the two columns beyond X): every row of the grid is the same
    for (int e = tid; e < (Ycs + 2) * LD; e += NT) {
      const int r = e / LD, i = e - r * LD;
      const bool boundary = (r == 0 && rank == 0) || (r == Ycs + 1 && rank == C - 1);
      A[e] = (i < X && !boundary) ? fmax(tabc[Lt.x + i] - strike, 0.0) : 0.0;
    }
    for (int e = tid; e < Ls.G * X; e += NT) sTop[e] = sBot[e] = fmax(tabc[Lt.x + e % X] - strike, 0.0);
    for (int e = tid; e < 3 * X; e += NT) {
      const int k = e / X, i = e - k * X;
      (k == 0 ? sW0 : k == 1 ? sW1 : sW2)[i] = tabc[Lt.wcol + k * (int64_t)((X + 1) & ~1) + i];
    }
    for (int e = tid; e < 3 * Ycs; e += NT) {
      const int k = e / Ycs, j = e - k * Ycs;
      sGx[e] = tabc[Lt.rowc + 4LL * (r0 + j) + k];
    }
    if (steps == 0) {
      if (tid == 0 && c.yindex >= r0 && c.yindex < r0 + Ycs)
        args.out[c.out + item.strike] = fmax(tabc[Lt.x + c.xindex] - strike, 0.0);
      continue;
    }
    const unsigned tab_bytes = (unsigned)(Ycs * 64);
    const unsigned tabh_bytes = has_prev ? 64u : 0u;
    auto issue_copies = [&](int k, unsigned buf) {
      if (tid == 0) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        mbar_expect_tx(bar, tab_bytes + tabh_bytes);
        bulk_g2s(buf ? sT1 : sT0, tabc + Lt.stab + ((int64_t)k * Y + r0) * 8, tab_bytes, bar);
        if (has_prev) bulk_g2s(sTh + 8 * buf, tabc + Lt.stab + ((int64_t)k * Y + r0 - 1) * 8, 64, bar);
      }
    };
    issue_copies(steps - 1, sc & 1);

    // X units u = 2 * warp + q of a round: rows (round * RG + rg) * 32 + lane, columns
    // chx * 16 ..; a warp's two are neighbouring chunks of one row group
    const int WPG = Ls.CHx / 2;          // warps per row group
    const int rg = warp / WPG, wg0 = rg * WPG;
    const int ib0 = (2 * (warp - wg0)) * K;  // first column of unit 0; unit 1 starts K on
    // Y units 2 * warp + t: columns col0, col0 + 1, rows (chy0 + t) * 16 ..
    const int cgy = 2 * warp / Ls.CHy, chy0 = 2 * warp - cgy * Ls.CHy;
    const int col0 = cgy * 64 + 2 * lane;
    // output lane: the column and element holding myResult[myYindex, myXindex]
    int out_h = -1, out_m = 0;
    {
      const int jy = c.yindex - r0 - chy0 * K;
      if (c.xindex >= col0 && c.xindex < col0 + 2 && jy >= 0 && jy < 2 * K) {
        out_h = c.xindex - col0;
        out_m = jy;
      }
    }
    __syncthreads();  // after issue_copies and out_h (a __syncwarp at either place spills 24 bytes more)
    // Batch b of a step's pivots, unit b % 2 of round b / 2: loaded, and later stored.
    double2 pv[K / 2];
    double rb0[R];  // 1/b' of the column before unit 0's first, by round
    auto piv_load = [&](int k, int b) {
      const int j = r0 + ((b / 2) * Ls.RG + rg) * 32 + lane, i = ib0 + (b % 2) * K;
      const double* p = piv + tall_piv(X, Y, k, j, i);
#pragma unroll
      for (int t = 0; t < K / 2; t++) pv[t] = __ldcg(reinterpret_cast<const double2*>(p + 64 * t));
      if (b % 2 == 0) rb0[b / 2] = i > 0 ? p[-64 + 1] : 0.0;
    };
    auto piv_store = [&](int b) {
#pragma unroll
      for (int t = 0; t < K / 2; t += 2) tmem_st2(tmem + (uint32_t)(b * 2 * K + 4 * t), pv[t], pv[t + 1]);
    };
#pragma unroll
    for (int b = 0; b < 2 * R; b++) {
      piv_load(steps - 1, b);
      piv_store(b);
    }
    tmem_wait_st();

    bool timed_out = false;  // a bulk-copy wait of this item gave up
    for (int s = 0; s < steps; s++, sc++) {
      const int k = steps - 1 - s;
      if (!mbar_wait(bar, phase, timed_out ? kWaitPollsAfterTimeout : kWaitPolls)) {
        timed_out = true;
        atomicExch(args.err, 3);
      }
      phase ^= 1u;
      const double* tb = (sc & 1) ? sT1 : sT0;
      for (int j = tid; j < Ycs; j += NT) sE[j] = tb[j * 8 + kSlotE];
      __syncthreads();
      const double dt = tabc[Lt.dtinv + k];

#pragma unroll 1
      for (int rd = 0; rd < R; rd++) {
        const int g = rd * Ls.RG + rg;  // this warp's row group
        const int jl = g * 32 + lane;
        double* const Arow = A + (jl + 1) * LD;
        // the rows above and below: in A, or the neighbouring group's kept copy
        const double* const Aup = lane > 0 || g == 0 ? Arow - LD : sBot + (g - 1) * X;
        const double* const Adn = lane < 31 || g == Ls.G - 1 ? Arow + LD : sTop + (g + 1) * X;
        const double e = sE[jl], g0 = sGx[jl], g1 = sGx[Ycs + jl], g2 = sGx[2 * Ycs + jl];
        const uint32_t tm = tmem + (uint32_t)(rd * 4 * K);
        double z[2][K], PQ[2][K];
        double zl[2], Pl[2];
        // -------- pass 1: explicitX + explicitY, forward recurrence (chunk-local) --------
        {
          double Rl[2], rbp[2];
          double2 Rc[2];
#pragma unroll
          for (int q = 0; q < 2; q++) {
            const int ib = ib0 + q * K;
            Rl[q] = ib > 0 ? Arow[ib - 1] : 0.0;
            Rc[q] = V::ld(Arow + ib);
            zl[q] = 0;
            Pl[q] = 1;
          }
          rbp[0] = rd == 0 ? rb0[0] : rb0[1];
          {  // unit 0's last pivot
            double2 a[2], b[2];
            tmem_ld2x2(tm + 2 * K - 8, tm + 2 * K - 8, a, b);
            rbp[1] = a[1].y;
          }
#pragma unroll
          for (int p = 0; p < K / 2; p += 2) {
            double2 rb[2][2];  // [unit][pair]
            tmem_ld2x2(tm + 4 * p, tm + 2 * K + 4 * p, rb[0], rb[1]);
#pragma unroll
            for (int h = 0; h < 2; h++) {
#pragma unroll
              for (int q = 0; q < 2; q++) {
                const int i = ib0 + q * K + 2 * (p + h);
                const double2 Rn = V::ld(Arow + i + 2);  // columns i+2, i+3 (numX, numX+1 are zero)
                const double2 up = V::ld(Aup + i);
                const double2 dn = V::ld(Adn + i);
                const double2 w0 = V::ld(sW0 + i);
                const double2 w1 = V::ld(sW1 + i);
                const double2 w2 = V::ld(sW2 + i);
                {  // column i
                  const double v = g0 * up.x + g1 * Rc[q].x + g2 * dn.x;               // explicitY (:199)
                  const double sx = w0.x * Rl[q] + w1.x * Rc[q].x + w2.x * Rc[q].y;    // explicitX / (0.5 e)
                  const double u = e * sx + (dt * Rc[q].x + v);                        // :195-200
                  const double mult = (e * w0.x) * rbp[q];                             // -a_i / b'_{i-1}
                  zl[q] = u + mult * zl[q];
                  Pl[q] = mult * Pl[q];
                  z[q][2 * (p + h)] = zl[q];
                  PQ[q][2 * (p + h)] = Pl[q];
                }
                {  // column i + 1
                  const double v = g0 * up.y + g1 * Rc[q].y + g2 * dn.y;
                  const double sx = w0.y * Rc[q].x + w1.y * Rc[q].y + w2.y * Rn.x;
                  const double u = e * sx + (dt * Rc[q].y + v);
                  const double mult = (e * w0.y) * rb[q][h].x;
                  zl[q] = u + mult * zl[q];
                  Pl[q] = mult * Pl[q];
                  z[q][2 * (p + h) + 1] = zl[q];
                  PQ[q][2 * (p + h) + 1] = Pl[q];
                }
                rbp[q] = rb[q][h].y;
                Rl[q] = Rc[q].y;
                Rc[q] = Rn;
              }
            }
          }
          V::st(xf + (warp * 32 + lane) * 2, zl[1] + Pl[1] * zl[0], Pl[1] * Pl[0]);
        }
        __syncthreads();
        // -------- pass 2: forward fix-up, backward recurrence (chunk-local) --------
        double xl[2], Ql[2];
        {
          double zin[2];
          {
            double a = 0;
            for (int w = wg0; w < warp; w++) {
              const double2 f = V::ld(xf + (w * 32 + lane) * 2);
              a = f.x + f.y * a;
            }
            zin[0] = a;
            zin[1] = zl[0] + Pl[0] * a;
          }
#pragma unroll
          for (int q = 0; q < 2; q++) {
            xl[q] = 0;
            Ql[q] = 1;
          }
#pragma unroll
          for (int p = K / 2 - 2; p >= 0; p -= 2) {
            double2 rb[2][2];
            tmem_ld2x2(tm + 4 * p, tm + 2 * K + 4 * p, rb[0], rb[1]);
#pragma unroll
            for (int h = 1; h >= 0; h--) {
#pragma unroll
              for (int q = 0; q < 2; q++) {
                const int i = ib0 + q * K + 2 * (p + h), m = 2 * (p + h);
                const double2 w2 = V::ld(sW2 + i);
                {  // column i + 1
                  const double zz = z[q][m + 1] + PQ[q][m + 1] * zin[q];
                  const double aR = e * w2.y;
                  xl[q] = rb[q][h].y * (zz + aR * xl[q]);  // x_i = (z_i - c_i x_{i+1}) / b'_i
                  Ql[q] = (aR * rb[q][h].y) * Ql[q];
                  z[q][m + 1] = xl[q];
                  PQ[q][m + 1] = Ql[q];
                }
                {  // column i
                  const double zz = z[q][m] + PQ[q][m] * zin[q];
                  const double aR = e * w2.x;
                  xl[q] = rb[q][h].x * (zz + aR * xl[q]);
                  Ql[q] = (aR * rb[q][h].x) * Ql[q];
                  z[q][m] = xl[q];
                  PQ[q][m] = Ql[q];
                }
              }
            }
          }
          V::st(xb + (warp * 32 + lane) * 2, xl[0] + Ql[0] * xl[1], Ql[0] * Ql[1]);
        }
        __syncthreads();
        // -------- pass 3: backward fix-up; dtInv * u - 0.5 * explicitY (:205) in the grid's place --------
        {
          double xin[2];
          {
            double a = 0;
            for (int w = wg0 + WPG - 1; w > warp; w--) {
              const double2 f = V::ld(xb + (w * 32 + lane) * 2);
              a = f.x + f.y * a;
            }
            xin[1] = a;
            xin[0] = xl[1] + Ql[1] * a;
          }
#pragma unroll
          for (int p = 0; p < K / 2; p++) {
            double2 y2[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
              const int i = ib0 + q * K + 2 * p;
              const double2 up = V::ld(Aup + i), cu = V::ld(Arow + i), dn = V::ld(Adn + i);
              const double v0 = g0 * up.x + g1 * cu.x + g2 * dn.x, v1 = g0 * up.y + g1 * cu.y + g2 * dn.y;
              y2[q].x = dt * (z[q][2 * p] + PQ[q][2 * p] * xin[q]) - 0.5 * v0;
              y2[q].y = dt * (z[q][2 * p + 1] + PQ[q][2 * p + 1] * xin[q]) - 0.5 * v1;
            }
            __syncwarp();  // the rows' neighbours have read what is replaced
#pragma unroll
            for (int q = 0; q < 2; q++) V::st(Arow + ib0 + q * K + 2 * p, y2[q].x, y2[q].y);
          }
        }
      }
      __syncthreads();

      // -------- Y sweep: columns col0, col0 + 1; two chunks of 16 rows --------
      // the next step's pivots come in as its batches of tensor memory are used up
      const bool more = s + 1 < steps;
      if (more) piv_load(k - 1, 0);
      double y[2][2][K], zz[2][2];
#pragma unroll
      for (int t = 0; t < 2; t++) zz[t][0] = zz[t][1] = 0;
#pragma unroll
      for (int m = 0; m < K; m++) {
#pragma unroll
        for (int t = 0; t < 2; t++) {
          const int j = (chy0 + t) * K + m;
          const double2 rhs = V::ld(A + (j + 1) * LD + col0);
          const double my = tb[j * 8 + kSlotMY];
          zz[t][0] = rhs.x + my * zz[t][0];  // forward recurrence
          zz[t][1] = rhs.y + my * zz[t][1];
          y[t][0][m] = zz[t][0];
          y[t][1][m] = zz[t][1];
        }
      }
#pragma unroll
      for (int t = 0; t < 2; t++) V::st(yf + (2 * warp + t) * 64 + 2 * lane, zz[t][0], zz[t][1]);
      if (more) {
        piv_store(0);
        piv_load(k - 1, 1);
        issue_copies(k - 1, (sc + 1) & 1);  // into the table that the step before has read
      }
      __syncthreads();
      if (clustered) {
        for (int col = tid; col < X; col += NT) {
          const int cg2 = col >> 6, w = col & 63;
          double a = 0;
          for (int c2 = 0; c2 < Ls.CHy; c2++)
            a = yf[(cg2 * Ls.CHy + c2) * 64 + w] + tb[(c2 * K + K - 1) * 8 + kSlotCP] * a;
          for (int h = rank + 1; h < C; h++)
            st_async(cluster_addr(inF + rank * X + col, h), a, cluster_addr(barF, h));
        }
        if (tid == 0) {
          double b = 1;
          for (int c2 = 0; c2 < Ls.CHy; c2++) b = tb[(c2 * K + K - 1) * 8 + kSlotCP] * b;
          for (int h = rank + 1; h < C; h++) st_async(cluster_addr(totF + rank, h), b, cluster_addr(barF, h));
          mbar_expect_tx(barF, fold_bytes_F);
        }
        if (!mbar_wait_cluster(barF, phF, timed_out ? kWaitPollsAfterTimeout : kWaitPolls)) {
          timed_out = true;
          atomicExch(args.err, 3);
        }
        phF ^= 1u;
        for (int col = tid; col < X; col += NT) {
          double zv = 0;
          for (int q = 0; q < rank; q++) zv = inF[q * X + col] + totF[q] * zv;
          s_zin[col] = zv;
        }
        __syncthreads();
      }
      {
        double zin[2][2], xx[2][2];
        zin[0][0] = zin[0][1] = 0;
        if (clustered) {
          const double2 t = V::ld(s_zin + col0);
          zin[0][0] = t.x;
          zin[0][1] = t.y;
        }
        for (int c2 = 0; c2 < chy0; c2++) {
          const double2 a = V::ld(yf + (cgy * Ls.CHy + c2) * 64 + 2 * lane);
          const double cp = tb[(c2 * K + K - 1) * 8 + kSlotCP];
          zin[0][0] = a.x + cp * zin[0][0];
          zin[0][1] = a.y + cp * zin[0][1];
        }
        {
          const double cp = tb[(chy0 * K + K - 1) * 8 + kSlotCP];
          zin[1][0] = zz[0][0] + cp * zin[0][0];
          zin[1][1] = zz[0][1] + cp * zin[0][1];
        }
#pragma unroll
        for (int t = 0; t < 2; t++) xx[t][0] = xx[t][1] = 0;
#pragma unroll
        for (int m = K - 1; m >= 0; m--) {
#pragma unroll
          for (int t = 0; t < 2; t++) {
            const int j = (chy0 + t) * K + m;
            const double2 nr = V::ld(tb + j * 8 + kSlotNY);  // nY, 1/b'
            const double cp = tb[j * 8 + kSlotCP];
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const double zv = y[t][h][m] + cp * zin[t][h];
              xx[t][h] = nr.y * zv + nr.x * xx[t][h];
              y[t][h][m] = xx[t][h];
            }
          }
        }
#pragma unroll
        for (int t = 0; t < 2; t++) V::st(yb + (2 * warp + t) * 64 + 2 * lane, xx[t][0], xx[t][1]);
      }
      if (more) {
        piv_store(1);
        piv_load(k - 1, 2);
      }
      __syncthreads();
      if (clustered) {
        for (int col = tid; col < X; col += NT) {
          const int cg2 = col >> 6, w = col & 63;
          double a = 0;
          for (int c2 = Ls.CHy - 1; c2 >= 0; c2--)
            a = yb[(cg2 * Ls.CHy + c2) * 64 + w] + tb[(c2 * K) * 8 + kSlotCQ] * a;
          for (int h = 0; h < rank; h++)
            st_async(cluster_addr(inB + rank * X + col, h), a, cluster_addr(barB, h));
        }
        if (tid == 0) {
          double b = 1;
          for (int c2 = Ls.CHy - 1; c2 >= 0; c2--) b = tb[(c2 * K) * 8 + kSlotCQ] * b;
          for (int h = 0; h < rank; h++) st_async(cluster_addr(totB + rank, h), b, cluster_addr(barB, h));
          mbar_expect_tx(barB, fold_bytes_B);
        }
        if (!mbar_wait_cluster(barB, phB, timed_out ? kWaitPollsAfterTimeout : kWaitPolls)) {
          timed_out = true;
          atomicExch(args.err, 3);
        }
        phB ^= 1u;
        for (int col = tid; col < X; col += NT) {
          double xv = 0;
          for (int q = C - 1; q > rank; q--) xv = inB[q * X + col] + totB[q] * xv;
          s_xin[col] = xv;
        }
        __syncthreads();
      }
      if (more) {
        piv_store(2);
        piv_load(k - 1, 3);
      }
      {
        double xin[2][2];
        xin[1][0] = xin[1][1] = 0;
        if (clustered) {
          const double2 t = V::ld(s_xin + col0);
          xin[1][0] = t.x;
          xin[1][1] = t.y;
        }
        for (int c2 = Ls.CHy - 1; c2 > chy0 + 1; c2--) {
          const double2 b = V::ld(yb + (cgy * Ls.CHy + c2) * 64 + 2 * lane);
          const double cq = tb[(c2 * K) * 8 + kSlotCQ];
          xin[1][0] = b.x + cq * xin[1][0];
          xin[1][1] = b.y + cq * xin[1][1];
        }
        {
          const double cq = tb[((chy0 + 1) * K) * 8 + kSlotCQ];
          xin[0][0] = y[1][0][0] + cq * xin[1][0];
          xin[0][1] = y[1][1][0] + cq * xin[1][1];
        }
#pragma unroll
        for (int t = 0; t < 2; t++) {
#pragma unroll
          for (int m = 0; m < K; m++) {
            const int j = (chy0 + t) * K + m;
            const double cq = tb[j * 8 + kSlotCQ];
#pragma unroll
            for (int h = 0; h < 2; h++) y[t][h][m] = y[t][h][m] + cq * xin[t][h];
            V::st(A + (j + 1) * LD + col0, y[t][0][m], y[t][1][m]);
          }
        }
        // the row group's first and last rows, for the groups around it
        {
          const int g = chy0 / 2;
          V::st(sTop + g * X + col0, y[0][0][0], y[0][1][0]);
          V::st(sBot + g * X + col0, y[1][0][K - 1], y[1][1][K - 1]);
        }
        // cluster halo rows for the next step (see the paired kernel)
        if (has_prev && chy0 == 0) {
          const double* th = sTh + 8 * (sc & 1);
          const double rbh = th[kSlotRB], nyh = th[kSlotNY];
          const double2 zr = V::ld(s_zin + col0);
          V::st(A + col0, rbh * zr.x + nyh * y[0][0][0], rbh * zr.y + nyh * y[0][1][0]);
        }
        if (has_next && chy0 + 2 == Ls.CHy) V::st(A + (Ycs + 1) * LD + col0, xin[1][0], xin[1][1]);
        if (s == steps - 1 && out_h >= 0) {
          double pvl = 0;
#pragma unroll
          for (int t = 0; t < 2; t++)
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
              for (int m = 0; m < K; m++)
                if (h == out_h && t * K + m == out_m) pvl = y[t][h][m];
          args.out[c.out + item.strike] = pvl;  // myResult[myYindex, myXindex]
        }
      }
      __syncwarp();
      if (more) {
        piv_store(3);
        tmem_wait_st();
      }
    }
  }
  if (clustered) cg::this_cluster().sync();
  tmem_fence_before_sync();
  __syncthreads();
  tmem_fence_after_sync();
  if (warp == 0) tmem_dealloc(*s_taddr, kCols);
}

}  // namespace lvc
