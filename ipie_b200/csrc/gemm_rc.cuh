// FP64 tensor-core products of real left operands with complex right operands:
//
//     C[m][n] = sum_s c_s sum_k A_s[m][k] B_s[k][n],      c_s = 1 or i,
//
// up to four segments s, each with its own operands and K extent, summed into one accumulator: both
// spin blocks of the force bias, or the real and imaginary parts of complex Cholesky vectors, are
// one launch.  A_s is row-major (K_s doubles per row); B_s is complex, either walker-major
// B[n][k] (k contiguous) or B[k][n] (n contiguous).
//
// A CTA computes BM x BN complex entries with mma.sync m8n8k4 f64: a lane's complex right fragment
// is one 16-byte shared-memory load that feeds two MMAs (real and imaginary part), so each k step
// of a 32 x 16 warp tile is 4 + 2 loads for 16 MMAs.  Both operands reach shared memory through a
// three-stage ring of cp.async copies in their own layouts (16-byte copies where the rows of A
// are 16-byte aligned, 8-byte ones otherwise), two chunks of BK = 16 ahead, with one barrier per
// chunk; the row strides (4 mod 16 doubles for A, 4 or 2 mod 8 complex for B) keep the fragment
// loads free of bank conflicts.
//
// Small outputs leave most SMs idle and make K a serial chain (a 120 x 64 output is two 128 x 32
// tiles), so the tile shape and a split of K over a cluster of S CTAs are chosen together from the
// sizes (rc_plan): the S partial tiles are added through distributed shared memory in rank order,
// which needs no workspace and keeps the result the same from run to run (for one batch size: another
// one can take another split and so add a walker's terms in another order).
//
// The bound is the f64 tensor pipe (36.9 TFLOP/s with operands in registers).  Measured, with two
// register-staged 128 x 64 tiles and one launch per operand before: force bias of 1024 walkers,
// X = 960, K = 4160: 788 -> 632 us (26 TFLOP/s); 640 walkers, X = 600, two spins of K = 1620: 400 ->
// 212 us; 64 walkers, X = 120, K = 130: 18.1 -> 4.7 us; VHS of 1024 walkers, M = 160, X = 960: 1920 ->
// 1683 us (30 TFLOP/s); complex vectors, 256 walkers, M = 40, X = 160: force bias 234 -> 37 us, VHS
// 79 -> 57 us.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace ipie_b200 {

constexpr int kRcBK = 16;
constexpr int kRcStages = 3;
constexpr int kRcMaxSeg = 4;

struct RcSegment {
  const double* a;
  const double2* b;
  int K;
  int times_i;
};

struct RcOperands {
  RcSegment seg[kRcMaxSeg];
  int nseg;
  int vec_a, vec_b;  // 16-byte copies allowed
  int chunks;        // chunks of kRcBK over all segments
};

template <int BM_, int BN_, int WARPS_M_, int WARPS_N_, int OCC_>
struct RcCfg {
  static constexpr int BM = BM_, BN = BN_, WARPS_M = WARPS_M_, WARPS_N = WARPS_N_, OCC = OCC_;
  static constexpr int THREADS = 32 * WARPS_M * WARPS_N;
  static constexpr int WTM = BM / WARPS_M, WTN = BN / WARPS_N, FM = WTM / 8, FN = WTN / 8;
  static constexpr int LDA = kRcBK + 4;
  static constexpr int LDBK = kRcBK + 4;  // B[n][k]: complex row stride
  static constexpr int LDBN = BN + 2;     // B[k][n]: complex row stride
  static constexpr int A_DOUBLES = BM * LDA;
  static constexpr int B_DOUBLES = 2 * (BN * LDBK > kRcBK * LDBN ? BN * LDBK : kRcBK * LDBN);
  static constexpr int LDC = BN + 1;  // parked partial tile
  static constexpr size_t SMEM = sizeof(double) * kRcStages * (A_DOUBLES + B_DOUBLES);
  static_assert(WTM % 8 == 0 && WTN % 8 == 0, "whole 8 x 8 tiles per warp");
  static_assert(sizeof(double2) * BM * LDC <= SMEM, "the partial tile parks in the copy ring");
  static_assert(BN % 8 == 0 && (LDBN & 7) == 2 && (LDBK & 7) == 4 && (LDA & 15) == 4, "conflict-free strides");
};

// One lane's accumulators: real and imaginary parts of rows 8 i + g, columns 8 j + 2 t + q of its warp tile.
template <class C>
struct RcAcc {
  double re[C::FM][C::FN][2], im[C::FM][C::FN][2];
};

// Chunks c0 .. c1 - 1 of the tile at (m0, n0).  WALKER_MAJOR: B[n][k]; else B[k][n].  TIMES_I: some
// segment has times_i.
template <class C, bool WALKER_MAJOR, bool TIMES_I>
__device__ __forceinline__ void rc_mainloop(int M, int N, int m0, int n0, const RcOperands& op, int c0, int c1,
                                            double* rc_sm, RcAcc<C>& acc) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wm0 = (warp / C::WARPS_N) * C::WTM, wn0 = (warp % C::WARPS_N) * C::WTN;
  // next chunk to copy: its segment and first k
  int lseg = 0, lk = c0;
  while (lseg < op.nseg - 1 && lk >= (op.seg[lseg].K + kRcBK - 1) / kRcBK) {
    lk -= (op.seg[lseg].K + kRcBK - 1) / kRcBK;
    ++lseg;
  }
  int cseg = lseg, ck = lk;  // segment of the chunk being multiplied, for TIMES_I
  lk *= kRcBK;
  auto load = [&](int c) {
    if (c < c1) {
      double* sA = rc_sm + (c - c0) % kRcStages * (C::A_DOUBLES + C::B_DOUBLES);
      double2* sB = reinterpret_cast<double2*>(sA + C::A_DOUBLES);
      const RcSegment& sg = op.seg[lseg];
      const int K = sg.K;
      if (op.vec_a) {
        constexpr int V = kRcBK / 2;
#pragma unroll
        for (int i = 0; i < (C::BM * V + C::THREADS - 1) / C::THREADS; ++i) {
          const int e = tid + i * C::THREADS, r = e / V, k = 2 * (e % V);
          if (C::BM * V % C::THREADS && r >= C::BM) break;
          const bool in = m0 + r < M && lk + k < K;
          cp_async16(sA + r * C::LDA + k, in ? sg.a + (size_t)(m0 + r) * K + lk + k : sg.a, in ? 16 : 0);
        }
      } else {
#pragma unroll
        for (int i = 0; i < (C::BM * kRcBK + C::THREADS - 1) / C::THREADS; ++i) {
          const int e = tid + i * C::THREADS, r = e / kRcBK, k = e % kRcBK;
          if (C::BM * kRcBK % C::THREADS && r >= C::BM) break;
          const bool in = m0 + r < M && lk + k < K;
          cp_async8(sA + r * C::LDA + k, in ? sg.a + (size_t)(m0 + r) * K + lk + k : sg.a, in ? 8 : 0);
        }
      }
#pragma unroll
      for (int i = 0; i < (C::BN * kRcBK + C::THREADS - 1) / C::THREADS; ++i) {
        const int e = tid + i * C::THREADS;
        if (C::BN * kRcBK % C::THREADS && e >= C::BN * kRcBK) break;
        const int n = WALKER_MAJOR ? e / kRcBK : e % C::BN, k = WALKER_MAJOR ? e % kRcBK : e / C::BN;
        const bool in = n0 + n < N && lk + k < K;
        double2* dst = WALKER_MAJOR ? sB + n * C::LDBK + k : sB + k * C::LDBN + n;
        const double2* src =
            in ? (WALKER_MAJOR ? sg.b + (size_t)(n0 + n) * K + lk + k : sg.b + (size_t)(lk + k) * N + n0 + n) : sg.b;
        if (op.vec_b) {
          cp_async16(dst, src, in ? 16 : 0);
        } else {
          cp_async8(&dst->x, &src->x, in ? 8 : 0);
          cp_async8(&dst->y, &src->y, in ? 8 : 0);
        }
      }
      lk += kRcBK;
      if (lk >= K) {
        lk = 0;
        ++lseg;
      }
    }
    cp_async_commit();  // an empty group past the end keeps one group per chunk
  };

#pragma unroll
  for (int i = 0; i < C::FM; ++i)
#pragma unroll
    for (int j = 0; j < C::FN; ++j) acc.re[i][j][0] = acc.re[i][j][1] = acc.im[i][j][0] = acc.im[i][j][1] = 0.0;

  load(c0);
  load(c0 + 1);
  for (int c = c0; c < c1; ++c) {
    cp_async_wait<1>();
    __syncthreads();  // chunk c has landed for everyone, chunk c - 1 is consumed
    load(c + 2);
    const double* sA = rc_sm + (c - c0) % kRcStages * (C::A_DOUBLES + C::B_DOUBLES) + (wm0 + g) * C::LDA + t;
    const double2* sB = reinterpret_cast<const double2*>(rc_sm + (c - c0) % kRcStages * (C::A_DOUBLES + C::B_DOUBLES) +
                                                         C::A_DOUBLES) +
                        (WALKER_MAJOR ? (wn0 + g) * C::LDBK + t : t * C::LDBN + wn0 + g);
    const bool ti = TIMES_I && op.seg[cseg].times_i;
#pragma unroll
    for (int kk = 0; kk < kRcBK; kk += 4) {
      double a[C::FM];
      double2 b[C::FN];
#pragma unroll
      for (int i = 0; i < C::FM; ++i) a[i] = sA[8 * i * C::LDA + kk];
#pragma unroll
      for (int j = 0; j < C::FN; ++j) {
        b[j] = WALKER_MAJOR ? sB[8 * j * C::LDBK + kk] : sB[kk * C::LDBN + 8 * j];
        if (TIMES_I && ti) b[j] = make_double2(-b[j].y, b[j].x);
      }
#pragma unroll
      for (int i = 0; i < C::FM; ++i)
#pragma unroll
        for (int j = 0; j < C::FN; ++j) {
          dmma884(acc.re[i][j], a[i], b[j].x);
          dmma884(acc.im[i][j], a[i], b[j].y);
        }
    }
    if (TIMES_I && (++ck) * kRcBK >= op.seg[cseg].K) {
      ck = 0;
      cseg = min(cseg + 1, op.nseg - 1);
    }
  }
}

template <class C, bool WALKER_MAJOR, bool TIMES_I, class Epi>
__global__ void __launch_bounds__(C::THREADS, C::OCC)
    rc_gemm_kernel(int M, int N, const __grid_constant__ RcOperands op, int S, Epi epi) {
  extern __shared__ __align__(16) double rc_sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wm0 = (warp / C::WARPS_N) * C::WTM, wn0 = (warp % C::WARPS_N) * C::WTN;
  const int rank = (int)(blockIdx.x % S);
  const int m0 = (int)blockIdx.y * C::BM, n0 = (int)(blockIdx.x / S) * C::BN;
  RcAcc<C> acc;
  rc_mainloop<C, WALKER_MAJOR, TIMES_I>(M, N, m0, n0, op, (int)((long long)op.chunks * rank / S),
                                        (int)((long long)op.chunks * (rank + 1) / S), rc_sm, acc);
  if (S == 1) {
#pragma unroll
    for (int i = 0; i < C::FM; ++i)
#pragma unroll
      for (int j = 0; j < C::FN; ++j) {
        const int m = m0 + wm0 + 8 * i + g, n = n0 + wn0 + 8 * j + 2 * t;
        if (m >= M) continue;
#pragma unroll
        for (int q = 0; q < 2; ++q)
          if (n + q < N) epi(m, n + q, make_double2(acc.re[i][j][q], acc.im[i][j][q]));
      }
    return;
  }
  // partial tiles of the cluster: park, then each CTA adds and writes its share of the rows
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  cp_async_wait<0>();
  __syncthreads();
  double2* sC = reinterpret_cast<double2*>(rc_sm);
#pragma unroll
  for (int i = 0; i < C::FM; ++i)
#pragma unroll
    for (int j = 0; j < C::FN; ++j) {
      double2* d = sC + (wm0 + 8 * i + g) * C::LDC + wn0 + 8 * j + 2 * t;
      d[0] = make_double2(acc.re[i][j][0], acc.im[i][j][0]);
      d[1] = make_double2(acc.re[i][j][1], acc.im[i][j][1]);
    }
  cl.sync();
  const int rows = C::BM / S;  // BM and S are powers of two, S <= 8 <= BM
  for (int e = tid; e < rows * C::BN; e += C::THREADS) {
    const int r = rank * rows + e % rows, n = e / rows;
    if (m0 + r >= M || n0 + n >= N) continue;
    double2 v = make_double2(0.0, 0.0);
    for (int q = 0; q < S; ++q) v = cadd(v, *cl.map_shared_rank(sC + r * C::LDC + n, q));
    epi(m0 + r, n0 + n, v);
  }
  cl.sync();  // nobody leaves while its tile is being read
}

using RcBig = RcCfg<128, 32, 4, 2, 2>;
using RcMid = RcCfg<64, 32, 4, 2, 2>;
using RcSmall = RcCfg<32, 16, 2, 2, 4>;

// Tile shape (0: 128 x 32, 1: 64 x 32, 2: 32 x 16) and K split from the sizes: the SM with the most
// CTAs bounds the launch, at the tensor pipe's BM BN / 2 cycles per chunk of 16 where enough of them
// run at once, or at the latency of a CTA's own chunks (copy, barrier and a dependent MMA chain:
// about 450 cycles for the small tile, 1100 and 2100 for the larger ones, whose chunks hold 4 and 8
// times its MMAs) plus the start, the epilogue and, when split, the exchange of partial tiles.
struct RcPlan {
  int tile, S;
};
inline RcPlan rc_plan(int M, int N, int chunks) {
  static const struct {
    int bm, bn, occ;
    double latency, pipe;
  } tiles[3] = {{128, 32, 2, 2100.0, 1.05}, {64, 32, 2, 1100.0, 1.1}, {32, 16, 4, 450.0, 1.25}};
  RcPlan best{0, 1};
  double best_cost = 1e300;
  for (int c = 0; c < 3; ++c) {
    const long long out = (long long)((M + tiles[c].bm - 1) / tiles[c].bm) * ((N + tiles[c].bn - 1) / tiles[c].bn);
    if (c > 0 && (M + tiles[c].bm - 1) / tiles[c].bm > 65535) break;  // grid rows
    for (int S = 1; S <= 8; S *= 2) {
      if (S > 1 && chunks < 2 * S) break;
      const double per = (chunks + S - 1) / S;
      const double n = (double)((out * S + 147) / 148), rounds = (double)(((int)n + tiles[c].occ - 1) / tiles[c].occ);
      const double pipe = n * per * tiles[c].bm * tiles[c].bn / 2.0 * tiles[c].pipe;
      const double serial = rounds * per * tiles[c].latency;
      const double cost = (pipe > serial ? pipe : serial) + rounds * (S > 1 ? 5000.0 : 3000.0);
      if (cost < best_cost) {
        best_cost = cost;
        best = RcPlan{c, S};
      }
    }
  }
  return best;
}

template <class C, bool WALKER_MAJOR, bool TIMES_I, class Epi>
inline cudaError_t rc_launch_cfg(int M, int N, const RcOperands& op, int S, Epi epi, cudaStream_t st) {
  auto k = rc_gemm_kernel<C, WALKER_MAJOR, TIMES_I, Epi>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((N + C::BN - 1) / C::BN * S), (unsigned)((M + C::BM - 1) / C::BM));
  cfg.blockDim = dim3(C::THREADS);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)S;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, k, M, N, op, S, epi);
  if (e != cudaSuccess) return e;
  note_launch();
  return cudaGetLastError();
}

// C (M x N complex) from the segments through the epilogue epi(m, n, value).
template <bool WALKER_MAJOR, bool TIMES_I, class Epi>
inline cudaError_t rc_gemm(int M, int N, const RcSegment* seg, int nseg, Epi epi, cudaStream_t st) {
  if (M <= 0 || N <= 0 || nseg < 0 || nseg > kRcMaxSeg) return cudaErrorInvalidValue;
  RcOperands op = {};
  op.vec_a = op.vec_b = 1;
  for (int s = 0; s < nseg; ++s) {
    if (seg[s].K < 0) return cudaErrorInvalidValue;
    if (seg[s].K == 0) continue;  // an empty spin block adds nothing (all empty: C = 0)
    op.seg[op.nseg++] = seg[s];
    op.chunks += (seg[s].K + kRcBK - 1) / kRcBK;
    if (seg[s].K % 2 != 0 || reinterpret_cast<uintptr_t>(seg[s].a) % 16 != 0) op.vec_a = 0;
    if (reinterpret_cast<uintptr_t>(seg[s].b) % 16 != 0) op.vec_b = 0;
  }
  const RcPlan p = rc_plan(M, N, op.chunks);
  switch (p.tile) {
    case 0: return rc_launch_cfg<RcBig, WALKER_MAJOR, TIMES_I>(M, N, op, p.S, epi, st);
    case 1: return rc_launch_cfg<RcMid, WALKER_MAJOR, TIMES_I>(M, N, op, p.S, epi, st);
    default: return rc_launch_cfg<RcSmall, WALKER_MAJOR, TIMES_I>(M, N, op, p.S, epi, st);
  }
}

}  // namespace ipie_b200
