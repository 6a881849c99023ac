// Hand-written adjoint of the local energy with respect to the one-body
// Hamiltonian: e1b_w = sum_s tr(G_s^w h1_s) with the mixed Green's function
// G_s^w = psi_s^* Ghalf_s^w (M x M), so for upstream gradients g_w
//     dL/dh1_s = sum_w g_w G_s^w = psi_s^* (sum_w g_w Ghalf_s^w).
// With g_w = w_w / sum w this is the mixed-estimator one-body density matrix.
#include <cooperative_groups.h>

#include "../../include/ipie_b200.h"
#include "common.cuh"
#include "kernels.h"

namespace ipie_b200 {

// acc[k] = sum_w coeff[w] * ghalf[w][k]   (k over N*M), fixed summation order.
__global__ void weighted_walker_sum_kernel(const double2* __restrict__ ghalf, const double* __restrict__ coeff, int W,
                                           int K, double2* __restrict__ acc) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  double2 s = make_double2(0.0, 0.0);
  for (int w = 0; w < W; ++w) {
    const double2 g = ghalf[(size_t)w * K + k];
    const double c = coeff[w];
    s.x += c * g.x;
    s.y += c * g.y;
  }
  acc[k] = s;
}

// out[p][q] (+)= sum_i psi_c[p][i] * A[i][q]   (psi_c (M, N), A (N, M), out (M, M))
__global__ void expand_half_kernel(const double2* __restrict__ psi_c, const double2* __restrict__ A, int M, int N,
                                   double2* __restrict__ out, int accumulate) {
  const int p = blockIdx.y, q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= M) return;
  double2 s = make_double2(0.0, 0.0);
  for (int i = 0; i < N; ++i) s = cadd(s, cmul(psi_c[(size_t)p * N + i], A[(size_t)i * M + q]));
  const size_t o = (size_t)p * M + q;
  out[o] = accumulate ? cadd(out[o], s) : s;
}

// rH1[i][q] = sum_p psi_c[p][i] * h1[p][q]   (psi_c (M, N), h1 (M, M) real, rH1 (N, M) complex)
__global__ void rotate_onebody_kernel(const double2* __restrict__ psi_c, const double* __restrict__ h1, int M, int N,
                                      double2* __restrict__ rh1) {
  const int i = blockIdx.y, q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= M) return;
  double2 s = make_double2(0.0, 0.0);
  for (int p = 0; p < M; ++p) {
    const double2 c = psi_c[(size_t)p * N + i];
    const double h = h1[(size_t)p * M + q];
    s.x += c.x * h;
    s.y += c.y * h;
  }
  rh1[(size_t)i * M + q] = s;
}


// Vector-Jacobian product of the single-determinant local energy with respect to one spin's
// half-rotated Green's function G (N, M):
//     E = f1 sum G . rH1 + fc (sum_x X_x^2) - fx sum_x tr(T_x T_x) + (other spin, ecore),
//     X_x = sum_s L_s,x . G_s,   T_x = L_x G^T (N, N),   L_x (N, M) row x of rchol,
//     dE/dG = f1 rH1 + 2 fc sum_x X_x L_x - 2 fx sum_x T_x L_x,
// gbar = ebar[w] * dE/dG.
//
// Two chained products on the f64 tensor cores, T never in global memory: a CTA owns WB walkers
// (R = WB N rows) and walks the Cholesky rows in blocks of XB vectors, copied to shared memory one
// block ahead.  Per block
//     S[(w,i), (x,j)] = sum_p G_w[i,p] L_x[j,p]                     (R x XB N, K = M)
//     Q[(w,j), (x,i)] = 2 fc X_wx [i == j] - 2 fx S[(w,i), (x,j)]   (transposed inside each (w, x))
//     acc[(w,j), p] += sum_(x,i) Q[(w,j), (x,i)] L_x[i,p]           (R x M, K = XB N)
// G stays in shared memory, acc in registers; both products read the same copy of L (its row
// stride, 4 mod 16 doubles, serves it as either right operand without bank conflicts).  Work per
// L entry read is 8 R operations, so the bound is the f64 tensor pipe.  Few walkers: the x range
// is split over a cluster of S CTAs whose accumulators are added through distributed shared memory
// in rank order.  512 walkers, M = 76, N = 10, X = 400, one spin: 6.91 ms as scalar products from
// shared memory, 0.64 ms here (19.4 TFLOP/s; the tensor pipe's peak is 36.9; 0.70 ms with blocks of 40
// Cholesky rows instead of 80, X_wx read from global memory and the index divisions in the loop).
constexpr int kVjWarps = 16;
constexpr int kVjThreads = 32 * kVjWarps;
constexpr int kVjMaxUnits = 8;  // 8 x 8 accumulator tiles per warp (4 doubles per lane each)

struct VjpShape {
  int WB, XB, S;      // walkers per CTA, Cholesky vectors per block, CTAs per cluster
  int RT, R;          // 8-row tiles and rows of the CTA's walkers
  int KB, CT1, KB4;   // Cholesky rows per block, their 8-row tiles, rounded up to 4
  int MP4, CT2;       // columns rounded up to 4, 8-column tiles
  int ldg, ldl, ldq;  // row strides: G and Q in double2 (4 mod 8), L in double (4 mod 16)
  int nbuf;           // buffers of L
  int units;          // accumulator tiles per warp
  size_t smem;
};

// smallest stride >= n that is 4 modulo m (m a power of two)
static int stride4(int n, int m) { return n + ((4 - n) & (m - 1)); }

// The split with the least time: the rounds in which the clusters run, times a CTA's blocks -- 10 per step of
// 4 K and round of S tiles over the warps, a warp's 1 to 8 accumulator tiles per 4 K of the second product
// (kVjTiles: odd counts check each tile, seven and eight spill), 1350 for barriers and the copy -- and 9000 for
// start and end, 3000 more for the cluster's sum.  The units are relative; they and the clusters that run
// at once (whole ones per group of SMs: 33 of four, 15 of eight) are fitted to 251 shapes with every split of
// each (1 to 777 walkers, M = 26 to 250, N = 1 to 32): the choice is within 0.4 % of the best on average, 13 %
// at worst.  31 walkers, X = 500, M = 110, N = 2: 22 us with clusters of eight, 76 with single CTAs; 31, X = 1000, M =
// 200, N = 20: 1.25 ms with clusters of four, 2.67 of eight.
constexpr double kVjTiles[kVjMaxUnits] = {20.0, 48.0, 87.0, 103.0, 160.0, 197.0, 248.0, 344.0};
static bool vjp_shape(int W, int X, int M, int N, VjpShape& best) {
  if (M > 256 || N > 32) return false;
  double best_cost = 0.0;
  bool found = false;
  VjpShape s;
  s.MP4 = (M + 3) & ~3;
  s.CT2 = (M + 7) / 8;
  s.ldg = stride4(s.CT2 * 8, 8);
  s.ldl = stride4(s.CT2 * 8, 16);
  for (s.WB = 1; s.WB <= W; ++s.WB) {
    s.R = s.WB * N;
    s.RT = (s.R + 7) / 8;
    s.units = (s.RT * s.CT2 + kVjWarps - 1) / kVjWarps;
    if (s.RT > 5 || s.units > kVjMaxUnits) break;
    // blocks of up to 80 Cholesky rows, double buffered, where shared memory holds them
    bool fits = false;
    for (s.nbuf = 2; s.nbuf >= 1 && !fits; --s.nbuf) {
      for (s.XB = 80 / N; s.XB >= 1 && !fits; --s.XB) {
        s.KB = s.XB * N;
        s.CT1 = (s.KB + 7) / 8;
        s.KB4 = (s.KB + 3) & ~3;
        s.ldq = stride4(s.KB4, 8);
        s.smem = sizeof(double2) * ((size_t)s.RT * 8 * (s.ldg + s.ldq) + 2 * s.WB * s.XB) +
                 sizeof(double) * s.nbuf * s.CT1 * 8 * s.ldl + sizeof(int) * 3 * (s.R + s.KB);
        fits = s.smem <= 232448;
        if (fits) break;
      }
      if (fits) break;
    }
    if (!fits) break;
    const int nblk = (X + s.XB - 1) / s.XB;
    for (s.S = 1; s.S <= 8; s.S *= 2) {
      if (s.S > nblk) break;
      const int at_once = s.S == 1 ? 148 : s.S == 2 ? 74 : s.S == 4 ? 33 : 15;
      const double rounds = (double)(((W + s.WB - 1) / s.WB + at_once - 1) / at_once);
      const double block = 10.0 * ((s.RT * s.CT1 + kVjWarps - 1) / kVjWarps) * s.MP4 + kVjTiles[s.units - 1] * s.KB4 + 1350.0;
      const double cost = rounds * (block * ((nblk + s.S - 1) / s.S) + (s.S > 1 ? 12000.0 : 9000.0));
      if (!found || cost < best_cost) {
        best = s;
        best_cost = cost;
        found = true;
      }
    }
  }
  return found;
}

template <int U2>
__global__ void __launch_bounds__(kVjThreads, 1)
    energy_vjp_mma_kernel(const double* __restrict__ rchol, const double2* __restrict__ ghalf,
                          const double2* __restrict__ rh1, const double2* __restrict__ xv,
                          const double2* __restrict__ ebar, int W, int X, int M, int N, double f1, double fc2,
                          double fx2, VjpShape s, int vec, double2* __restrict__ gbar) {
  extern __shared__ __align__(16) unsigned char vjp_sm[];
  double2* const sG = reinterpret_cast<double2*>(vjp_sm);  // (8 RT, ldg)
  double2* const sQ = sG + s.RT * 8 * s.ldg;               // (8 RT, ldq)
  double2* const sX = sQ + s.RT * 8 * s.ldq;                // 2 x (WB, XB): X_wx of a block
  double* const sL = reinterpret_cast<double*>(sX + 2 * s.WB * s.XB);  // nbuf x (8 CT1, ldl)
  int* const tr = reinterpret_cast<int*>(sL + s.nbuf * s.CT1 * 8 * s.ldl);  // rows of S: place in Q, w, i
  int* const tc = tr + 3 * s.R;                                             // columns of S: place in Q, x, j
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int w0 = (int)(blockIdx.x / s.S) * s.WB, rank = (int)(blockIdx.x % s.S);
  const int lsize = s.CT1 * 8 * s.ldl;
  // zeros everywhere first: the padding rows and columns keep them
  for (int e = tid; e < s.RT * 8 * (s.ldg + s.ldq); e += kVjThreads) sG[e] = make_double2(0.0, 0.0);
  for (int e = tid; e < s.nbuf * lsize; e += kVjThreads) sL[e] = 0.0;
  for (int r = tid; r < s.R; r += kVjThreads) {
    const int wl = r / N, i = r - wl * N;
    tr[r] = wl * N * s.ldq + i;
    tr[s.R + r] = wl;
    tr[2 * s.R + r] = i;
  }
  for (int c = tid; c < s.KB; c += kVjThreads) {
    const int xl = c / N, j = c - xl * N;
    tc[c] = j * s.ldq + xl * N;
    tc[s.KB + c] = xl;
    tc[2 * s.KB + c] = j;
  }
  __syncthreads();
  // Cholesky rows of block b (contiguous in rchol) into buffer `buf`, zeros for vectors past X, and
  // its X_wx (zeros past X and W) into the buffer of b's parity
  auto load_block = [&](int b, int buf) {
    const long long row0 = (long long)b * s.KB, rows = (long long)X * N - row0;
    const double* src = rchol + row0 * M;
    double* dst = sL + buf * lsize;
    if (vec) {
      const int mv = M >> 1;
      for (int e = tid; e < s.KB * mv; e += kVjThreads) {
        const int r = e / mv, c = 2 * (e - r * mv);
        const bool in = r < rows;
        cp_async16(dst + r * s.ldl + c, in ? src + (size_t)r * M + c : rchol, in ? 16 : 0);
      }
    } else {
      for (int e = tid; e < s.KB * M; e += kVjThreads) {
        const int r = e / M, c = e - r * M;
        const bool in = r < rows;
        cp_async8(dst + r * s.ldl + c, in ? src + (size_t)r * M + c : rchol, in ? 8 : 0);
      }
    }
    for (int e = tid; e < s.WB * s.XB; e += kVjThreads) {
      const int wl = e / s.XB, x = b * s.XB + e - wl * s.XB;
      const bool in = x < X && w0 + wl < W;
      cp_async16(sX + (b & 1) * s.WB * s.XB + e, in ? xv + (size_t)(w0 + wl) * X + x : xv, in ? 16 : 0);
    }
    cp_async_commit();
  };
  const int nblk = (X + s.XB - 1) / s.XB;
  const int b0 = (int)((long long)nblk * rank / s.S), b1 = (int)((long long)nblk * (rank + 1) / s.S);
  load_block(b0, 0);
  {
    // the walkers' G rows are contiguous
    const double2* gw = ghalf + (size_t)w0 * N * M;
    const int live = min(s.R, (W - w0) * N);
    for (int e = tid; e < live * M; e += kVjThreads) sG[(e / M) * s.ldg + e % M] = gw[e];
  }
  // this warp's accumulator tiles: ids warp U2 .. warp U2 + U2 - 1, the row tile running fastest
  double2 acc[U2][2];  // [tile][column 2t + q]
  int arow[U2], bcol[U2];
  const int ntile = s.RT * s.CT2;
#pragma unroll
  for (int u = 0; u < U2; ++u) {
    const int id = min(warp * U2 + u, ntile - 1);  // tiles past the end repeat the last one, unused
    arow[u] = ((id % s.RT) * 8 + g) * s.ldq + t;
    bcol[u] = t * s.ldl + (id / s.RT) * 8 + g;
    acc[u][0] = acc[u][1] = make_double2(0.0, 0.0);
  }
  const int mine = max(0, min(U2, ntile - warp * U2));
  for (int b = b0; b < b1; ++b) {
    const int cur = s.nbuf == 2 ? (b - b0) & 1 : 0;
    const double* l = sL + cur * lsize;
    cp_async_wait<0>();
    __syncthreads();  // block b has landed; everyone is done with block b - 1
    if (s.nbuf == 2 && b + 1 < b1) load_block(b + 1, cur ^ 1);
    // S tiles, one per warp at a time; two accumulator sets shorten the dependent chain
    for (int id = warp; id < s.RT * s.CT1; id += kVjWarps) {
      const int rt = id % s.RT, ct = id / s.RT;
      const double2* pa = sG + (rt * 8 + g) * s.ldg + t;
      const double* pb = l + (ct * 8 + g) * s.ldl + t;
      double dr[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, di[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
      int k = 0;
#pragma unroll 2
      for (; k + 8 <= s.MP4; k += 8) {
        const double2 a0 = pa[k], a1 = pa[k + 4];
        const double v0 = pb[k], v1 = pb[k + 4];
        dmma884(dr[0], a0.x, v0);
        dmma884(di[0], a0.y, v0);
        dmma884(dr[1], a1.x, v1);
        dmma884(di[1], a1.y, v1);
      }
      if (k < s.MP4) {
        const double2 a0 = pa[k];
        const double v0 = pb[k];
        dmma884(dr[0], a0.x, v0);
        dmma884(di[0], a0.y, v0);
      }
      const int r = rt * 8 + g;
      if (r < s.R) {
        const int qr = tr[r], wl = tr[s.R + r], i = tr[2 * s.R + r];
        const double2* cx = sX + (b & 1) * s.WB * s.XB + wl * s.XB;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int c = ct * 8 + 2 * t + q;
          if (c < s.KB) {
            double2 v = make_double2(-fx2 * (dr[0][q] + dr[1][q]), -fx2 * (di[0][q] + di[1][q]));
            if (i == tc[2 * s.KB + c]) {
              const double2 x = cx[tc[s.KB + c]];
              v.x += fc2 * x.x;
              v.y += fc2 * x.y;
            }
            sQ[qr + tc[c]] = v;
          }
        }
      }
    }
    __syncthreads();
    // acc += Q L, each block summed by itself first: one chain over all X N terms doubles the rounding error
    if (mine > 0) {
      double re[U2][2], im[U2][2];
#pragma unroll
      for (int u = 0; u < U2; ++u) re[u][0] = re[u][1] = im[u][0] = im[u][1] = 0.0;
      if (mine == U2) {
        for (int k = 0; k < s.KB4; k += 4) {
          const double* lk = l + k * s.ldl;
#pragma unroll
          for (int u = 0; u < U2; ++u) {
            const double2 a = sQ[arow[u] + k];
            const double v = lk[bcol[u]];
            dmma884(re[u], a.x, v);
            dmma884(im[u], a.y, v);
          }
        }
      } else {
        for (int k = 0; k < s.KB4; k += 4) {
          const double* lk = l + k * s.ldl;
#pragma unroll
          for (int u = 0; u < U2; ++u) {
            if (u >= mine) break;
            const double2 a = sQ[arow[u] + k];
            const double v = lk[bcol[u]];
            dmma884(re[u], a.x, v);
            dmma884(im[u], a.y, v);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U2; ++u)
#pragma unroll
        for (int q = 0; q < 2; ++q) acc[u][q] = cadd(acc[u][q], make_double2(re[u][q], im[u][q]));
    }
    if (s.nbuf == 1) {
      __syncthreads();  // the one buffer is free
      if (b + 1 < b1) load_block(b + 1, 0);
    }
  }
  auto finish = [&](int r, int p, double2 a) {
    const int wl = r / N, j = r - wl * N, w = w0 + wl;
    if (w >= W) return;
    const double2 h = rh1[(size_t)j * M + p];
    gbar[((size_t)w * N + j) * M + p] = cmul(ebar[w], make_double2(f1 * h.x + a.x, f1 * h.y + a.y));
  };
  if (s.S > 1) {
    // the cluster's partial sums: each CTA parks its own where G was, then adds a share of the
    // entries over all of them
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    __syncthreads();
#pragma unroll
    for (int u = 0; u < U2; ++u) {
      const int id = warp * U2 + u;
      if (id >= ntile) break;
      double2* d = sG + ((id % s.RT) * 8 + g) * s.ldg + (id / s.RT) * 8 + 2 * t;
      d[0] = acc[u][0];
      d[1] = acc[u][1];
    }
    cl.sync();
    for (int e = rank * kVjThreads + tid; e < s.R * M; e += s.S * kVjThreads) {
      const int r = e / M, p = e - r * M;
      double2 a = make_double2(0.0, 0.0);
      for (int q = 0; q < s.S; ++q) a = cadd(a, *cl.map_shared_rank(sG + r * s.ldg + p, q));
      finish(r, p, a);
    }
    cl.sync();  // nobody leaves while its sums are being read
    return;
  }
#pragma unroll
  for (int u = 0; u < U2; ++u) {
    const int id = warp * U2 + u;
    if (id >= ntile) break;
    const int r = (id % s.RT) * 8 + g, p = (id / s.RT) * 8 + 2 * t;
    if (r < s.R) {
      if (p < M) finish(r, p, acc[u][0]);
      if (p + 1 < M) finish(r, p + 1, acc[u][1]);
    }
  }
}

template <int U2>
static cudaError_t launch_vjp_mma(const double* rchol, const double2* ghalf, const double2* rh1, const double2* xv,
                                  const double2* ebar, int W, int X, int M, int N, double f1, double fc2, double fx2,
                                  const VjpShape& s, double2* gbar, cudaStream_t st) {
  auto k = energy_vjp_mma_kernel<U2>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
  if (e != cudaSuccess) return e;
  const int vec = (M % 2 == 0 && reinterpret_cast<uintptr_t>(rchol) % 16 == 0) ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((W + s.WB - 1) / s.WB * s.S));
  cfg.blockDim = dim3(kVjThreads);
  cfg.dynamicSmemBytes = s.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)s.S;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, k, rchol, ghalf, rh1, xv, ebar, W, X, M, N, f1, fc2, fx2, s, vec, gbar);
  if (e != cudaSuccess) return e;
  note_launch();
  return cudaGetLastError();
}

// Blocks the tensor-core kernel does not take (M > 256, whose G and L_x do not fit shared memory
// together, or N > 32, more row tiles than a warp holds at large M): one CTA per walker runs the sum over x with L_x, G and T_x in shared memory and the
// accumulator (N M complex) in registers, 16 entries per thread at most.
constexpr int kVjpThreads = 512;
constexpr int kVjpPer = 16;  // N * M <= 8192
__global__ void __launch_bounds__(kVjpThreads, 1)
    energy_vjp_kernel(const double* __restrict__ rchol, const double2* __restrict__ ghalf,
                      const double2* __restrict__ rh1, const double2* __restrict__ xv, const double2* __restrict__ ebar,
                      int X, int M, int N, double f1, double fc2, double fx2, double2* __restrict__ gbar) {
  extern __shared__ __align__(16) double vjp_smem[];
  const int NM = N * M, w = blockIdx.x;
  double2* g = reinterpret_cast<double2*>(vjp_smem);  // (N, M)
  double2* t = g + NM;                                // (N, N)
  double* l = reinterpret_cast<double*>(t + N * N);   // (N, M), last: N M may be odd
  const double2* gw = ghalf + (size_t)w * NM;
  for (int e = threadIdx.x; e < NM; e += kVjpThreads) g[e] = gw[e];
  double2 acc[kVjpPer];
#pragma unroll
  for (int r = 0; r < kVjpPer; ++r) acc[r] = make_double2(0.0, 0.0);
  for (int x = 0; x < X; ++x) {
    __syncthreads();  // the previous L_x and T_x are consumed
    const double* lx = rchol + (size_t)x * NM;
    for (int e = threadIdx.x; e < NM; e += kVjpThreads) l[e] = lx[e];
    __syncthreads();
    for (int q = threadIdx.x; q < N * N; q += kVjpThreads) {
      const int j = q / N, i = q - j * N;
      double2 s = make_double2(0.0, 0.0);
      for (int p = 0; p < M; ++p) {
        const double a = l[j * M + p];
        const double2 b = g[i * M + p];
        s.x += a * b.x;
        s.y += a * b.y;
      }
      t[q] = s;
    }
    __syncthreads();
    const double2 c = xv[(size_t)w * X + x];
#pragma unroll
    for (int r = 0; r < kVjpPer; ++r) {
      const int e = threadIdx.x + r * kVjpThreads;
      if (e < NM) {
        const int j = e / M, p = e - j * M;
        double2 s = make_double2(0.0, 0.0);
        for (int i = 0; i < N; ++i) {
          const double2 tj = t[j * N + i];
          const double li = l[i * M + p];
          s.x += tj.x * li;
          s.y += tj.y * li;
        }
        const double lv = l[e];
        acc[r].x += fc2 * c.x * lv - fx2 * s.x;
        acc[r].y += fc2 * c.y * lv - fx2 * s.y;
      }
    }
  }
  const double2 eb = ebar[w];
#pragma unroll
  for (int r = 0; r < kVjpPer; ++r) {
    const int e = threadIdx.x + r * kVjpThreads;
    if (e < NM) {
      const double2 h = rh1[e];
      const double2 d = make_double2(f1 * h.x + acc[r].x, f1 * h.y + acc[r].y);
      gbar[(size_t)w * NM + e] = cmul(eb, d);
    }
  }
}

cudaError_t launch_energy_vjp(const double* rchol, const double2* ghalf, const double2* rh1, const double2* xv,
                              const double2* ebar, int W, int X, int M, int N, double f1, double fc, double fx,
                              double2* gbar, cudaStream_t st) {
  const int NM = N * M;
  if (NM > kVjpPer * kVjpThreads || W <= 0 || X <= 0) return cudaErrorInvalidValue;
  VjpShape s;
  if (vjp_shape(W, X, M, N, s)) {
    const double fc2 = 2.0 * fc, fx2 = 2.0 * fx;
    if (s.units <= 2) return launch_vjp_mma<2>(rchol, ghalf, rh1, xv, ebar, W, X, M, N, f1, fc2, fx2, s, gbar, st);
    if (s.units <= 4) return launch_vjp_mma<4>(rchol, ghalf, rh1, xv, ebar, W, X, M, N, f1, fc2, fx2, s, gbar, st);
    if (s.units <= 6) return launch_vjp_mma<6>(rchol, ghalf, rh1, xv, ebar, W, X, M, N, f1, fc2, fx2, s, gbar, st);
    return launch_vjp_mma<8>(rchol, ghalf, rh1, xv, ebar, W, X, M, N, f1, fc2, fx2, s, gbar, st);
  }
  const size_t smem = (size_t)NM * 24 + (size_t)N * N * 16;
  if (smem > 232448) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(energy_vjp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  energy_vjp_kernel<<<W, kVjpThreads, smem, st>>>(rchol, ghalf, rh1, xv, ebar, X, M, N, f1, 2.0 * fc, 2.0 * fx,
                                                  gbar);
  note_launch();
  return cudaGetLastError();
}

}  // namespace ipie_b200

using namespace ipie_b200;

extern "C" int ipie_b200_onebody_adjoint(int W, int M, int na, int nb, const void* ghalfa, const void* ghalfb,
                                         const void* psia_conj, const void* psib_conj, const double* coeff, void* work,
                                         void* rdm, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  double2* acc = reinterpret_cast<double2*>(work);
  double2* out = reinterpret_cast<double2*>(rdm);
  const void* g[2] = {ghalfa, ghalfb};
  const void* p[2] = {psia_conj, psib_conj};
  const int n[2] = {na, nb};
  for (int s = 0; s < 2; ++s) {
    double2* o = out + (size_t)s * M * M;
    if (n[s] == 0) {
      cudaMemsetAsync(o, 0, sizeof(double2) * M * M, st);
      continue;
    }
    const int K = n[s] * M;
    weighted_walker_sum_kernel<<<(K + 255) / 256, 256, 0, st>>>(reinterpret_cast<const double2*>(g[s]), coeff, W, K,
                                                                 acc);
    note_launch();
    expand_half_kernel<<<dim3((M + 127) / 128, M), 128, 0, st>>>(reinterpret_cast<const double2*>(p[s]), acc, M, n[s],
                                                                  o, 0);
    note_launch();
  }
  return (int)cudaGetLastError();
}

extern "C" int ipie_b200_rotate_onebody(const void* psi_conj, const double* h1, int M, int N, void* rh1, void* stream) {
  if (N == 0) return 0;
  rotate_onebody_kernel<<<dim3((M + 127) / 128, N), 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const double2*>(psi_conj), h1, M, N, reinterpret_cast<double2*>(rh1));
  note_launch();
  return (int)cudaGetLastError();
}

extern "C" int ipie_b200_local_energy_vjp(int rhf, const double* rchola, const double* rcholb, const void* rH1a,
                                          const void* rH1b, const void* ghalfa, const void* ghalfb, int W, int X,
                                          int M, int na, int nb, const void* ebar, void* work, void* gbara,
                                          void* gbarb, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (W <= 0 || X <= 0 || M <= 0 || na <= 0 || (!rhf && nb < 0)) return (int)cudaErrorInvalidValue;
  double2* xv = reinterpret_cast<double2*>(work);
  const double2* ga = reinterpret_cast<const double2*>(ghalfa);
  const double2* gb = reinterpret_cast<const double2*>(ghalfb);
  const double2* eb = reinterpret_cast<const double2*>(ebar);
  // the factors of ipie_b200_local_energy_single_det_batch: UHF f1 = 1, fc = 1/2, fx = 1/2;
  // RHF (alpha only, doubled) f1 = 2, fc = 2, fx = 1
  const double f1 = rhf ? 2.0 : 1.0, fc = rhf ? 2.0 : 0.5, fx = rhf ? 1.0 : 0.5;
  const bool alias = !rhf && nb == na && rcholb == rchola && ghalfb == ghalfa;
  const bool use_b = !rhf && nb > 0;
  // X_x = sum over the spins in the energy of L_s,x . G_s
  const bool two = use_b && !alias;
  cudaError_t e = launch_force_bias(rchola, ga, na * M, two ? rcholb : nullptr, gb, nb * M, W, X, xv, st,
                                    alias ? 2.0 : 1.0);
  if (e == cudaSuccess)
    e = launch_energy_vjp(rchola, ga, reinterpret_cast<const double2*>(rH1a), xv, eb, W, X, M, na, f1, fc, fx,
                          reinterpret_cast<double2*>(gbara), st);
  if (e != cudaSuccess || !use_b) return (int)e;
  if (alias) {
    if (gbarb != gbara)
      e = cudaMemcpyAsync(gbarb, gbara, (size_t)W * na * M * sizeof(double2), cudaMemcpyDeviceToDevice, st);
    return (int)e;
  }
  return (int)launch_energy_vjp(rcholb, gb, reinterpret_cast<const double2*>(rH1b), xv, eb, W, X, M, nb, f1, fc, fx,
                                reinterpret_cast<double2*>(gbarb), st);
}
