// GEMM-shaped stages of the FP64 walker step on the f64 tensor cores
// (DMMA): force bias, VHS assembly, one-body propagation, the Taylor series
// of exp(VHS), and the fused exchange energy.
#include "../../include/ipie_b200_testing.h"
#include "gemm_f64.cuh"
#include "gemm_rc.cuh"
#include "kernels.h"

namespace ipie_b200 {

// Batched per-walker GEMMs: 64-row tile; the column tile follows 2N.
using CfgW64 = TileCfg<64, 64, 16, 2, 4>;
using CfgW32 = TileCfg<64, 32, 16, 4, 2>;
using CfgW16 = TileCfg<64, 16, 16, 4, 2>;

// ---------------------------------------------------------------------------
// Force bias: vbias[w][x] = scale sum_s sum_k rchol_s[x][k] Ghalf_s[w][k]  (rchol real), both spin
// blocks in one launch.
// ---------------------------------------------------------------------------
struct EpiVbias {
  double2* v;
  int ld, xoff;
  int accumulate;
  double scale;  // 2 for spin-aliased walkers: exactly t + t
  __device__ __forceinline__ void operator()(int x, int w, double2 c) const {
    const size_t idx = (size_t)w * ld + xoff + x;
    double2 r = cscale(c, scale);
    if (accumulate) r = cadd(r, v[idx]);
    v[idx] = r;
  }
};

cudaError_t launch_force_bias(const double* rchola, const double2* ghalfa, int Ka, const double* rcholb,
                              const double2* ghalfb, int Kb, int W, int X, double2* vbias, cudaStream_t st,
                              double scale) {
  const RcSegment seg[2] = {{rchola, ghalfa, Ka, 0}, {rcholb, ghalfb, Kb, 0}};
  return rc_gemm<true, false>(X, W, seg, rcholb != nullptr ? 2 : 1, EpiVbias{vbias, X, 0, 0, scale}, st);
}

// ---------------------------------------------------------------------------
// VHS: VHS_packed[p][w] = sum_x L_packed[p][x] xshifted[x][w], scaled
// by i sqrt(dt) and scattered to both triangles of the symmetric (W, M, M).
// ---------------------------------------------------------------------------
struct EpiVHS {
  double2* vhs;
  const int* ii;
  const int* jj;
  int M;
  double sdt;
  __device__ __forceinline__ void operator()(int p, int w, double2 c) const {
    const double2 val = make_double2(-sdt * c.y, sdt * c.x);
    const int i = ii[p], j = jj[p];
    double2* base = vhs + (size_t)w * M * M;
    base[(size_t)i * M + j] = val;
    base[(size_t)j * M + i] = val;
  }
};

cudaError_t launch_vhs(const double* chol_packed, const int* idx_i, const int* idx_j, int P, int X, int M,
                       const double2* xshifted, int W, double sqrt_dt, double2* vhs, cudaStream_t st) {
  const RcSegment seg{chol_packed, xshifted, X, 0};
  return rc_gemm<false, false>(P, W, &seg, 1, EpiVHS{vhs, idx_i, idx_j, M, sqrt_dt}, st);
}

// ---------------------------------------------------------------------------
// Complex-Cholesky pieces (ipie's GenericComplexChol): a complex operand R = R_re + i R_im enters
// as two segments of one product, the second times i.
//
// Force bias / Coulomb vector: out[w][xoff + x] (+)= sum_k R[x][k] Ghalf[w][k], out rows of `ld` complex.
// ---------------------------------------------------------------------------
cudaError_t launch_force_bias_c(const double* r_re, const double* r_im, const double2* ghalf, int W, int X, int K,
                                double2* out, int ld, int xoff, int accumulate, cudaStream_t st) {
  const RcSegment seg[2] = {{r_re, ghalf, K, 0}, {r_im, ghalf, K, 1}};
  return rc_gemm<true, true>(X, W, seg, 2, EpiVbias{out, ld, xoff, accumulate, 1.0}, st);
}

// VHS of a complex Cholesky: V_w = i sqrt(dt) C . xs_w with C = [A | B] (M*M, F) complex and
// xs (F, W) complex.  Rows p = i M + j of C map to V_w[i][j] directly (no symmetry).
struct EpiVHSFull {
  double2* vhs;
  int M;
  double sdt;
  __device__ __forceinline__ void operator()(int p, int w, double2 c) const {
    vhs[(size_t)w * M * M + p] = make_double2(-sdt * c.y, sdt * c.x);
  }
};

cudaError_t launch_vhs_full(const double* c_re, const double* c_im, int M, int F, const double2* xshifted, int W,
                            double sqrt_dt, double2* vhs, cudaStream_t st) {
  const RcSegment seg[2] = {{c_re, xshifted, F, 0}, {c_im, xshifted, F, 1}};
  return rc_gemm<false, true>(M * M, W, seg, 2, EpiVHSFull{vhs, M, sqrt_dt}, st);
}

// Local energy of the complex-Cholesky form, one CTA per walker:
//   e1b = sum_s Ghalf_s . rH1_s + ecore,  ecoul = 1/2 sum_x X1[x] X2[x],  e2b = ecoul - exx.
__global__ void __launch_bounds__(256) energy_complex_kernel(const double2* __restrict__ ga,
                                                              const double2* __restrict__ gb, int NMa, int NMb,
                                                              const double2* __restrict__ rh1a,
                                                              const double2* __restrict__ rh1b, double ecore,
                                                              const double2* __restrict__ x1,
                                                              const double2* __restrict__ x2, int X,
                                                              const double2* __restrict__ exx,
                                                              double2* __restrict__ energy) {
  __shared__ double2 red[2][8];
  const int w = blockIdx.x, tid = threadIdx.x;
  double2 e1 = make_double2(0.0, 0.0), ec = make_double2(0.0, 0.0);
  for (int k = tid; k < NMa; k += 256) e1 = cadd(e1, cmul(ga[(size_t)w * NMa + k], rh1a[k]));
  for (int k = tid; k < NMb; k += 256) e1 = cadd(e1, cmul(gb[(size_t)w * NMb + k], rh1b[k]));
  for (int x = tid; x < X; x += 256) ec = cadd(ec, cmul(x1[(size_t)w * X + x], x2[(size_t)w * X + x]));
  e1 = warp_sum2(e1);
  ec = warp_sum2(ec);
  if ((tid & 31) == 0) {
    red[0][tid >> 5] = e1;
    red[1][tid >> 5] = ec;
  }
  __syncthreads();
  if (tid == 0) {
    double2 a = make_double2(ecore, 0.0), c = make_double2(0.0, 0.0);
    for (int k = 0; k < 8; ++k) {
      a = cadd(a, red[0][k]);
      c = cadd(c, red[1][k]);
    }
    const double2 e2 = csub(cscale(c, 0.5), exx[w]);
    energy[(size_t)w * 3 + 0] = cadd(a, e2);
    energy[(size_t)w * 3 + 1] = a;
    energy[(size_t)w * 3 + 2] = e2;
  }
}

// out[w] (accumulate: +=) coef * sum_t part[t][w]
__global__ void scaled_row_sum_kernel(const double2* __restrict__ part, int rows, int W, double2 coef,
                                      double2* __restrict__ out, int accumulate) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= W) return;
  double2 acc = make_double2(0.0, 0.0);
  for (int t = 0; t < rows; ++t) acc = cadd(acc, part[(size_t)t * W + w]);
  const double2 r = cmul(coef, acc);
  out[w] = accumulate ? cadd(out[w], r) : r;
}

cudaError_t launch_scaled_row_sum(const double2* part, int rows, int W, double2 coef, double2* out, int accumulate,
                                  cudaStream_t st) {
  scaled_row_sum_kernel<<<(W + 127) / 128, 128, 0, st>>>(part, rows, W, coef, out, accumulate);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_energy_complex(const double2* ga, const double2* gb, int W, int NMa, int NMb, const double2* rh1a,
                                  const double2* rh1b, double ecore, const double2* x1, const double2* x2, int X,
                                  const double2* exx, double2* energy, cudaStream_t st) {
  energy_complex_kernel<<<W, 256, 0, st>>>(ga, gb, NMa, NMb, rh1a, rh1b, ecore, x1, x2, X, exx, energy);
  note_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// One-body: phi_out[w] = expH1 . phi_in[w]; expH1 real (M x M) or complex.
// ---------------------------------------------------------------------------
struct EpiStoreC {
  double2* out;
  long long bs;
  int ld;  // complex row stride
  __device__ __forceinline__ void operator()(int b, int row, int col, double v0, double v1) const {
    out[(size_t)b * bs + (size_t)row * ld + (col >> 1)] = make_double2(v0, v1);
  }
};

template <class C>
static cudaError_t one_body_cfg(const double* expH1, int cplx, const double2* phi_in, double2* phi_out, int W, int M,
                                int N, cudaStream_t st) {
  EpiStoreC epi{phi_out, (long long)M * N, N};
  if (!cplx) {
    LoadRowK<C, C::BM> la{expH1, 0, M};
    LoadRowR<C, C::BN> lb{reinterpret_cast<const double*>(phi_in), 2LL * M * N, 2LL * N};
    return launch_dmma_gemm<C>(M, 2 * N, M, W, la, lb, epi, st);
  }
  LoadRowK<C, C::BM> la{expH1, 0, 2LL * M};
  LoadCplxEmbed<C, C::BN> lb{phi_in, (long long)M * N, N};
  return launch_dmma_gemm<C>(M, 2 * N, 2 * M, W, la, lb, epi, st);
}

cudaError_t launch_one_body(const double* expH1, int cplx, const double2* phi_in, double2* phi_out, int W, int M, int N,
                            cudaStream_t st) {
  if (2 * N > 32) return one_body_cfg<CfgW64>(expH1, cplx, phi_in, phi_out, W, M, N, st);
  if (2 * N > 16) return one_body_cfg<CfgW32>(expH1, cplx, phi_in, phi_out, W, M, N, st);
  return one_body_cfg<CfgW16>(expH1, cplx, phi_in, phi_out, W, M, N, st);
}

// ---------------------------------------------------------------------------
// Taylor series of exp(VHS) applied to phi:
//   T_0 = phi_in;  T_n = VHS T_{n-1} / n;  phi_out = phi_in + sum_{n=1..nmax} T_n
// One batched complex GEMM per term (VHS complex natural layout as the left
// operand, T embedded 2x2 as the right operand), phi_out updated in the
// epilogue.  t0/t1 are ping-pong buffers of the size of phi.
// ---------------------------------------------------------------------------
struct EpiTaylor {
  double2* tout;
  const double2* phi_in;
  double2* phi_out;
  long long bs;
  int ld;
  double inv_n;
  int first;
  __device__ __forceinline__ void operator()(int b, int row, int col, double v0, double v1) const {
    const size_t idx = (size_t)b * bs + (size_t)row * ld + (col >> 1);
    const double2 t = make_double2(v0 * inv_n, v1 * inv_n);
    if (tout) tout[idx] = t;
    const double2 base = first ? phi_in[idx] : phi_out[idx];
    phi_out[idx] = cadd(base, t);
  }
};

template <class C>
static cudaError_t taylor_cfg(const double2* vhs, const double2* phi_in, double2* phi_out, double2* t0, double2* t1,
                              int W, int M, int N, int nmax, cudaStream_t st) {
  const double2* src = phi_in;
  double2* bufs[2] = {t0, t1};
  for (int n = 1; n <= nmax; ++n) {
    double2* dst = (n == nmax) ? nullptr : bufs[n & 1];
    LoadRowK<C, C::BM> la{reinterpret_cast<const double*>(vhs), 2LL * M * M, 2LL * M};
    LoadCplxEmbed<C, C::BN> lb{src, (long long)M * N, N};
    EpiTaylor epi{dst, phi_in, phi_out, (long long)M * N, N, 1.0 / n, n == 1};
    cudaError_t e = launch_dmma_gemm<C>(M, 2 * N, 2 * M, W, la, lb, epi, st);
    if (e != cudaSuccess) return e;
    src = dst;
  }
  return cudaSuccess;
}

cudaError_t launch_taylor(const double2* vhs, const double2* phi_in, double2* phi_out, double2* t0, double2* t1, int W,
                          int M, int N, int nmax, cudaStream_t st) {
  if (nmax < 1) return cudaErrorInvalidValue;
  if (2 * N > 32) return taylor_cfg<CfgW64>(vhs, phi_in, phi_out, t0, t1, W, M, N, nmax, st);
  if (2 * N > 16) return taylor_cfg<CfgW32>(vhs, phi_in, phi_out, t0, t1, W, M, N, nmax, st);
  return taylor_cfg<CfgW16>(vhs, phi_in, phi_out, t0, t1, W, M, N, nmax, st);
}

// ---------------------------------------------------------------------------
// Fused exchange:  raw_w = sum_x sum_ij T_ij T_ji,  T = rchol_x (N x M) Ghalf_w^T.
// One product of the stacked rows (x, i) of rchol with the stacked columns (w, j) of Ghalf, K = M.
// A tile takes as many whole vectors x and walkers w as fit its BM rows and BN columns, so no row or
// column is spent on rounding N up (N = 10 in 16 x 16 blocks did 2.6 times the work); the tile shape
// is the one of two that N fills better.  The epilogue parks T in shared memory and sums each
// walker's products over x and the unordered pairs (i, j) into one partial per (tile row, walker); T
// never reaches global memory.  Its terms are dealt to the lanes one by one, with the places of T_ij
// and T_ji from a table: a warp per (x, w) block left it 512 blocks in a row with one lane at work at N = 1
// (31 walkers, M = 20, X = 150: 167 -> 7.9 us; 64, M = 26, X = 120, N = 5: 13.5 -> 7.5 us) and divided by N
// for every term.  At 2 CTAs per SM one's epilogue runs under the other's products.
// UHF, 640 walkers, M = 108, N = 15, X = 600, one spin: 1.99 -> 1.56 ms (37.3 GFLOP: 24
// TFLOP/s, 27 with the padding of 15 to 120 / 8 rows); 512 walkers, M = 76, N = 10, X = 400: 0.77 -> 0.30 ms,
// against N rounded up to 8, 16 or 32.
// ---------------------------------------------------------------------------
using ExWide = RcCfg<128, 32, 4, 2, 2>;
using ExTall = RcCfg<96, 48, 4, 2, 2>;

template <class C>
__global__ void __launch_bounds__(C::THREADS, C::OCC)
    exchange_kernel(const __grid_constant__ RcOperands op, int W, int X, int N, int XB, int WB, int rows,
                    double2* __restrict__ part) {
  extern __shared__ __align__(16) double rc_sm[];
  constexpr int LDC = C::BN + 2;  // T_ij at stride LDC + 1 over i: odd, conflict-free
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wm0 = (warp / C::WARPS_N) * C::WTM, wn0 = (warp % C::WARPS_N) * C::WTN;
  const int x0 = (int)blockIdx.y * XB, w0 = (int)blockIdx.x * WB;
  constexpr int NW = C::THREADS / 32, MAXN = 32;
  __shared__ double2 red[C::BN][NW];
  // unordered pairs of {0 .. N-1} as (i, i + d mod N), d = 0 .. N/2 (half of the last d when N is
  // even): the places of T_ij and T_ji within a block
  __shared__ unsigned place[MAXN * (MAXN + 1) / 2];
  const int pairs = N * (N + 1) / 2;
  for (int e = tid; e < pairs; e += C::THREADS) {
    const int d = e / N, i = e - d * N, j = i + d < N ? i + d : i + d - N;
    place[e] = (unsigned)(i * LDC + j) | (unsigned)(j * LDC + i) << 16;
  }
  for (int e = tid; e < WB * NW; e += C::THREADS) red[e / NW][e % NW] = make_double2(0.0, 0.0);
  RcAcc<C> acc;
  rc_mainloop<C, true, false>(X * N, W * N, x0 * N, w0 * N, op, 0, op.chunks, rc_sm, acc);
  cp_async_wait<0>();
  __syncthreads();
  double2* sT = reinterpret_cast<double2*>(rc_sm);
#pragma unroll
  for (int i = 0; i < C::FM; ++i)
#pragma unroll
    for (int j = 0; j < C::FN; ++j) {
      double2* d = sT + (wm0 + 8 * i + g) * LDC + wn0 + 8 * j + 2 * t;
      d[0] = make_double2(acc.re[i][j][0], acc.im[i][j][0]);
      d[1] = make_double2(acc.re[i][j][1], acc.im[i][j][1]);
    }
  __syncthreads();
  // The (x, pair) terms of the tile, walker by walker, in equal shares per warp: the lanes take
  // consecutive terms, whatever N is, and a warp reduces once per walker it meets.
  const int xn = min(XB, X - x0), wn = min(WB, W - w0), terms = xn * pairs;
  const int dx = 32 / pairs, dp = 32 - dx * pairs;
  int e0 = wn * terms * warp / NW;
  const int e1 = wn * terms * (warp + 1) / NW;
  int wl = e0 / terms, q = e0 - wl * terms;
  while (e0 < e1) {
    const int qe = min(terms, q + e1 - e0);
    const int first = q + lane;
    int xl = first / pairs, p = first - xl * pairs;
    double2 s = make_double2(0.0, 0.0);
    for (int e = first; e < qe; e += 32) {
      const double2* blk = sT + xl * N * LDC + wl * N;
      const unsigned ij = place[p];
      const double2 v = cmul(blk[ij & 0xffffu], blk[ij >> 16]);
      const double f = p < N ? 1.0 : 2.0;
      s.x += f * v.x;
      s.y += f * v.y;
      xl += dx;
      p += dp;
      if (p >= pairs) {
        p -= pairs;
        ++xl;
      }
    }
    s = warp_sum2(s);
    if (lane == 0) red[wl][warp] = s;
    e0 += qe - q;
    q = 0;
    ++wl;
  }
  __syncthreads();
  if (tid < wn) {
    double2 v = red[tid][0];
#pragma unroll
    for (int q = 1; q < NW; ++q) v = cadd(v, red[tid][q]);
    part[(size_t)blockIdx.y * W + w0 + tid] = v;
  }
  if (blockIdx.y == gridDim.y - 1)
    for (int e = tid; e < (rows - (int)gridDim.y) * wn; e += C::THREADS)
      part[(size_t)((int)gridDim.y + e / wn) * W + w0 + e % wn] = make_double2(0.0, 0.0);
}

template <class C>
static cudaError_t exchange_cfg(const double* rchol, const double2* ghalf, int W, int X, int M, int N, int rows,
                                double2* part, cudaStream_t st) {
  const int XB = C::BM / N, WB = C::BN / N;
  const size_t need = sizeof(double2) * C::BM * (C::BN + 2), smem = need > C::SMEM ? need : C::SMEM;
  auto kern = exchange_kernel<C>;
  cudaError_t e = set_smem(kern, smem);
  if (e != cudaSuccess) return e;
  RcOperands op = {};
  op.seg[0] = RcSegment{rchol, ghalf, M, 0};
  op.nseg = 1;
  op.chunks = (M + kRcBK - 1) / kRcBK;
  op.vec_a = M % 2 == 0 && reinterpret_cast<uintptr_t>(rchol) % 16 == 0;
  op.vec_b = reinterpret_cast<uintptr_t>(ghalf) % 16 == 0;
  kern<<<dim3((W + WB - 1) / WB, (X + XB - 1) / XB), C::THREADS, smem, st>>>(op, W, X, N, XB, WB, rows, part);
  note_launch();
  return cudaGetLastError();
}

// Partial rows that callers provide and sum: one per 128 rows of N rounded up to 8, 16 or 32 (the last
// row tile zeroes those that packing leaves over).
static int exchange_row_vectors(int N) { return 128 / (N <= 8 ? 8 : N <= 16 ? 16 : 32); }

// The shape whose rows and columns N fills better, among those that need no more partial rows.
static bool exchange_tall(int N) {
  if (ExTall::BM / N < exchange_row_vectors(N)) return false;
  const int wide = (ExWide::BM / N * N) * (ExWide::BN / N * N) * (ExTall::BM * ExTall::BN);
  const int tall = (ExTall::BM / N * N) * (ExTall::BN / N * N) * (ExWide::BM * ExWide::BN);
  return tall > wide;
}

cudaError_t launch_exchange(const double* rchol, const double2* ghalf, int W, int X, int M, int N, double2* part,
                            int* ntiles, cudaStream_t st) {
  if (N <= 0) {
    *ntiles = 0;
    return cudaSuccess;
  }
  if (N > 32) return cudaErrorInvalidValue;
  const int vectors = exchange_row_vectors(N);
  *ntiles = (X + vectors - 1) / vectors;
  if (part == nullptr) return cudaSuccess;
  return exchange_tall(N) ? exchange_cfg<ExTall>(rchol, ghalf, W, X, M, N, *ntiles, part, st)
                          : exchange_cfg<ExWide>(rchol, ghalf, W, X, M, N, *ntiles, part, st);
}

}  // namespace ipie_b200

extern "C" int ipie_b200_rc_plan_test(int M, int N, int chunks, int* tile, int* split) {
  const ipie_b200::RcPlan p = ipie_b200::rc_plan(M, N, chunks);
  *tile = p.tile;
  *split = p.S;
  return 0;
}
