// Green's function, overlap and reorthogonalisation for spin blocks of N <= 32 electrons: one CTA of
// 96 or 128 threads per walker and distinct spin block, four per SM, on the f64 tensor cores.
// ovlp_w = prod_s phase_s * exp(sum_s log|det O_s| - log_shift_w).
// Same contracts as gf_overlap_kernel and reortho_kernel (walkers.cu), which keep N > 32.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace ipie_b200 {

namespace {

constexpr int kChunk = 8;  // rows of phi / psi* per shared-memory chunk of the overlap and Gram products

// ---------------------------------------------------------------------------------------------
// The Green's function on the f64 tensor cores, N padded to NT tiles of 8.  Per walker and spin:
//   O = phi^T psi*: chunks of 8 rows of phi and psi* through a three-deep cp.async ring; warp w
//       owns row tile w of O (NT = 1: a quarter of the rows m, NT = 2: one of the four tiles).
//   O^-1 by Gauss-Jordan elimination in place, partial pivoting on |.|, in panels of 8 columns: one
//       warp factors the panel with a row per lane and the 8 columns in registers (the pivot by one
//       redux.sync on the high word of |a|^2 above the row index, so one within 2^-15 of the largest
//       |a|^2; its row by shuffles; pivots stay in their rows), then all warps apply it to the other
//       columns as one rank-8 MMA update
//         A[:, J] <- A[:, J] (pivot rows zeroed) + panel' A[pivot rows, J].
//       So a column costs no barrier and a panel three, where the column by column form took two
//       per column.
//       The halves of a complex product are summed apart, here and in O, and an entry takes a panel's
//       products in one addition: Ghalf 4.3e-16 and the overlap 1.6e-15 off at M = 200, N = 32, complex trial
//       (6.9e-16 and 3.5e-15 with every product added to the entries in turn).
//   With p_k the pivot row of column k the stored array B holds O^-1[k, p_j] = B[p_k, j].
//   Ghalf[i, m] = sum_c O^-1[i, c] phi[m, c]: warp w keeps its rows of O^-1 as MMA fragments in
//       registers (gathered through p once) while chunks of 16 rows of phi pass through the ring.
//       The eight rows m of a tile are dealt to the MMA's columns as 0 4 1 5 2 6 3 7, so that four
//       lanes store four neighbouring entries of Ghalf; rows of an odd stride keep the fragment
//       loads free of bank conflicts.
// The floor is the f64 tensor pipe's time for the two products (28k cycles per SM and walker at
// M = 200, N = 32).  2048 walkers, M = 200, N = 32: 535 -> 324 us; 512, M = 76, N = 10: 46 -> 19 us; 777, M =
// 149, N = 23 + 17: 280 -> 175 us (against DFMA products and the column by column elimination), and 175 ->
// 151 us with a CTA per spin instead of both in one (640, M = 108, N = 15 + 15: 89 -> 72 us): the pivot chains of
// the two spins run side by side and the last round of CTAs is shorter (144 us with the sums above).
template <int NT>
struct GfShape {
  static constexpr int WARPS = NT == 3 ? 3 : 4, THREADS = 32 * WARPS, NP = 8 * NT;
  static constexpr int LDO = NP + 4;   // O (MMA left operand: 4 mod 8)
  static constexpr int LDP = 12;       // panel
  static constexpr int LDC = NP + 2;   // chunks of the O product (2 mod 8)
  static constexpr int LDG = NP + 1;   // chunks of the Ghalf product (odd)
  static constexpr int GM = 16;        // rows of phi per Ghalf chunk
  static constexpr int RING = 3;
  static constexpr int OSTAGE = 2 * kChunk * LDC, GSTAGE = GM * LDG;
  static constexpr int STAGE = RING * (OSTAGE > GSTAGE ? OSTAGE : GSTAGE);
  static constexpr int MW = WARPS / NT;  // warps sharing a row tile in the Ghalf product
  static_assert(STAGE >= 4 * 64, "partial sums of the split O product fit the ring");
};

template <int NT>
struct GfShared {
  using S = GfShape<NT>;
  double2 O[S::NP * S::LDO];
  double2 P[S::NP * S::LDP];
  double2 stage[S::STAGE];
  double2 piv[32];
  double2 red[4];
  int perm[32], inv[32];
  unsigned used;
};

template <int NT>
__device__ __forceinline__ void gf_overlap_tiles(const double2* __restrict__ phi, const double2* __restrict__ psic,
                                                 int M, int N, GfShared<NT>& sm) {
  using S = GfShape<NT>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nch = (M + kChunk - 1) / kChunk;
  auto issue = [&](int ch) {
    if (ch < nch) {
      double2* st = sm.stage + (ch % S::RING) * S::OSTAGE;
      for (int e = tid; e < kChunk * S::NP; e += S::THREADS) {
        const int r = e / S::NP, c = e % S::NP, m = ch * kChunk + r;
        const bool in = m < M && c < N;
        const size_t off = in ? (size_t)m * N + c : 0;
        cp_async16(st + r * S::LDC + c, phi + off, in ? 16 : 0);
        cp_async16(st + (kChunk + r) * S::LDC + c, psic + off, in ? 16 : 0);
      }
    }
    cp_async_commit();  // (an empty group past the end keeps the group count per chunk)
  };
  constexpr int CT = NT >= 3 ? NT : 1;  // column tiles per warp
  const int rt = NT >= 3 ? warp : NT == 2 ? (warp & 1) : 0, ct0 = NT == 2 ? (warp >> 1) : 0;
  // (the halves of a complex product in chains of their own: one chain of 2 M terms rounds more)
  double re[CT][2], im[CT][2], re2[CT][2], im2[CT][2];
#pragma unroll
  for (int j = 0; j < CT; ++j)
    re[j][0] = re[j][1] = im[j][0] = im[j][1] = re2[j][0] = re2[j][1] = im2[j][0] = im2[j][1] = 0.0;
  issue(0);
  issue(1);
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<1>();
    __syncthreads();
    issue(ch + 2);
    // NT = 1: the warps take turns at the 4-row steps
    if (NT == 1 && (ch >> 1) % 2 != (warp >> 1)) continue;
    const double2* a = sm.stage + (ch % S::RING) * S::OSTAGE + t * S::LDC + rt * 8 + g;
    const double2* b = sm.stage + (ch % S::RING) * S::OSTAGE + (kChunk + t) * S::LDC + ct0 * 8 + g;
#pragma unroll
    for (int kk = 0; kk < kChunk; kk += 4) {
      if (NT == 1 && (kk >> 2) != (warp & 1)) continue;
      const double2 av = a[kk * S::LDC];
#pragma unroll
      for (int j = 0; j < CT; ++j) {
        const double2 bv = b[kk * S::LDC + 8 * j];
        dmma884(re[j], av.x, bv.x);
        dmma884(im[j], av.x, bv.y);
        dmma884(re2[j], -av.y, bv.y);
        dmma884(im2[j], av.y, bv.x);
      }
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int j = 0; j < CT; ++j)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      re[j][q] += re2[j][q];
      im[j][q] += im2[j][q];
    }
  if (NT == 1) {
    __syncthreads();  // the ring is free: the four partial tiles
    double2* part = sm.stage + warp * 64 + g * 8 + 2 * t;
    part[0] = make_double2(re[0][0], im[0][0]);
    part[1] = make_double2(re[0][1], im[0][1]);
    __syncthreads();
    if (tid < 64) {
      double2 v = sm.stage[tid];
      for (int q = 1; q < 4; ++q) v = cadd(v, sm.stage[q * 64 + tid]);
      sm.O[(tid >> 3) * S::LDO + (tid & 7)] = v;
    }
  } else {
#pragma unroll
    for (int j = 0; j < CT; ++j)
#pragma unroll
      for (int q = 0; q < 2; ++q)
        sm.O[(rt * 8 + g) * S::LDO + (ct0 + j) * 8 + 2 * t + q] = make_double2(re[j][q], im[j][q]);
  }
}

__device__ __forceinline__ double2 shfl2(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// Gauss-Jordan inverse of the N x N block in sm.O (see above); sm.perm, sm.inv, sm.piv.
template <int NT>
__device__ __forceinline__ void gf_invert(int N, GfShared<NT>& sm, unsigned* status) {
  using S = GfShape<NT>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  if (tid < 32) {
    sm.perm[tid] = sm.inv[tid] = tid;
    if (tid == 0) sm.used = 0u;
  }
  __syncthreads();
#pragma unroll 1
  for (int kb = 0; kb < NT; ++kb) {
    if (warp == kb % S::WARPS) {
      double2 a[8];
      const int row = lane < S::NP ? lane : 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = sm.O[row * S::LDO + 8 * kb + j];
      unsigned used = sm.used;
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        const int k = 8 * kb + jj;
        if (k < N) {
          unsigned key = 0u;
          const double2 own = a[jj];
          if (lane < N && !((used >> lane) & 1u))
            key = ((unsigned)__double2hiint(cabs2(own)) & ~31u) | (unsigned)(31 - lane);
          // every lane scales its row as if it held the pivot, while the pivot is found
          const double rn = __drcp_rn(own.x * own.x + own.y * own.y);
          const double2 pinv = make_double2(own.x * rn, -own.y * rn);
          double2 s[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] = j == jj ? pinv : cmul(a[j], pinv);
          key = __reduce_max_sync(0xffffffffu, key);
          int p = 31 - (int)(key & 31u);
          if (key < 32u) {
            // every free |a|^2 is zero (an exactly singular block, or |a| below 1e-154): any free row.  A
            // NaN has a large key and is taken.
            p = __ffs(~used) - 1;
          }
          const bool mine = lane == p;
          if (mine) {
            if (own.x == 0.0 && own.y == 0.0) flag(status, STATUS_SINGULAR);
            sm.piv[k] = own;
            sm.perm[k] = lane;
            sm.inv[lane] = k;
          }
          used |= 1u << p;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const double2 r = shfl2(s[j], p);
            if (mine) {
              a[j] = s[j];
            } else if (j == jj) {
              const double2 v = cmul(own, r);
              a[j] = make_double2(-v.x, -v.y);
            } else {
              a[j] = csub(a[j], cmul(own, r));
            }
          }
        }
      }
      if (lane < S::NP) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          sm.P[lane * S::LDP + j] = a[j];
          sm.O[lane * S::LDO + 8 * kb + j] = a[j];
        }
      }
      if (lane == 0) sm.used = used;
    }
    if (NT == 1) break;
    __syncthreads();
    // rank-8 update of the other columns.  Row tile rt, column tiles ct0, ct0 + 1, ... but kb
    constexpr int CT = NT >= 3 ? NT : 1;
    const int rt = NT >= 3 ? warp : (warp & 1), ct0 = NT == 2 ? (warp >> 1) : 0;
    double2 b[CT][2];  // pivot rows of the columns, before anyone rewrites them
#pragma unroll
    for (int j = 0; j < CT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) b[j][h] = sm.O[sm.perm[8 * kb + 4 * h + t] * S::LDO + 8 * (ct0 + j) + g];
    const int row = rt * 8 + g;
    bool pivot = false;
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) pivot |= sm.perm[8 * kb + jj] == row;
    const double2 a0 = sm.P[row * S::LDP + t], a1 = sm.P[row * S::LDP + 4 + t];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < CT; ++j) {
      if (ct0 + j == kb) continue;
      // the products summed by themselves, their halves apart: small beside the entries they change, so
      // that an entry is rounded once a panel and not with every term
      double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0}, re2[2] = {0.0, 0.0}, im2[2] = {0.0, 0.0};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double2 a = h == 0 ? a0 : a1;
        dmma884(re, a.x, b[j][h].x);
        dmma884(im, a.x, b[j][h].y);
        dmma884(re2, -a.y, b[j][h].y);
        dmma884(im2, a.y, b[j][h].x);
      }
      double2* c = sm.O + row * S::LDO + 8 * (ct0 + j) + 2 * t;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const double2 v = make_double2(re[q] + re2[q], im[q] + im2[q]);
        c[q] = pivot ? v : cadd(c[q], v);
      }
    }
    __syncthreads();
  }
  __syncthreads();
}

// log|det O| and its phase from the pivots and the parity of the pivot order, by warp 0:
// sm.red[0].x, sm.red[1].
template <int NT>
__device__ __forceinline__ void gf_determinant(int N, GfShared<NT>& sm) {
  const int lane = threadIdx.x;
  if (lane >= 32) return;
  double la = 0.0;
  double2 ph = make_double2(1.0, 0.0);
  const int p = sm.perm[lane];
  int inversions = 0;
#pragma unroll 8
  for (int j = 1; j < 8 * NT; ++j) inversions += (j > lane && sm.perm[j] < p) ? 1 : 0;
  if (lane < N) {
    const double2 u = sm.piv[lane];
    const double a = cabs_(u);
    la = log(a);
    ph = make_double2(u.x / a, u.y / a);
    if (inversions & 1) ph = make_double2(-ph.x, -ph.y);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    la += __shfl_xor_sync(0xffffffffu, la, o);
    ph = cmul(ph, make_double2(__shfl_xor_sync(0xffffffffu, ph.x, o), __shfl_xor_sync(0xffffffffu, ph.y, o)));
  }
  if (lane == 0) {
    sm.red[0] = make_double2(la, 0.0);
    sm.red[1] = ph;
  }
}

template <int NT>
__device__ __forceinline__ void gf_ghalf(const double2* __restrict__ phi, int M, int N, GfShared<NT>& sm,
                                         double2* __restrict__ ghalf, double2* __restrict__ ghalf2) {
  using S = GfShape<NT>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nch = (M + S::GM - 1) / S::GM;
  auto issue = [&](int ch) {
    if (ch < nch) {
      double2* st = sm.stage + (ch % S::RING) * S::GSTAGE;
      for (int e = tid; e < S::GM * S::NP; e += S::THREADS) {
        const int r = e / S::NP, c = e % S::NP, m = ch * S::GM + r;
        const bool in = m < M && c < N;
        cp_async16(st + r * S::LDG + c, phi + (in ? (size_t)m * N + c : 0), in ? 16 : 0);
      }
    }
    cp_async_commit();
  };
  issue(0);
  issue(1);
  const int rt = warp % NT, mw = warp / NT, i = rt * 8 + g;
  double2 a[2 * NT];
#pragma unroll
  for (int k = 0; k < 2 * NT; ++k) a[k] = sm.O[sm.perm[i] * S::LDO + sm.inv[4 * k + t]];
  const int col = 4 * (g & 1) + (g >> 1);  // row of phi behind MMA column g
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<1>();
    __syncthreads();
    issue(ch + 2);
#pragma unroll
    for (int mt = 0; mt < S::GM / 8; ++mt) {
      if (S::MW > 1 && mt % S::MW != mw) continue;
      const int m0 = ch * S::GM + 8 * mt;
      if (m0 >= M) break;
      const double2* b = sm.stage + (ch % S::RING) * S::GSTAGE + (8 * mt + col) * S::LDG + t;
      double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0}, re2[2] = {0.0, 0.0}, im2[2] = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 2 * NT; ++k) {
        const double2 bv = b[4 * k];
        dmma884(re, a[k].x, bv.x);
        dmma884(im, a[k].x, bv.y);
        dmma884(re2, -a[k].y, bv.y);
        dmma884(im2, a[k].y, bv.x);
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int m = m0 + 4 * q + t;
        if (i < N && m < M) {
          const double2 v = make_double2(re[q] + re2[q], im[q] + im2[q]);
          ghalf[(size_t)i * M + m] = v;
          if (ghalf2 != nullptr) ghalf2[(size_t)i * M + m] = v;
        }
      }
    }
  }
  cp_async_wait<0>();
}

template <int NT, bool WITH_GHALF>
__global__ void __launch_bounds__(GfShape<NT>::THREADS, 4)
    gf_mma_kernel(const double2* __restrict__ phia, const double2* __restrict__ phib, int M, int na, int nb,
                  const double2* __restrict__ psia_c, const double2* __restrict__ psib_c,
                  const double* __restrict__ log_shift, double2* __restrict__ ghalfa, double2* __restrict__ ghalfb,
                  double2* __restrict__ ovlp, double2* __restrict__ logdet, unsigned* status, int S) {
  extern __shared__ __align__(16) unsigned char gf_sm[];
  GfShared<NT>& sm = *reinterpret_cast<GfShared<NT>*>(gf_sm);
  // two distinct spin blocks: a cluster of two CTAs, one per spin (S = 2); one block, or one
  // counted twice (phib == phia with nb == na): one CTA.  (na >= 1: the launchers refuse less)
  const int w = blockIdx.x / S, s = blockIdx.x % S;
  const bool alias = S == 1 && nb > 0;
  const int N = s == 0 ? na : nb;
  const bool beta = s == 1;
  const double2* phi = (beta ? phib : phia) + (size_t)w * M * N;
  gf_overlap_tiles<NT>(phi, beta ? psib_c : psia_c, M, N, sm);
  __syncthreads();
  gf_invert<NT>(N, sm, status);
  gf_determinant<NT>(N, sm);
  if (threadIdx.x == 0 && logdet != nullptr) {
    const double2 ld = make_double2(sm.red[0].x, atan2(sm.red[1].y, sm.red[1].x));
    logdet[(size_t)w * 2 + (beta ? 1 : 0)] = ld;
    if (alias) logdet[(size_t)w * 2 + 1] = ld;
  }
  if (S == 2) cooperative_groups::this_cluster().barrier_arrive();  // this spin's determinant is in place
  if (WITH_GHALF) {
    double2* g1 = (beta ? ghalfb : ghalfa) + (size_t)w * N * M;
    double2* g2 = (alias && ghalfb != ghalfa) ? ghalfb + (size_t)w * N * M : nullptr;
    gf_ghalf<NT>(phi, M, N, sm, g1, g2);
  }
  double logsum = sm.red[0].x;  // (thread 0 wrote them)
  double2 phase = sm.red[1];
  if (S == 2) {
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    cl.barrier_wait();
    if (s == 0 && threadIdx.x == 0) {
      const double2* other = cl.map_shared_rank(sm.red, 1);
      logsum += other[0].x;
      phase = cmul(phase, other[1]);
    }
    cl.sync();  // the peer stays until its determinant is read
  } else if (alias) {
    logsum += logsum;
    phase = cmul(phase, phase);
  }
  if (s == 0 && threadIdx.x == 0) {
    const double2 o = cscale(phase, exp(logsum - log_shift[w]));
    if (!finite2(o)) flag(status, STATUS_NONFINITE);
    ovlp[w] = o;
  }
}

// grid and cluster of a kernel that gives each distinct spin block of a walker a CTA of its own
static void spin_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr, int W, int S, int threads, int smem,
                        cudaStream_t st) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3((unsigned)(W * S));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)S;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
}

template <int NT>
cudaError_t launch_gf_mma(const double2* phia, const double2* phib, int W, int M, int na, int nb,
                          const double2* psia_c, const double2* psib_c, const double* log_shift, double2* ghalfa,
                          double2* ghalfb, double2* ovlp, double2* logdet, unsigned* status, cudaStream_t st) {
  const int smem = (int)sizeof(GfShared<NT>);
  auto k = ghalfa != nullptr ? gf_mma_kernel<NT, true> : gf_mma_kernel<NT, false>;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const int S = nb > 0 && !(phib == phia && nb == na) ? 2 : 1;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  spin_config(cfg, attr, W, S, GfShape<NT>::THREADS, smem, st);
  const cudaError_t le = cudaLaunchKernelEx(&cfg, k, phia, phib, M, na, nb, psia_c, psib_c, log_shift, ghalfa, ghalfb,
                                            ovlp, logdet, status, S);
  if (le != cudaSuccess) return le;
  note_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Reorthogonalisation of spin blocks of N <= 32 orbitals by Cholesky QR, the same unique thin QR
// (positive real diag R) as Gram-Schmidt or a sign-fixed Householder factorisation, on the f64
// tensor cores (N padded to NT tiles of 8):
//   S = phi^H phi (lower tiles): chunks of 8 rows of phi through a cp.async ring;
//   S = L L^H (L = R^H) and W = L^-1 in panels of 8 columns: one warp factors the panel with a row
//       per lane (shuffles, no barriers) and solves L_KK x = (rows K of W) with a column per lane,
//       then all warps apply them as 8 x 8 x 8 products, two barriers per panel:
//         S[I, J] -= L[I, K] L[J, K]^H (I >= J > K),  W[I, J] -= L[I, K] W[K, J] (I > K, J <= K).
//       W replaces S tile by tile in sm.O (column block J of S is spent once panel J is factored);
//   phi <- phi W^H in place, chunks of 32 rows, a row tile per warp, the zero tiles of W skipped.
// The halves of a complex product of the Gram matrix are summed in chains of their own, a panel's products by
// themselves before they change an entry, and phi W^H with its largest terms last.  That and the solves keep
// the rounding of plain sums: orbitals 2.5e-16 and det R 1.25e-15 off at M = 200, N = 32 (joint chains, every
// product added to the entry in turn and explicit inverses of the L_KK: 3.8e-16 and 1.8e-15).
// log det R = sum log L_kk.  Its error is that of the Gram matrix, ~cond(phi)^2 eps: walkers are
// reorthogonalised every few steps, so phi stays close to orthonormal and cond(phi) near 1.
// 2048 walkers, M = 200, N = 32: 537 -> 288 us (419 MB of orbitals in and out: 63 us; the products' floor is
// 100 us); 512, M = 76, N = 10: 72 -> 20 us (against DFMA products, a barrier pair per Cholesky column and
// a serial triangular inverse).
template <int NT>
struct RoShape {
  static constexpr int WARPS = NT == 3 ? 3 : 4, THREADS = 32 * WARPS, NP = 8 * NT;
  static constexpr int LDO = NP + 4, LDP = 12;
  static constexpr int LDC = NP + 2;      // chunks of the Gram product (2 mod 8)
  static constexpr int LDX = NP + 4;      // chunks of phi W^H (4 mod 8)
  static constexpr int XM = 8 * WARPS;    // rows of phi per chunk of phi W^H
  static constexpr int RING = 3;
  static constexpr int CSTAGE = kChunk * LDC, XSTAGE = XM * LDX;
  static constexpr int XRING = NT == 4 ? 2 : 3;  // (two keep four walkers of 32 electrons on an SM)
  static constexpr int STAGE = RING * CSTAGE > XRING * XSTAGE ? RING * CSTAGE : XRING * XSTAGE;
  static_assert(STAGE >= NP * LDP, "the panel lives in the rings' room");
  static constexpr int UNITS = NT * (NT + 1) / 2, PER = (UNITS + WARPS - 1) / WARPS;  // lower tiles, per warp
};

template <int NT>
struct RoShared {
  using S = RoShape<NT>;
  double2 O[S::NP * S::LDO];
  union {
    double2 stage[S::STAGE];    // copy rings of the two products with phi
    double2 P[S::NP * S::LDP];  // between them
  };
  double diag[32];
  double spread, logsum;
};

// row and column tile of lower tile u (row-major over J <= I)
__device__ __forceinline__ void lower_tile(int u, int& I, int& J) {
  I = u < 1 ? 0 : u < 3 ? 1 : u < 6 ? 2 : 3;
  J = u - I * (I + 1) / 2;
}

// (re, im) of one 8 x 8 tile += a b over 4 columns of k; the products with b's real part last, which hold
// the large terms where b is near a real diagonal
__device__ __forceinline__ void cmma(double (&re)[2], double (&im)[2], double2 a, double2 b) {
  dmma884(re, -a.y, b.y);
  dmma884(im, a.x, b.y);
  dmma884(re, a.x, b.x);
  dmma884(im, a.y, b.x);
}
__device__ __forceinline__ double2 conj_(double2 z) { return make_double2(z.x, -z.y); }

template <int NT>
__device__ __noinline__ double cholqr_block(double2* __restrict__ phi, int M, int N, RoShared<NT>& sm,
                                            unsigned* status) {
  using S = RoShape<NT>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  // ---- S = phi^H phi, tile (I, J) = sum_m conj(phi[m, I]) phi[m, J]
  {
    const int nch = (M + kChunk - 1) / kChunk;
    auto issue = [&](int ch) {
      if (ch < nch) {
        double2* st = sm.stage + (ch % S::RING) * S::CSTAGE;
        for (int e = tid; e < kChunk * S::NP; e += S::THREADS) {
          const int r = e / S::NP, c = e % S::NP, m = ch * kChunk + r;
          const bool in = m < M && c < N;
          cp_async16(st + r * S::LDC + c, phi + (in ? (size_t)m * N + c : 0), in ? 16 : 0);
        }
      }
      cp_async_commit();
    };
    // (the products of the two real and of the two mixed parts are summed apart: one chain of 2 M terms
    // rounds 1.4 times as often)
    double re[S::PER][2], im[S::PER][2], re2[S::PER][2], im2[S::PER][2];
    int arow[S::PER], bcol[S::PER];
#pragma unroll
    for (int q = 0; q < S::PER; ++q) {
      re[q][0] = re[q][1] = im[q][0] = im[q][1] = re2[q][0] = re2[q][1] = im2[q][0] = im2[q][1] = 0.0;
      int I, J;
      lower_tile(min(warp + q * S::WARPS, S::UNITS - 1), I, J);
      arow[q] = t * S::LDC + 8 * I + g;
      bcol[q] = t * S::LDC + 8 * J + g;
    }
    issue(0);
    issue(1);
    for (int ch = 0; ch < nch; ++ch) {
      cp_async_wait<1>();
      __syncthreads();
      issue(ch + 2);
      const double2* st = sm.stage + (ch % S::RING) * S::CSTAGE;
#pragma unroll
      for (int kk = 0; kk < kChunk; kk += 4)
#pragma unroll
        for (int q = 0; q < S::PER; ++q) {
          if (warp + q * S::WARPS >= S::UNITS) break;
          const double2 a = st[arow[q] + kk * S::LDC], b = st[bcol[q] + kk * S::LDC];
          dmma884(re[q], a.x, b.x);
          dmma884(im[q], a.x, b.y);
          dmma884(re2[q], a.y, b.y);
          dmma884(im2[q], -a.y, b.x);
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int q = 0; q < S::PER; ++q) {
      if (warp + q * S::WARPS >= S::UNITS) break;
      int I, J;
      lower_tile(warp + q * S::WARPS, I, J);
      // S[j, i] = conj(S[i, j]): with rows I and columns J of phi^H phi this is the lower tile
#pragma unroll
      for (int h = 0; h < 2; ++h)
        sm.O[(8 * I + g) * S::LDO + 8 * J + 2 * t + h] = make_double2(re[q][h] + re2[q][h], im[q][h] + im2[q][h]);
    }
  }
  __syncthreads();
  // ---- panels
#pragma unroll 1
  for (int kb = 0; kb < NT; ++kb) {
    if (warp == kb % S::WARPS) {
      double2 a[8];
      const int row = min(lane, S::NP - 1);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = sm.O[row * S::LDO + 8 * kb + j];
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        const int k = 8 * kb + jj;
        const double skk = __shfl_sync(0xffffffffu, a[jj].x, k < S::NP ? k : 0);
        double d = 0.0, dinv = 0.0;
        if (k < N) {
          if (!(skk > 0.0)) flag(status, STATUS_ZERO_NORM);
          d = sqrt(skk);
          dinv = 1.0 / d;
        }
        if (lane == 0) sm.diag[k] = d;
        // column k of L: rows below k (and the diagonal)
        a[jj] = lane > k ? cscale(a[jj], dinv) : lane == k ? make_double2(d, 0.0) : make_double2(0.0, 0.0);
#pragma unroll
        for (int j = jj + 1; j < 8; ++j) {
          const double2 lj = shfl2(a[jj], 8 * kb + j);
          a[j] = csub(a[j], cmul(a[jj], conj_(lj)));
        }
      }
      if (lane < S::NP)
#pragma unroll
        for (int j = 0; j < 8; ++j) sm.P[lane * S::LDP + j] = a[j];
      __syncwarp();
      // rows K of W: lane c solves L_KK x = (rows K of column c) by forward substitution
      if (lane < 8 * kb + 8) {
        double2 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          double2* o = sm.O + (8 * kb + i) * S::LDO + lane;
          double2 acc = lane < 8 * kb ? *o : make_double2(i == lane - 8 * kb ? 1.0 : 0.0, 0.0);
#pragma unroll
          for (int p = 0; p < i; ++p) acc = csub(acc, cmul(sm.P[(8 * kb + i) * S::LDP + p], x[p]));
          const double d = sm.P[(8 * kb + i) * S::LDP + i].x;
          x[i] = d != 0.0 ? make_double2(acc.x / d, acc.y / d) : make_double2(0.0, 0.0);
          *o = x[i];
        }
      }
    }
    __syncthreads();
    // S[I, J] -= L[I, K] L[J, K]^H (I >= J > K), W[I, J] -= L[I, K] W[K, J] (I > K >= J; W[I, K] was zero)
    for (int u = warp; u < S::UNITS; u += S::WARPS) {
      int I, J;
      lower_tile(u, I, J);
      if (I <= kb) continue;
      double2* c = sm.O + (8 * I + g) * S::LDO + 8 * J + 2 * t;
      double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
#pragma unroll
      for (int h = 0; h < 8; h += 4) {
        const double2 l = sm.P[(8 * I + g) * S::LDP + h + t];
        const double2 r = J > kb ? conj_(sm.P[(8 * J + g) * S::LDP + h + t])
                                 : sm.O[(8 * kb + h + t) * S::LDO + 8 * J + g];
        cmma(re, im, l, r);
      }
      // (the products summed by themselves, then one rounding of the entry)
      c[0] = J == kb ? make_double2(-re[0], -im[0]) : make_double2(c[0].x - re[0], c[0].y - im[0]);
      c[1] = J == kb ? make_double2(-re[1], -im[1]) : make_double2(c[1].x - re[1], c[1].y - im[1]);
    }
    __syncthreads();
  }
  if (tid < 32) {
    double ls = 0.0, rmax = 0.0, rmin = 1.0e300;
    if (lane < N) {
      const double r = sm.diag[lane];
      ls = log(r);
      rmax = rmin = r;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ls += __shfl_xor_sync(0xffffffffu, ls, o);
      rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
      rmin = fmin(rmin, __shfl_xor_sync(0xffffffffu, rmin, o));
    }
    if (lane == 0) {
      sm.logsum = ls;
      sm.spread = ls == ls ? rmax / rmin : ls;  // a lower bound on cond(phi); NaN when a pivot failed
    }
  }
  // ---- phi <- phi W^H: out[m, j] = sum_{c <= j} phi[m, c] conj(W[j, c])
  const int nch = (M + S::XM - 1) / S::XM;
  auto issue = [&](int ch) {
    if (ch < nch) {
      double2* st = sm.stage + (ch % S::XRING) * S::XSTAGE;
      for (int e = tid; e < S::XM * S::NP; e += S::THREADS) {
        const int r = e / S::NP, c = e % S::NP, m = ch * S::XM + r;
        const bool in = m < M && c < N;
        cp_async16(st + r * S::LDX + c, phi + (in ? (size_t)m * N + c : 0), in ? 16 : 0);
      }
    }
    cp_async_commit();
  };
  issue(0);
  if (S::XRING == 3) issue(1);
  const int col = 4 * (g & 1) + (g >> 1);  // output column behind MMA column g (neighbouring stores)
  for (int ch = 0; ch < nch; ++ch) {
    if (S::XRING == 3)
      cp_async_wait<1>();
    else
      cp_async_wait<0>();
    __syncthreads();
    issue(ch + S::XRING - 1);  // rows ahead of the ones rewritten below
    const double2* a = sm.stage + (ch % S::XRING) * S::XSTAGE + (8 * warp + g) * S::LDX + t;
    const int m = ch * S::XM + 8 * warp + g;
    if (ch * S::XM + 8 * warp >= M) continue;
    double2 av[2 * NT];
#pragma unroll
    for (int k = 0; k < 2 * NT; ++k) av[k] = a[4 * k];
#pragma unroll
    for (int J = 0; J < NT; ++J) {
      double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
      const double2* w = sm.O + (8 * J + col) * S::LDO + t;
#pragma unroll
      for (int k = 0; k < 2 * (J + 1); ++k) cmma(re, im, av[k], conj_(w[4 * k]));
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int j = 8 * J + 4 * q + t;
        if (m < M && j < N) phi[(size_t)m * N + j] = make_double2(re[q], im[q]);
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  return sm.logsum;
}

constexpr double kCholQR2 = 20.0;  // R-diagonal spread above which a block gets a second pass

// detR = exp(sum log R_kk - detR_shift), log_detR += log detR, ovlp /= detR (the contract of
// reortho_kernel in walkers.cu, which keeps N > 32).
template <int NT>
__global__ void __launch_bounds__(RoShape<NT>::THREADS, 4)
    reortho_chol32_kernel(double2* __restrict__ phia, double2* __restrict__ phib, int M, int na, int nb,
                          const double* __restrict__ detR_shift, double* __restrict__ detR,
                          double* __restrict__ log_detR, double2* __restrict__ ovlp, unsigned* status, int S) {
  extern __shared__ __align__(16) unsigned char gf_sm[];
  RoShared<NT>& sm = *reinterpret_cast<RoShared<NT>*>(gf_sm);
  // as the Green's function: one CTA per distinct spin block, a walker's two in a cluster
  const int w = blockIdx.x / S, s = blockIdx.x % S;
  const bool alias = S == 1 && nb > 0;
  const int N = s == 0 ? na : nb;
  double2* phi = (s == 0 ? phia : phib) + (size_t)w * M * N;
  double l = cholqr_block<NT>(phi, M, N, sm, status);
  // CholQR2: a second pass over the (now nearly orthonormal) result when R's diagonal spreads
  // by more than kCholQR2 (the first pass's error grows like cond(phi)^2 eps); R = R2 R1, so
  // the log-determinants add
  if (!(sm.spread <= kCholQR2)) {
    __syncthreads();  // everyone has read the spread and the sum
    l += cholqr_block<NT>(phi, M, N, sm, status);
  }
  if (S == 2) {
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    if (threadIdx.x == 0) sm.logsum = l;
    cl.sync();
    if (s == 0 && threadIdx.x == 0) l += *cl.map_shared_rank(&sm.logsum, 1);
    cl.sync();  // the peer stays until its sum is read
  } else if (alias) {
    l += l;
  }
  if (s == 0 && threadIdx.x == 0) {
    const double d = exp(l - detR_shift[w]);
    detR[w] = d;
    log_detR[w] += log(d);
    ovlp[w] = cscale(ovlp[w], 1.0 / d);
  }
}

template <int NT>
cudaError_t launch_reortho_nt(double2* phia, double2* phib, int W, int M, int na, int nb, const double* detR_shift,
                              double* detR, double* log_detR, double2* ovlp, unsigned* status, cudaStream_t st) {
  const int smem = (int)sizeof(RoShared<NT>);
  auto k = reortho_chol32_kernel<NT>;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const int S = nb > 0 && !(phib == phia && nb == na) ? 2 : 1;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  spin_config(cfg, attr, W, S, RoShape<NT>::THREADS, smem, st);
  const cudaError_t le =
      cudaLaunchKernelEx(&cfg, k, phia, phib, M, na, nb, detR_shift, detR, log_detR, ovlp, status, S);
  if (le != cudaSuccess) return le;
  note_launch();
  return cudaGetLastError();
}

}  // namespace

bool gf_lu32_fits(int na, int nb) { return na >= 1 && na <= 32 && nb >= 0 && nb <= 32; }

cudaError_t launch_gf_lu32(const double2* phia, const double2* phib, int W, int M, int na, int nb,
                           const double2* psia_c, const double2* psib_c, const double* log_shift, double2* ghalfa,
                           double2* ghalfb, double2* ovlp, double2* logdet, unsigned* status, cudaStream_t st) {
  if (!gf_lu32_fits(na, nb) || M <= 0 || W <= 0) return cudaErrorInvalidValue;
  switch ((max(na, nb) + 7) / 8) {
    case 1: return launch_gf_mma<1>(phia, phib, W, M, na, nb, psia_c, psib_c, log_shift, ghalfa, ghalfb, ovlp, logdet, status, st);
    case 2: return launch_gf_mma<2>(phia, phib, W, M, na, nb, psia_c, psib_c, log_shift, ghalfa, ghalfb, ovlp, logdet, status, st);
    case 3: return launch_gf_mma<3>(phia, phib, W, M, na, nb, psia_c, psib_c, log_shift, ghalfa, ghalfb, ovlp, logdet, status, st);
    default: return launch_gf_mma<4>(phia, phib, W, M, na, nb, psia_c, psib_c, log_shift, ghalfa, ghalfb, ovlp, logdet, status, st);
  }
}

cudaError_t launch_reortho_chol32(double2* phia, double2* phib, int W, int M, int na, int nb,
                                  const double* detR_shift, double* detR, double* log_detR, double2* ovlp,
                                  unsigned* status, cudaStream_t st) {
  if (na < 1 || na > 32 || nb < 0 || nb > 32 || M <= 0 || W <= 0) return cudaErrorInvalidValue;
  switch ((max(na, nb) + 7) / 8) {
    case 1: return launch_reortho_nt<1>(phia, phib, W, M, na, nb, detR_shift, detR, log_detR, ovlp, status, st);
    case 2: return launch_reortho_nt<2>(phia, phib, W, M, na, nb, detR_shift, detR, log_detR, ovlp, status, st);
    case 3: return launch_reortho_nt<3>(phia, phib, W, M, na, nb, detR_shift, detR, log_detR, ovlp, status, st);
    default: return launch_reortho_nt<4>(phia, phib, W, M, na, nb, detR_shift, detR, log_detR, ovlp, status, st);
  }
}

}  // namespace ipie_b200
