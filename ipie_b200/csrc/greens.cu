// Green's function, overlap and reorthogonalisation for spin blocks of N <= 32 electrons: one CTA of
// 96 or 128 threads per walker, four per SM, the products on the f64 tensor cores.
// ovlp_w = prod_s phase_s * exp(sum_s log|det O_s| - log_shift_w).
// Same contracts as gf_overlap_kernel and reortho_kernel (walkers.cu), which keep N > 32.
#include "common.cuh"
#include "kernels.h"

namespace ipie_b200 {

namespace {

constexpr int kThreads = 128;
constexpr int kChunk = 8;   // rows of phi / psi* per shared-memory chunk of the O product
constexpr int kORing = 3;   // chunks in the O product's copy ring
constexpr int kNP = 33;     // row stride of O in shared memory
constexpr int kRC = 4;      // permuted columns of phi per staged step of the Ghalf product
constexpr int kMQ = 2;      // columns of Ghalf per lane and pass (64 per pass)
constexpr int kMS = 32 * kMQ + 1;  // row stride of the staged phi^T step (odd in 16-byte units)
constexpr int kGRing = 4;   // steps in the Ghalf product's copy ring
constexpr int kOStage = 2 * kChunk * 32;  // double2 per O chunk (phi and psi*)
constexpr int kGStage = kRC * kMS;        // double2 per Ghalf step
constexpr int kStage = kORing * kOStage > kGRing * kGStage ? kORing * kOStage : kGRing * kGStage;
static_assert(kChunk * 32 % kThreads == 0 && kRC * 32 * kMQ % kThreads == 0, "whole copies per thread");

struct SpinDet32 {
  double logabs;
  double2 phase;
};

// sO = phi^T psi* (or, GRAM, the Gram matrix phi^H phi: psic unused) of one spin block.  phi and
// psi* stream through shared memory in 8-row chunks, a three-deep ring of cp.async copies issued
// two chunks ahead (one barrier per chunk); thread (ti, tj) accumulates rows {ti, ti+16} x
// columns {tj + 8q} in registers.  The caller synchronises before reading sO.
template <bool GRAM>
__device__ void o_product(const double2* __restrict__ phi, const double2* __restrict__ psic, int M, int N,
                          double2 (*sO)[kNP], double2* sStage) {
  const int tid = threadIdx.x;
  const int ti = tid >> 3, tj = tid & 7;
  double2 acc[2][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[a][q] = make_double2(0.0, 0.0);
  const int nch = (M + kChunk - 1) / kChunk;
  // chunk ch (rows 8 ch ..) into ring slot ch % kORing: phi rows then psi* rows, zeros past M / N
  auto issue = [&](int ch) {
    if (ch < nch) {
      double2* st = sStage + (ch % kORing) * kOStage;
#pragma unroll
      for (int u = 0; u < kChunk * 32 / kThreads; ++u) {
        const int e = tid + u * kThreads, r = e >> 5, c = e & 31, m = ch * kChunk + r;
        const bool in = m < M && c < N;
        const size_t off = in ? (size_t)m * N + c : 0;
        cp_async16(st + e, phi + off, in ? 16 : 0);
        if (!GRAM) cp_async16(st + kChunk * 32 + e, psic + off, in ? 16 : 0);
      }
    }
    cp_async_commit();  // (an empty group past the end keeps the group count per chunk)
  };
  issue(0);
  issue(1);
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<1>();  // this thread's copies of chunk ch have landed
    __syncthreads();     // everyone's have, and everyone is done with chunk ch - 1
    issue(ch + 2);       // into the slot of chunk ch - 1
    const double2(*sPhi)[32] = reinterpret_cast<const double2(*)[32]>(sStage + (ch % kORing) * kOStage);
    const double2(*sPsi)[32] =
        GRAM ? sPhi : reinterpret_cast<const double2(*)[32]>(sStage + (ch % kORing) * kOStage + kChunk * 32);
#pragma unroll
    for (int r = 0; r < kChunk; ++r) {
      double2 a0 = sPhi[r][ti], a1 = sPhi[r][ti + 16];
      if (GRAM) {
        a0.y = -a0.y;
        a1.y = -a1.y;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double2 b = sPsi[r][tj + 8 * q];
        acc[0][q].x += a0.x * b.x - a0.y * b.y;
        acc[0][q].y += a0.x * b.y + a0.y * b.x;
        acc[1][q].x += a1.x * b.x - a1.y * b.y;
        acc[1][q].y += a1.x * b.y + a1.y * b.x;
      }
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int q = 0; q < 4; ++q) sO[ti + 16 * a][tj + 8 * q] = acc[a][q];
}

// ---------------------------------------------------------------------------------------------
// The Green's function on the f64 tensor cores, N padded to NT tiles of 8.  Per walker and spin:
//   O = phi^T psi*: chunks of 8 rows of phi and psi* through a three-deep cp.async ring; warp w
//       owns row tile w of O (NT = 1: a quarter of the rows m, NT = 2: one of the four tiles).
//   O^-1 by Gauss-Jordan elimination in place, partial pivoting on |.|, in panels of 8 columns: one
//       warp factors the panel with a row per lane and the 8 columns in registers (the pivot by one
//       redux.sync on the float bits of |a|^2 above the row index, its row by shuffles; pivots stay
//       in their rows), then all warps apply it to the other columns as one rank-8 MMA update
//         A[:, J] <- A[:, J] (pivot rows zeroed) + panel' A[pivot rows, J].
//       So a column costs no barrier and a panel three, where the column by column form took two
//       per column.
//   With p_k the pivot row of column k the stored array B holds O^-1[k, p_j] = B[p_k, j].
//   Ghalf[i, m] = sum_c O^-1[i, c] phi[m, c]: warp w keeps its rows of O^-1 as MMA fragments in
//       registers (gathered through p once) while chunks of 16 rows of phi pass through the ring.
//       The eight rows m of a tile are dealt to the MMA's columns as 0 4 1 5 2 6 3 7, so that four
//       lanes store four neighbouring entries of Ghalf; rows of an odd stride keep the fragment
//       loads free of bank conflicts.
// The floor is the f64 tensor pipe's time for the two products (28k cycles per SM and walker at
// M = 200, N = 32).  2048 walkers, M = 200, N = 32: 535 -> 354 us; 512, M = 76, N = 10: 46 -> 19 us; 777, M =
// 149, N = 23 + 17: 280 -> 175 us (against DFMA products and the column by column elimination).
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
  double re[CT][2], im[CT][2];
#pragma unroll
  for (int j = 0; j < CT; ++j) re[j][0] = re[j][1] = im[j][0] = im[j][1] = 0.0;
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
        dmma884(re[j], -av.y, bv.y);
        dmma884(im[j], av.y, bv.x);
      }
    }
  }
  cp_async_wait<0>();
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
            key = (__float_as_uint((float)cabs2(own)) & ~31u) | (unsigned)(31 - lane);
          // every lane scales its row as if it held the pivot, while the pivot is found
          const double rn = __drcp_rn(own.x * own.x + own.y * own.y);
          const double2 pinv = make_double2(own.x * rn, -own.y * rn);
          double2 s[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] = j == jj ? pinv : cmul(a[j], pinv);
          key = __reduce_max_sync(0xffffffffu, key);
          int p = 31 - (int)(key & 31u);
          if (key < 32u) {
            // no positive |a|^2 left (an exactly singular block, or NaN): any free row
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
      double2* c = sm.O + row * S::LDO + 8 * (ct0 + j) + 2 * t;
      double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
      if (!pivot) {
        const double2 c0 = c[0], c1 = c[1];
        re[0] = c0.x;
        re[1] = c1.x;
        im[0] = c0.y;
        im[1] = c1.y;
      }
      dmma884(re, a0.x, b[j][0].x);
      dmma884(im, a0.x, b[j][0].y);
      dmma884(re, -a0.y, b[j][0].y);
      dmma884(im, a0.y, b[j][0].x);
      dmma884(re, a1.x, b[j][1].x);
      dmma884(im, a1.x, b[j][1].y);
      dmma884(re, -a1.y, b[j][1].y);
      dmma884(im, a1.y, b[j][1].x);
      c[0] = make_double2(re[0], im[0]);
      c[1] = make_double2(re[1], im[1]);
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
                  double2* __restrict__ ovlp, double2* __restrict__ logdet, unsigned* status) {
  extern __shared__ __align__(16) unsigned char gf_sm[];
  GfShared<NT>& sm = *reinterpret_cast<GfShared<NT>*>(gf_sm);
  const int w = blockIdx.x;
  // spin aliasing: phib == phia with nb == na is one block counted twice
  const bool alias = (phib == phia) && (nb == na);
  double logsum = 0.0;
  double2 phase = make_double2(1.0, 0.0);  // (thread 0's are used)
  for (int s = 0; s < 2; ++s) {
    const int N = s == 0 ? na : nb;
    if (N == 0) continue;
    if (s == 1 && alias) {
      logsum += logsum;
      phase = cmul(phase, phase);
      if (logdet != nullptr && threadIdx.x == 0) logdet[(size_t)w * 2 + 1] = logdet[(size_t)w * 2];
      continue;
    }
    const double2* phi = (s == 0 ? phia : phib) + (size_t)w * M * N;
    gf_overlap_tiles<NT>(phi, s == 0 ? psia_c : psib_c, M, N, sm);
    __syncthreads();
    gf_invert<NT>(N, sm, status);
    gf_determinant<NT>(N, sm);
    if (threadIdx.x == 0) {
      logsum += sm.red[0].x;
      phase = cmul(phase, sm.red[1]);
      if (logdet != nullptr) logdet[(size_t)w * 2 + s] = make_double2(sm.red[0].x, atan2(sm.red[1].y, sm.red[1].x));
    }
    if (WITH_GHALF) {
      double2* g1 = (s == 0 ? ghalfa : ghalfb) + (size_t)w * N * M;
      double2* g2 = (s == 0 && alias && nb > 0 && ghalfb != ghalfa) ? ghalfb + (size_t)w * N * M : nullptr;
      gf_ghalf<NT>(phi, M, N, sm, g1, g2);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double2 o = cscale(phase, exp(logsum - log_shift[w]));
    if (!finite2(o)) flag(status, STATUS_NONFINITE);
    ovlp[w] = o;
  }
}

template <int NT>
cudaError_t launch_gf_mma(const double2* phia, const double2* phib, int W, int M, int na, int nb,
                          const double2* psia_c, const double2* psib_c, const double* log_shift, double2* ghalfa,
                          double2* ghalfb, double2* ovlp, double2* logdet, unsigned* status, cudaStream_t st) {
  const int smem = (int)sizeof(GfShared<NT>);
  auto k = ghalfa != nullptr ? gf_mma_kernel<NT, true> : gf_mma_kernel<NT, false>;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  k<<<W, GfShape<NT>::THREADS, smem, st>>>(phia, phib, M, na, nb, psia_c, psib_c, log_shift, ghalfa, ghalfb, ovlp,
                                           logdet, status);
  note_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Reorthogonalisation of spin blocks of N <= 32 orbitals by Cholesky QR, the same unique thin QR
// (positive real diag R) as Gram-Schmidt or a sign-fixed Householder factorisation:
//   S = phi^H phi (o_product<true>), S = R^H R (Cholesky, right-looking, in shared memory; warp 0
//   scales the pivot row, all threads update the trailing upper triangle), X = R^-1 (warp 0,
//   lane i solving row i of X R = I, kept in the lower triangle of sO transposed plus the
//   diagonal), phi <- phi X in place (16-row chunks of phi through the copy ring; lane i forms
//   column i of four rows per warp, so each output row is one coalesced 512-byte store).
// log det R = sum log R_kk.  Its error is that of the Gram matrix, ~cond(phi)^2 eps: walkers are
// reorthogonalised every few steps, so phi stays close to orthonormal and cond(phi) near 1.
__device__ __noinline__ double cholqr_block(double2* __restrict__ phi, int M, int N, double2 (*sO)[kNP], double2* sStage,
                               double2* sDinv, double* sSpread, unsigned* status) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  o_product<true>(phi, nullptr, M, N, sO, sStage);
  __syncthreads();
  // ---- S = R^H R in the upper triangle of sO
  const int uj = tid & 31, ui = tid >> 5;
  for (int k = 0; k < N; ++k) {
    if (tid < 32) {
      const double skk = sO[k][k].x;
      __syncwarp();  // every lane has read the pivot before lane 0 replaces it
      if (!(skk > 0.0)) flag(status, STATUS_ZERO_NORM);
      const double d = sqrt(skk), dinv = 1.0 / d;
      if (lane > k && lane < N) sO[k][lane] = cscale(sO[k][lane], dinv);
      if (lane == 0) {
        sO[k][k] = make_double2(d, 0.0);
        sDinv[k] = make_double2(dinv, 0.0);
      }
    }
    __syncthreads();
    // S_ij -= conj(R_ki) R_kj for k < i <= j (loads first, as in the Gauss-Jordan update)
    if (uj > k && uj < N) {
      const double2 rkj = sO[k][uj];
      double2 a[8], f[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int i = ui + 4 * r;
        a[r] = sO[i][uj];
        f[r] = sO[k][i];
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int i = ui + 4 * r;
        if (i > k && i <= uj) sO[i][uj] = csub(a[r], cmulc(f[r], rkj));
      }
    }
    __syncthreads();
  }
  double logsum = 0.0;
  if (tid < 32) {
    // ---- X = R^-1 (upper): lane i, row i: X_ii = 1 / R_ii, X_ij = -(sum_{i<=k<j} X_ik R_kj) / R_jj
    double2 x[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < j; ++k) {
        const double2 rkj = sO[k][j];  // the same for every lane: a broadcast
        acc.x += x[k].x * rkj.x - x[k].y * rkj.y;
        acc.y += x[k].x * rkj.y + x[k].y * rkj.x;
      }
      const double di = j < N ? sDinv[j].x : 0.0;
      x[j] = lane == j ? make_double2(di, 0.0) : (lane < j ? make_double2(-acc.x * di, -acc.y * di)
                                                           : make_double2(0.0, 0.0));
    }
    // X_ij (i < j) to sO[j][i], below the diagonal: R is no longer read after the barrier
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (lane < j && j < N) sO[j][lane] = x[j];
    double rmax = 0.0, rmin = 1.0e300;
    if (lane < N) {
      const double r = sO[lane][lane].x;
      logsum = log(r);
      rmax = rmin = r;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      logsum += __shfl_xor_sync(0xffffffffu, logsum, o);
      rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
      rmin = fmin(rmin, __shfl_xor_sync(0xffffffffu, rmin, o));
    }
    if (lane == 0) *sSpread = rmax / rmin;  // a lower bound on cond(phi); NaN when a pivot failed
  }
  __syncthreads();
  // ---- phi <- phi X: lane i = column i, rows m0 + 4 warp + a
  const int nch = (M + 15) / 16;
  auto issue = [&](int ch) {
    if (ch < nch) {
      double2* st = sStage + (ch % kORing) * kOStage;
#pragma unroll
      for (int u = 0; u < 16 * 32 / kThreads; ++u) {
        const int e = tid + u * kThreads, r = e >> 5, c = e & 31, m = ch * 16 + r;
        const bool in = m < M && c < N;
        cp_async16(st + e, phi + (in ? (size_t)m * N + c : 0), in ? 16 : 0);
      }
    }
    cp_async_commit();
  };
  issue(0);
  issue(1);
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<1>();
    __syncthreads();
    issue(ch + 2);  // rows ahead of the ones rewritten below
    const double2(*sPhi)[32] = reinterpret_cast<const double2(*)[32]>(sStage + (ch % kORing) * kOStage);
    double2 acc[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) acc[a] = make_double2(0.0, 0.0);
#pragma unroll 8
    for (int r = 0; r < 32; ++r) {
      // X[r][lane]: below the diagonal of sO transposed, the diagonal in sDinv, zero for r > lane
      const double2 xr = r < lane ? sO[lane][r] : (r == lane && r < N ? sDinv[r] : make_double2(0.0, 0.0));
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const double2 p = sPhi[4 * warp + a][r];
        acc[a].x += p.x * xr.x - p.y * xr.y;
        acc[a].y += p.x * xr.y + p.y * xr.x;
      }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int m = ch * 16 + 4 * warp + a;
      if (m < M && lane < N) phi[(size_t)m * N + lane] = acc[a];
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  return logsum;  // valid in warp 0
}

constexpr double kCholQR2 = 20.0;  // R-diagonal spread above which a block gets a second pass

// One CTA per walker: both spin blocks (the alpha block once when phib aliases it), then
// detR = exp(sum log R_kk - detR_shift), log_detR += log detR, ovlp /= detR (the contract of
// reortho_kernel in walkers.cu, which keeps N > 32).
__global__ void __launch_bounds__(kThreads, 4) reortho_chol32_kernel(double2* __restrict__ phia,
                                                                     double2* __restrict__ phib, int M, int na,
                                                                     int nb, const double* __restrict__ detR_shift,
                                                                     double* __restrict__ detR,
                                                                     double* __restrict__ log_detR,
                                                                     double2* __restrict__ ovlp, unsigned* status) {
  __shared__ double2 sO[32][kNP];
  __shared__ __align__(16) double2 sStage[kStage];
  __shared__ double2 sDinv[32];
  __shared__ double sSpread;
  const int w = blockIdx.x;
  const bool alias = (phib == phia) && (nb == na);
  double logsum = 0.0, log_a = 0.0;
  for (int s = 0; s < 2; ++s) {
    const int N = s == 0 ? na : nb;
    if (N == 0) continue;
    if (s == 1 && alias) {
      logsum += log_a;
      continue;
    }
    double2* phi = (s == 0 ? phia : phib) + (size_t)w * M * N;
    double l = cholqr_block(phi, M, N, sO, sStage, sDinv, &sSpread, status);
    // CholQR2: a second pass over the (now nearly orthonormal) result when R's diagonal spreads
    // by more than kCholQR2 (the first pass's error grows like cond(phi)^2 eps); R = R2 R1, so
    // the log-determinants add
    if (!(sSpread <= kCholQR2)) l += cholqr_block(phi, M, N, sO, sStage, sDinv, &sSpread, status);
    logsum += l;
    if (s == 0) log_a = l;
  }
  if (threadIdx.x == 0) {
    const double d = exp(logsum - detR_shift[w]);
    detR[w] = d;
    log_detR[w] += log(d);
    ovlp[w] = cscale(ovlp[w], 1.0 / d);
  }
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
  reortho_chol32_kernel<<<W, kThreads, 0, st>>>(phia, phib, M, na, nb, detR_shift, detR, log_detR, ovlp, status);
  note_launch();
  return cudaGetLastError();
}

}  // namespace ipie_b200
