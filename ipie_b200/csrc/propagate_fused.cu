// Fused orbital propagation for one walker-spin per CTA:
//
//   phi <- expH1 . phi                       (one-body, optional)
//   T_0 = phi;  T_n = VHS T_{n-1} / n;  phi <- phi + sum_{n=1..nmax} T_n
//   phi <- expH1 . phi                       (one-body, optional)
//
// the arithmetic of ipie's propagate_one_body (propagation/operations.py:26-55)
// and apply_exponential (operations.py:58-82), in one launch.  The running
// term T lives in shared memory for the whole chain, complex, and is the right
// operand of every pass; the left operand is this walker's VHS or the shared
// expH1.
//
// MMA: f64 tensor cores (mma.sync m8n8k4).  A lane reads a complex entry of VHS and
// of T with one 16-byte shared-memory load each and feeds four MMAs with them
// (re re, -im im, re im, im re): real and imaginary parts of a product sit in the
// same lane, so nothing is embedded or selected.  Warp r owns rows 8r..8r+7 and all
// (or a group of) columns: its row of VHS is read once per pass, and the 7 to 32 warps
// spread over the four schedulers to within one warp.
//
// The chain is bound by the f64 tensor pipe once a CTA's warps cover the MMA latency.  Two
// kernels by M:
//   M <= 80 (resident): VHS and expH1 are copied to shared memory once and all passes run
//     from there, two barriers per pass; phi's sum stays in registers.  (Streaming them again
//     for each pass is 6 x the L2 traffic and a barrier per 8 columns, which is what a small
//     walker's time went into.)
//   above: VHS streams through a ring of cp.async chunks (8 complex or 16 real columns of
//     all rows, 128-byte rows, swizzled), two chunks ahead, one barrier per chunk; its six
//     re-reads hit L2.
// The eight columns of a tile are dealt to the MMA's columns as 0 4 1 5 2 6 3 7, so that the four
// lanes of a row hold (and load and store) four neighbouring complex entries at a time; with a row
// stride of T of 1 modulo 8 the fragment loads stay free of bank conflicts.
// Measured against one kernel that streamed VHS for every M and embedded T as a real matrix: 640 walkers,
// M = 108, N = 15: 663 -> 346 us per spin; 1024 walkers, M = 160, N = 26: 2.69 -> 1.77 ms (38 GFLOP, 47 with
// N padded to 32: 27 TFLOP/s); 64 walkers, M = 26, N = 5: 24.3 -> 7 us.
#include "common.cuh"
#include "kernels.h"

namespace ipie_b200 {

namespace {

// acc (one 8 x 8 complex tile: re, im) += (ar + i ai) (b.x + i b.y) over 4 columns of k
__device__ __forceinline__ void cmma(double (&re)[2], double (&im)[2], double ar, double ai, double nai, double2 b) {
  dmma884(re, ar, b.x);
  dmma884(im, ar, b.y);
  dmma884(re, nai, b.y);
  dmma884(im, ai, b.x);
}

// column of a tile behind MMA column n
__device__ __forceinline__ int tile_col(int n) { return 4 * (n & 1) + (n >> 1); }

// ---------------------------------------------------------------- resident operands
constexpr int kResM = 80;
__host__ __device__ inline int res_stride(int n, int m) { return n + ((4 - n) & (m - 1)); }  // n or more, 4 mod m

struct ResShape {
  int RT, CT, CG;     // 8-row tiles, 8-column tiles, column groups of CW tiles
  int ldv, lde, ldt;  // row strides: VHS (double2, 4 mod 8), expH1 (double, 4 mod 16), T (double2, 1 mod 8)
  size_t smem;
};
ResShape res_shape(int M, int N, int CW, bool one_body) {
  ResShape s;
  s.RT = (M + 7) / 8;
  s.CT = (N + 7) / 8;
  s.CG = (s.CT + CW - 1) / CW;
  const int k4 = (M + 3) & ~3;
  s.ldv = res_stride(k4, 8);
  s.lde = res_stride(k4, 16);
  s.ldt = 8 * s.CG * CW + 1;
  s.smem = sizeof(double2) * ((size_t)8 * s.RT * s.ldv + (size_t)8 * s.RT * s.ldt) +
           (one_body ? sizeof(double) * 8 * s.RT * s.lde : 0);
  return s;
}

template <int CW>
__global__ void __launch_bounds__(640)
    propagate_resident_kernel(const double2* __restrict__ vhs, const double* __restrict__ expH1, int lda_e,
                              const double2* __restrict__ phi_in, double2* __restrict__ phi_out, int M, int N, int nmax,
                              int pre, int post, ResShape s) {
  extern __shared__ __align__(16) unsigned char pf_sm[];
  const int rows = 8 * s.RT, tid = threadIdx.x, nth = blockDim.x;
  double2* const sV = reinterpret_cast<double2*>(pf_sm);
  double2* const sT = sV + rows * s.ldv;
  double* const sE = reinterpret_cast<double*>(sT + rows * s.ldt);
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int rt = warp % s.RT, cg = warp / s.RT;
  const size_t w = blockIdx.x;
  const double2* vw = vhs + w * M * M;
  const double2* pin = phi_in + w * M * N;
  double2* pout = phi_out + w * M * N;
  // zeros in the padding (rows past M, columns past M or N), everything else copied: expH1 and phi
  // first, since the chain starts on them
  const double2 zero = make_double2(0.0, 0.0);
  const bool one_body = pre || post;
  for (int e = tid; e < rows * s.ldt; e += nth) {
    const int r = e / s.ldt, c = e - r * s.ldt;
    if (r < M && c < N)
      cp_async16(sT + e, pin + r * N + c, 16);
    else
      sT[e] = zero;
  }
  if (one_body) {
    const int half = s.lde / 2;
    for (int e = tid; e < rows * half; e += nth) {
      const int r = e / half, c = 2 * (e - r * half);
      const bool in = r < M && c < M;
      cp_async16(sE + r * s.lde + c, in ? expH1 + (size_t)r * lda_e + c : expH1, in ? (M - c >= 2 ? 16 : 8) : 0);
    }
  }
  cp_async_commit();
  for (int e = tid; e < rows * s.ldv; e += nth) {
    const int r = e / s.ldv, c = e - r * s.ldv;
    if (r < M && c < M)
      cp_async16(sV + e, vw + r * M + c, 16);
    else
      sV[e] = zero;
  }
  cp_async_commit();
  if (pre)
    cp_async_wait<1>();  // the first pass needs phi and expH1; VHS is waited for at its end
  else
    cp_async_wait<0>();
  __syncthreads();

  const int npass = nmax + (pre ? 1 : 0) + (post ? 1 : 0);
  const int r = rt * 8 + g, c0 = cg * CW * 8;
  double2 phi[CW][2];
  const double2* const tb = sT + t * s.ldt + c0 + tile_col(g);  // right fragments: rows k + t
#pragma unroll
  for (int j = 0; j < CW; ++j)
#pragma unroll
    for (int q = 0; q < 2; ++q) phi[j][q] = sT[r * s.ldt + c0 + 8 * j + 4 * q + t];
  for (int p = 0; p < npass; ++p) {
    const bool first = pre && p == 0, last = p == npass - 1, one = first || (post && last);
    double re[CW][2], im[CW][2], re2[CW][2], im2[CW][2];
#pragma unroll
    for (int j = 0; j < CW; ++j)
      re[j][0] = re[j][1] = im[j][0] = im[j][1] = re2[j][0] = re2[j][1] = im2[j][0] = im2[j][1] = 0.0;
    if (one) {
      const double* a = sE + r * s.lde + t;
#pragma unroll 4
      for (int k = 0; k < M; k += 4) {
        const double av = a[k];
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          const double2 b = tb[k * s.ldt + 8 * j];
          dmma884(re[j], av, b.x);
          dmma884(im[j], av, b.y);
        }
      }
    } else {
      const double2* a = sV + r * s.ldv + t;
#pragma unroll 4
      for (int k = 0; k < M; k += 4) {
        const double2 av = a[k];
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          const double2 b = tb[k * s.ldt + 8 * j];
          dmma884(re[j], av.x, b.x);
          dmma884(im[j], av.x, b.y);
          dmma884(re2[j], -av.y, b.y);
          dmma884(im2[j], av.y, b.x);
        }
      }
    }
    const bool to_post = post && p + 1 == npass - 1;
    const double sc = one ? 1.0 : 1.0 / (p + 1 - (pre ? 1 : 0));
    if (p == 0) cp_async_wait<0>();  // VHS, read from the next barrier on
    if (!last) __syncthreads();      // every warp has read the old term
#pragma unroll
    for (int j = 0; j < CW; ++j)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = c0 + 8 * j + 4 * q + t;
        const double2 v = make_double2((re[j][q] + re2[j][q]) * sc, (im[j][q] + im2[j][q]) * sc);
        phi[j][q] = one ? v : cadd(phi[j][q], v);
        if (last) {
          if (r < M && c < N) pout[(size_t)r * N + c] = phi[j][q];
        } else {
          sT[r * s.ldt + c] = to_post ? phi[j][q] : v;  // (rows past M and columns past N stay zero: zero products)
        }
      }
    if (!last) __syncthreads();
  }
}

template <int CW>
cudaError_t launch_resident(const double2* vhs, const double* expH1, int lda_e, const double2* phi_in,
                            double2* phi_out, int W, int M, int N, int nmax, int pre, int post, cudaStream_t st) {
  const ResShape s = res_shape(M, N, CW, pre || post);
  auto k = propagate_resident_kernel<CW>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
  if (e != cudaSuccess) return e;
  k<<<W, 32 * s.RT * s.CG, s.smem, st>>>(vhs, expH1, lda_e, phi_in, phi_out, M, N, nmax, pre, post, s);
  note_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------- streamed operands
constexpr int kRow = 128;  // bytes of one row of a chunk: 8 complex or 16 real columns

// smem rows of T: every k of either kind of chunk
__host__ __device__ inline int stream_trows(int M) { return (M + 15) & ~15; }

// CT: 8-column tiles (all of a warp's rows).  PHI_REG: phi's sum in registers, else in phi_out
// (each lane reads back its own entries).
template <int CT, int MAXT, bool PHI_REG>
__global__ void __launch_bounds__(MAXT)
    propagate_stream_kernel(const double2* __restrict__ vhs, const double* __restrict__ expH1, int lda_e,
                            const double2* __restrict__ phi_in, double2* __restrict__ phi_out, int M, int N, int nmax,
                            int pre, int post, int nstage) {
  extern __shared__ __align__(128) unsigned char pf_sm[];
  constexpr int TS = 8 * CT + 1;
  const int RT = (M + 7) / 8, rows = 8 * RT, tid = threadIdx.x;
  const int stage_bytes = rows * kRow;
  double2* const sT = reinterpret_cast<double2*>(pf_sm + nstage * stage_bytes);
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const size_t w = blockIdx.x;
  const double2* vw = vhs + w * M * M;
  const double2* pin = phi_in + w * M * N;
  double2* pout = phi_out + w * M * N;
  const int npass = nmax + (pre ? 1 : 0) + (post ? 1 : 0);
  const int nch_e = (M + 15) / 16, nch_v = (M + 7) / 8;

  // chunk copies: 8 rows x 8 segments of 16 bytes per warp, two per thread; the segments of a
  // row are permuted so that fragment loads of 2 (complex) or 4 (real) rows hit different banks
  int lp = 0, lc = 0, ls = 0;
  auto load = [&]() {
    if (lp < npass) {
      const bool one = (pre && lp == 0) || (post && lp == npass - 1);
      unsigned char* st = pf_sm + ls * stage_bytes;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int e = tid + i * 32 * RT, r = e >> 3, seg = e & 7;
        if (one) {
          const int k = lc * 16 + 2 * seg;
          const bool in = r < M && k < M;
          cp_async16(st + r * kRow + ((seg ^ ((r & 3) << 1)) << 4), in ? expH1 + (size_t)r * lda_e + k : expH1,
                     in ? (M - k >= 2 ? 16 : 8) : 0);
        } else {
          const int k = lc * 8 + seg;
          const bool in = r < M && k < M;
          cp_async16(st + r * kRow + ((seg ^ ((r & 1) << 2)) << 4), in ? vw + (size_t)r * M + k : vw, in ? 16 : 0);
        }
      }
      ls = ls == nstage - 1 ? 0 : ls + 1;
      if (++lc == (one ? nch_e : nch_v)) {
        lc = 0;
        ++lp;
      }
    }
    cp_async_commit();
  };
  load();
  if (nstage == 3) load();
  for (int e = tid; e < stream_trows(M) * TS; e += blockDim.x) {
    const int r = e / TS, c = e - r * TS;
    sT[e] = (r < M && c < N) ? pin[(size_t)r * N + c] : make_double2(0.0, 0.0);
  }
  const int r = warp * 8 + g;
  double2 phi[PHI_REG ? CT : 1][2];
  if (PHI_REG) {
#pragma unroll
    for (int j = 0; j < CT; ++j)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = 8 * j + 4 * q + t;
        phi[j][q] = (r < M && c < N) ? pin[(size_t)r * N + c] : make_double2(0.0, 0.0);
      }
  }
  int stage = 0;
  for (int p = 0; p < npass; ++p) {
    const bool first = pre && p == 0, last = p == npass - 1, one = first || (post && last);
    double re[CT][2], im[CT][2];
#pragma unroll
    for (int j = 0; j < CT; ++j) re[j][0] = re[j][1] = im[j][0] = im[j][1] = 0.0;
    const int nch = one ? nch_e : nch_v;
    for (int c = 0; c < nch; ++c) {
      if (nstage == 3)
        cp_async_wait<1>();
      else
        cp_async_wait<0>();
      __syncthreads();  // the chunk has landed for everyone, the previous one is consumed
      load();
      const unsigned char* st = pf_sm + stage * stage_bytes + r * kRow;
      stage = stage == nstage - 1 ? 0 : stage + 1;
      if (one) {
        const int k0 = c * 16;
#pragma unroll
        for (int kk = 0; kk < 16; kk += 4) {
          if (k0 + kk >= M) break;
          const int seg = (kk + t) >> 1;
          const double a =
              *reinterpret_cast<const double*>(st + ((seg ^ ((r & 3) << 1)) << 4) + ((t & 1) << 3));
          const double2* b = sT + (k0 + kk + t) * TS + tile_col(g);
#pragma unroll
          for (int j = 0; j < CT; ++j) {
            const double2 bv = b[8 * j];
            dmma884(re[j], a, bv.x);
            dmma884(im[j], a, bv.y);
          }
        }
      } else {
        const int k0 = c * 8;
#pragma unroll
        for (int kk = 0; kk < 8; kk += 4) {
          if (k0 + kk >= M) break;
          const double2 a = *reinterpret_cast<const double2*>(st + (((kk + t) ^ ((r & 1) << 2)) << 4));
          const double2* b = sT + (k0 + kk + t) * TS + tile_col(g);
#pragma unroll
          for (int j = 0; j < CT; ++j) cmma(re[j], im[j], a.x, a.y, -a.y, b[8 * j]);
        }
      }
    }
    const bool to_post = post && p + 1 == npass - 1;
    const int term = one ? 0 : p + 1 - (pre ? 1 : 0);
    const double sc = one ? 1.0 : 1.0 / term;
    if (!last) __syncthreads();  // every warp has read the old term (the next chunk's barrier follows the writes)
#pragma unroll
    for (int j = 0; j < CT; ++j)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = 8 * j + 4 * q + t;
        const double2 v = make_double2(re[j][q] * sc, im[j][q] * sc);
        if (r >= M || c >= N) continue;  // the padding of T stays zero
        const size_t gi = (size_t)r * N + c;
        double2 s = v;  // phi after this pass
        if (PHI_REG) {
          if (!one) s = cadd(phi[j][q], v);
          phi[j][q] = s;
          if (last) pout[gi] = s;
        } else {
          if (!one) s = cadd(term == 1 && !pre ? pin[gi] : pout[gi], v);
          if (!to_post) pout[gi] = s;
        }
        if (!last) sT[r * TS + c] = to_post ? s : v;
      }
  }
  cp_async_wait<0>();
}

template <int CT, int MAXT, bool PHI_REG>
cudaError_t launch_stream_t(const double2* vhs, const double* expH1, int lda_e, const double2* phi_in,
                            double2* phi_out, int W, int M, int N, int nmax, int pre, int post, cudaStream_t st) {
  const int rows = (M + 7) / 8 * 8;
  const size_t term = sizeof(double2) * stream_trows(M) * (8 * CT + 1);
  const int nstage = 3 * (size_t)rows * kRow + term <= 227 * 1024 ? 3 : 2;
  const size_t smem = nstage * (size_t)rows * kRow + term;
  if (smem > 227 * 1024) return cudaErrorInvalidValue;
  auto k = propagate_stream_kernel<CT, MAXT, PHI_REG>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<W, 4 * rows, smem, st>>>(vhs, expH1, lda_e, phi_in, phi_out, M, N, nmax, pre, post, nstage);
  note_launch();
  return cudaGetLastError();
}

// Threads are 4 per row (one warp per 8 rows): the register bound of each width.
template <int CT>
cudaError_t launch_stream(const double2* vhs, const double* expH1, int lda_e, const double2* phi_in, double2* phi_out,
                          int W, int M, int N, int nmax, int pre, int post, cudaStream_t st) {
  constexpr bool REG = CT <= 2;
  if (M <= 128)
    return launch_stream_t<CT, 512, true>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
  if (M <= 160)
    return launch_stream_t<CT, 640, REG>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
  if (M <= 208)
    return launch_stream_t<CT, 832, REG>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
  return launch_stream_t<CT, 1024, false>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
}

}  // namespace

// Returns cudaErrorInvalidValue for shapes it does not cover (M > 256, N > 32); callers then use
// the per-term GEMM path.  expH1: real (M x lda_e) row-major with lda_e even (16-byte aligned rows
// for the cp.async staging); may be null when pre = post = 0.
cudaError_t launch_propagate_fused(const double2* vhs, const double* expH1, int lda_e, const double2* phi_in,
                                   double2* phi_out, int W, int M, int N, int nmax, int pre, int post, cudaStream_t st) {
  if (M <= 0 || M > 256 || N <= 0 || N > 32 || nmax < 1 || phi_in == phi_out) return cudaErrorInvalidValue;
  if ((pre || post) && (expH1 == nullptr || (lda_e & 1) || lda_e < M)) return cudaErrorInvalidValue;
  if (M <= kResM) {
    // one column tile per warp while that leaves at most 16 warps, else two
    const int rt = (M + 7) / 8, ct = (N + 7) / 8;
    if (rt * ct <= 16)
      return launch_resident<1>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
    return launch_resident<2>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
  }
  switch ((N + 7) / 8) {
    case 1: return launch_stream<1>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
    case 2: return launch_stream<2>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
    case 3: return launch_stream<3>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
    default: return launch_stream<4>(vhs, expH1, lda_e, phi_in, phi_out, W, M, N, nmax, pre, post, st);
  }
}

}  // namespace ipie_b200
