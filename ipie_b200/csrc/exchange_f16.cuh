// Exchange of the mixed-precision energy with the walkers' Green's functions held in tensor memory
// (M <= 256 and more than a tile or two per SM, see exchange_streams in mixed.cu; the rest takes
// umma_gemm_kernel<EpiExchange>):
//
//     raw_w = sum_x sum_ij T_ij T_ji,      T = L_x G_w^T (N x N complex),
//
// as a 3-pass binary16 product of the padded planar Green's function rows (w, re/im, j) with the padded
// half-rotated Cholesky rows (x, i), both K-major with Mp halves per row.
//
// One persistent CTA per SM.  The 128 rows (w, c, j) of a walker tile are the left operand and stay in
// tensor memory (head and remainder, 8 columns per 16 K and plane) while 128-row tiles of the Cholesky
// operand stream through a TMA ring of two 64 KB stages as the right operand, so a tile reads half the bytes
// from L2 and a third of the shared memory that two streamed operands would.  A CTA reloads the left
// operand when it enters a walker tile and leaves one partial per walker behind when it leaves it.
//
// The product accumulates 128 K at a time into one of two TMEM buffers, as umma_gemm_kernel does (FP32
// truncation, see there).  Eight epilogue warps drain it: warp w takes TMEM lanes 32 (w % 4) .. + 31, a row
// (w, c, j) per thread, and 64 columns (w / 4), that is 64 / NP vectors x.  They park the values in shared
// memory; a thread then multiplies its own T^c_ij (registers) with T^c_ji (row i, its column j) and, for
// half of its vectors, with the other component's T_ji:
//     re = sum_ij (re_ij re_ji - im_ij im_ji),      im = 2 sum_ij re_ij im_ji = 2 sum_ij im_ij re_ji,
// 96 loads and multiply-adds per thread where a lane per column and component pairs took 256 and 512.
// 32 products at a time are summed in FP32, the rest in FP64 per lane until the run leaves the walker.
//
// What bounds it: the tensor pipe (39 products of 128 x 128 x 16 per tile at M = 200; the products alone,
// without copies and epilogue, take 5.6 ms of the 7.2 below).  Three things cost the issuing warp: a
// lane-0 branch around the products (140 cycles each to issue; an elected lane of a converged warp
// 117), a commit per 32 KB stage and per chunk (~550 cycles apiece; one per 64 KB stage that is also the chunk
// takes the empty pipeline from 4.7 to 2.7 ms), and CTAs at different places of the Cholesky rows.
// 2048 walkers, M = 200, N = 32, X = 1600: 12.3 -> 7.2 ms (1120 TFLOP/s executed); 512, M = 76, N = 10, X = 400:
// 206 -> 74 us, against streaming both operands through umma_gemm_kernel with one epilogue warp group.
#pragma once

#include "umma_gemm.cuh"

namespace ipie_b200 {
namespace umma {

// 128 x N x 16 FP16 product with the left operand in tensor memory (row = lane, two K per column)
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(
          d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

struct ExTmemShape {
  static constexpr int BN = 128, STAGES = 2;
  static constexpr int TILE = BN * 128;        // 64 K of one plane
  static constexpr int BLOCK_BYTES = 2 * TILE;  // both planes
  static constexpr int STAGE_BYTES = 2 * BLOCK_BYTES;  // 128 K, one chunk of the accumulation
  static constexpr int EPI_WARPS = 8, PRODUCERS = 2, THREADS = 32 * (EPI_WARPS + PRODUCERS + 1);
  static constexpr int MMA_WARP = EPI_WARPS + PRODUCERS;
  static constexpr int LD = 68;                // floats per parked row (4 mod 32: 16-byte stores free of conflicts)
  static constexpr int PARK_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int RED_OFFSET = PARK_OFFSET + 2 * kBM * LD * 4;
  static constexpr int BAR_OFFSET = RED_OFFSET + 2 * EPI_WARPS * 2 * 16;
  static constexpr int SMEM_BYTES = 1024 + BAR_OFFSET + 256;
  static constexpr int A_COL = 2 * BN;         // first TMEM column of the left operand
  static constexpr int MAX_K = 256;            // 2 planes x 128 columns
  static_assert(SMEM_BYTES <= 232448, "shared memory per CTA exceeded");
};

// Who computes which of the nwt x nxt tiles: CTA b takes the whole walker tiles b, b + g, ... of the full
// rounds, then its share of the tiles of the walker tiles left over (x fastest, g contiguous runs of nearly
// equal length).  So the CTAs sweep the Cholesky rows together through the full rounds and read each
// of them at about the same time.
struct ExRuns {
  int nwt, nxt, g;
  __host__ __device__ int rounds() const { return nwt / g; }
  __host__ __device__ long long left() const { return (long long)(nwt % g) * nxt; }
  // runs of the tiles left over (none is empty) and the first tile of run b
  __host__ __device__ int nruns() const { return left() < g ? (int)left() : g; }
  __host__ __device__ long long first(int b) const { return b < nruns() ? left() * b / nruns() : left(); }
  // the run that holds tile t of those: the largest b with first(b) <= t
  __host__ __device__ int run_of(long long t) const { return (int)(((t + 1) * nruns() - 1) / left()); }
  // partials a walker can get: the runs its nxt tiles may touch
  __host__ __device__ int rows() const {
    if (left() == 0) return 1;
    const int len = (int)(left() / nruns());  // the shorter runs
    const int n = (nxt - 1) / len + 2;
    return n < nxt ? n : nxt;
  }
};

inline ExRuns exchange_tmem_runs(int W, int X, int NP, int sms) {
  ExRuns r;
  r.nwt = (W * 2 * NP + kBM - 1) / kBM;
  r.nxt = (X * NP + kBM - 1) / kBM;
  const long long t = (long long)r.nwt * r.nxt;
  r.g = t < sms ? (int)t : sms;
  return r;
}

template <int NP>
__global__ void __launch_bounds__(ExTmemShape::THREADS, 1)
    exchange_tmem_kernel(const __grid_constant__ GemmMaps maps, const __half* __restrict__ g_hi,
                         const __half* __restrict__ g_lo, int K, int Mp, ExRuns runs, int W, double inv_rscale2,
                         const double* __restrict__ walker_scale, int rows, double2* __restrict__ part,
                         unsigned* status) {
  using S = ExTmemShape;
  constexpr int WT = kBM / (2 * NP);  // walkers per tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  double2* red = reinterpret_cast<double2*>(smem + S::RED_OFFSET);  // [2][EPI_WARPS][2]
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::BAR_OFFSET);
  uint64_t* done = full + S::STAGES;    // [2] chunk accumulated: its stage is free, its buffer readable
  uint64_t* cempty = done + S::STAGES;  // [2] chunk drained
  uint64_t* aready = cempty + 2;        // left operand of the next walker tile in place
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aready + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&done[s], 1);
      mbar_init(&cempty[s], S::EPI_WARPS);
    }
    mbar_init(aready, 4);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  constexpr int KC = 128;        // K per chunk
  const int ks = (K + 15) / 16;  // K steps
  const int nchunks = (K + KC - 1) / KC;
  // this CTA's tiles: `whole` of whole walker tiles, then up to `tiles` from x tile xr of walker tile unitr
  const int nxt = runs.nxt, whole = runs.rounds() * nxt;
  const long long r0 = runs.first((int)blockIdx.x);
  const int tiles = whole + (int)(runs.first((int)blockIdx.x + 1) - r0);
  const int unitr = runs.rounds() * runs.g + (int)(r0 / nxt), xr = (int)(r0 % nxt);

  if (warp >= S::EPI_WARPS && warp < S::MMA_WARP) {
    if (lane == 0) {
      const uint32_t chunks = (uint32_t)tiles * nchunks;
      for (uint32_t c = warp - S::EPI_WARPS; c < chunks; c += S::PRODUCERS) {
        const uint32_t s = c & 1, r = c >> 1;
        if (r > 0 && !mbar_wait(&done[s], (r - 1) & 1, abort_flag, status)) break;
        const uint32_t tile = c / (uint32_t)nchunks;
        const uint32_t x = ((int)tile < whole ? tile : tile - whole + xr) % (uint32_t)nxt;
        const int brow = (int)x * S::BN, k0 = (int)(c - tile * nchunks) * KC;
        uint8_t* st = smem + s * S::STAGE_BYTES;
        const int blocks = K - k0 > 64 ? 2 : 1;
        mbar_expect_tx(&full[s], blocks * S::BLOCK_BYTES);
        for (int q = 0; q < blocks; ++q, st += S::BLOCK_BYTES) {
          if (maps.b_planes) {
            tma_load_3d(st, &maps.b_hi, k0 + 64 * q, brow, 0, &full[s]);
          } else {
            tma_load_2d(st, &maps.b_hi, k0 + 64 * q, brow, &full[s]);
            tma_load_2d(st + S::TILE, &maps.b_lo, k0 + 64 * q, brow, &full[s]);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == S::MMA_WARP) {
    // the whole warp runs the loop and one elected lane issues: addresses and descriptors stay
    // warp-uniform
    {
      constexpr uint32_t idesc = idesc_f16(kBM, S::BN);
      const uint32_t a_hi = tmem + S::A_COL, a_lo = a_hi + 8 * ks;
      uint32_t c = 0, units = 0;
      bool ok = true;
      for (int t = 0, x = 0; t < tiles && ok; ++t, x = x + 1 == nxt ? 0 : x + 1) {
        if (t == whole) x = xr;
        if (t == 0 || t == whole || x == 0) {
          if (!mbar_wait_warp(aready, units & 1, abort_flag, status)) break;
          ++units;
        }
        for (int ch = 0; ch < nchunks; ++ch, ++c) {
          const uint32_t s = c & 1, r = c >> 1;
          if ((r > 0 && !mbar_wait_warp(&cempty[s], (r - 1) & 1, abort_flag, status)) ||
              !mbar_wait_warp(&full[s], r & 1, abort_flag, status)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem + s * S::BN;
          const int steps = min(KC / 16, ks - ch * (KC / 16));
          const uint32_t ah = a_hi + ch * (KC / 2), al = a_lo + ch * (KC / 2);
          const uint64_t b0 = desc_kmajor_sw128(smem + s * S::STAGE_BYTES);
#pragma unroll
          for (int k = 0; k < KC / 16; ++k) {
            if (k >= steps) break;
            // (descriptor addresses count 16 bytes)
            const uint64_t b_hi = b0 + (k >> 2) * (S::BLOCK_BYTES >> 4) + 2 * (k & 3), b_lo = b_hi + (S::TILE >> 4);
            if (elect_one()) {
              mma_f16_ts(d, ah + 8 * k, b_hi, idesc, k > 0 ? 1u : 0u);
              mma_f16_ts(d, ah + 8 * k, b_lo, idesc, 1u);
              mma_f16_ts(d, al + 8 * k, b_hi, idesc, 1u);
            }
          }
          if (elect_one()) mma_commit(&done[s]);
        }
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3, group = warp >> 2;
    const int row = quarter * 32 + lane;
    const int comp = (row / NP) & 1, j = row % NP;
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
    // rows of one component start 0 mod 32 banks apart: their columns are rotated by NP instead
    auto swz = [](int r) { return ((r / NP) & (32 / NP - 1)) * NP; };
    float* park = reinterpret_cast<float*>(smem + S::PARK_OFFSET) + group * (kBM * S::LD);
    const int own0 = row - j, other0 = comp ? own0 - NP : own0 + NP;
    const float* own = park + own0 * S::LD + j;
    const float* other = park + other0 * S::LD + j;
    const int own_swz = swz(own0), other_swz = swz(other0);
    auto load_a = [&](int unit) {  // (group 0: one thread per row)
      const long long gr = (long long)unit * kBM + row;
      const bool in = gr < (long long)W * 2 * NP;
      const uint4* ph = reinterpret_cast<const uint4*>(g_hi + gr * Mp);
      const uint4* pl = reinterpret_cast<const uint4*>(g_lo + gr * Mp);
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 2
      for (int k = 0; k < ks; ++k) {
        const bool second = in && 16 * k + 8 < Mp;
        const uint4 h0 = in ? ph[2 * k] : zero, h1 = second ? ph[2 * k + 1] : zero;
        const uint4 l0 = in ? pl[2 * k] : zero, l1 = second ? pl[2 * k + 1] : zero;
        const uint32_t h[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
        const uint32_t l[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
        tmem_st8(lanes + S::A_COL + 8 * k, h);
        tmem_st8(lanes + S::A_COL + 8 * (ks + k), l);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cta(aready);
    };
    // the warps that read each other's parked rows
    auto walker_sync = [&]() {
      if (NP == 32)
        asm volatile("bar.sync %0, 64;\n" ::"r"(1 + group * 2 + (quarter >> 1)) : "memory");
      else
        __syncwarp();
    };
    if (group == 0 && tiles > 0) load_a(whole > 0 ? (int)blockIdx.x : unitr);
    uint32_t c = 0;
    int parity = 0;
    double dr = 0.0, di = 0.0;
    // a wait that gives up leaves ok false for the rest: no more tensor-memory reads, every barrier kept
    bool ok = true;
    for (int t = 0, x = 0, unit = (int)blockIdx.x; t < tiles; ++t) {
      if (t == whole) {
        x = xr;
        unit = unitr;
      }
      const bool last = t + 1 == tiles || x + 1 == nxt;
      float v[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) v[i] = 0.0f;
      for (int ch = 0; ch < nchunks; ++ch, ++c) {
        const uint32_t buf = c & 1;
        if (ok && !mbar_wait(&done[buf], (c >> 1) & 1, abort_flag, status)) ok = false;
        ok = __all_sync(0xffffffffu, ok) != 0;  // tcgen05.ld is warp-collective
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float d[32];
          tmem_ld32(lanes + buf * S::BN + group * 64 + q * 32, d);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[q * 32 + i] += d[i];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cta(&cempty[buf]);  // one arrival per warp
      }
      // the last products of this walker tile are complete: the next one's rows replace the operand
      if (ok && last && t + 1 < tiles && group == 0)
        load_a(t + 1 == whole ? unitr : t < whole ? unit + runs.g : unit + 1);
      walker_sync();  // the previous tile's rows are read
      {
        float* dst = park + row * S::LD;
        const int sw = own_swz;
#pragma unroll
        for (int q = 0; q < 16; ++q)
          *reinterpret_cast<float4*>(dst + ((4 * q) ^ sw)) =
              make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      }
      walker_sync();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float f0 = 0.0f, f1 = 0.0f;
#pragma unroll
        for (int xb = 0; xb < 32 / NP; ++xb) {
          const float* p = own + ((h * 32 + xb * NP) ^ own_swz);
#pragma unroll
          for (int i = 0; i < NP; i += 2) {
            f0 = fmaf(v[h * 32 + xb * NP + i], p[i * S::LD], f0);
            f1 = fmaf(v[h * 32 + xb * NP + i + 1], p[(i + 1) * S::LD], f1);
          }
        }
        dr += (double)(f0 + f1);
      }
      {
        // the other component: the real rows take the first 32 columns, the imaginary ones the rest
        float f0 = 0.0f, f1 = 0.0f;
#pragma unroll
        for (int xb = 0; xb < 32 / NP; ++xb) {
          const float* p = other + ((comp * 32 + xb * NP) ^ other_swz);
#pragma unroll
          for (int i = 0; i < NP; i += 2) {
            const float a0 = comp ? v[32 + xb * NP + i] : v[xb * NP + i];
            const float a1 = comp ? v[32 + xb * NP + i + 1] : v[xb * NP + i + 1];
            f0 = fmaf(a0, p[i * S::LD], f0);
            f1 = fmaf(a1, p[(i + 1) * S::LD], f1);
          }
        }
        di += (double)(f0 + f1);
      }
      if (last) {
        // one partial per walker: lanes, then the warps that hold the walker's rows and vectors
        double sr = comp ? -dr : dr, si = di;
        dr = di = 0.0;
        constexpr int SPAN = NP == 8 ? 16 : 32;  // lanes of one walker
#pragma unroll
        for (int o = SPAN / 2; o > 0; o >>= 1) {
          sr += __shfl_xor_sync(0xffffffffu, sr, o);
          si += __shfl_xor_sync(0xffffffffu, si, o);
        }
        double2* rd = red + parity * (2 * S::EPI_WARPS);
        parity ^= 1;
        if (lane % SPAN == 0) rd[2 * warp + lane / SPAN] = make_double2(sr, si);
        asm volatile("bar.sync 5, 256;\n" ::: "memory");
        const int w = unit * WT + (int)threadIdx.x;
        if (threadIdx.x < WT && w < W) {
          constexpr int WARPS = NP == 32 ? 2 : 1;  // warps of a group that share a walker
          const int w0 = NP == 8 ? (int)threadIdx.x / 2 : (int)threadIdx.x * WARPS;
          const int sub = NP == 8 ? (int)threadIdx.x & 1 : 0;
          double2 s = make_double2(0.0, 0.0);
#pragma unroll
          for (int gq = 0; gq < 2; ++gq)
#pragma unroll
            for (int q = 0; q < WARPS; ++q) s = cadd(s, rd[2 * (4 * gq + w0 + q) + sub]);
          // undo the operand scales: T = acc / (s_r s_w), the sum is quadratic in T
          const double iw = 1.0 / walker_scale[w], f = inv_rscale2 * iw * iw;
          const int slot =
              t < whole ? 0 : (int)blockIdx.x - runs.run_of((long long)(unit - runs.rounds() * runs.g) * nxt);
          part[(size_t)slot * W + w] = make_double2(f * s.x, 2.0 * f * s.y);
          if (x + 1 == nxt)  // nobody comes after: rows left over are zero
            for (int q = slot + 1; q < rows; ++q) part[(size_t)q * W + w] = make_double2(0.0, 0.0);
        }
      }
      if (++x == nxt) {
        x = 0;
        unit += t < whole ? runs.g : 1;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace umma
}  // namespace ipie_b200
