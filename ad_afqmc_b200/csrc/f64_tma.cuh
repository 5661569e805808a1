// Persistent FP64 tensor-core (DMMA m8n8k4) GEMM fed by TMA.
//
//   D (M x N) = A (M x K) . B (K x N)            real, or
//   D = (Ar + i Ai) . B                          B's columns interleaved (re, im)
//
// One producer warp streams 16-wide K stages into a shared-memory ring, running
// ahead over tile boundaries; 4 x WN consumer warps each own FM 8-row tiles and
// NG 16-column groups.  What the layouts are chosen for:
//  * A arrives as two boxes of BM rows x 8 doubles (64-byte rows, no swizzle).
//    Lane (g, t) reads row g, k = 2t and 2t + 1 in one 16-byte load: a warp reads
//    512 consecutive bytes.  So the first MMA of eight K takes k = 0, 2, 4, 6 and the
//    second k = 1, 3, 5, 7 (B follows).
//  * B (n contiguous) arrives as boxes of 16 rows x 16 columns, 128-byte swizzled;
//    lane (g, t) reads row 2t (2t + 1), columns 2g and 2g + 1 in one load without
//    conflicts.  Column 2g goes to the group's first MMA tile and 2g + 1 to its
//    second, so a lane ends up with four consecutive columns, and an interleaved
//    complex column gives re and im of the same number: the product with i z is
//    the same registers exchanged, one negated.
//  * B (k contiguous) is laid out like A; lane (g, t) reads rows 4 (g / 2) + g % 2 and the
//    row two further on for the group's two MMA tiles, so that a lane ends up with four
//    consecutive columns here too.  Its rows may be fewer than the tile's columns (F64Tile's
//    LIVE): MMA tiles of eight columns beyond them are left out, and a group of which eight
//    are in use takes them in order.
// Registers-only DMMA runs at 36.5 TF/s on this chip; a cp.async main loop with
// address arithmetic in every warp and a block barrier per stage reached 22.4.
// Measured, that loop -> this, N = 200, No = 40, G = 1000, 512 walkers, per step: VHS 3.65 ->
// 2.65 ms (31 TF/s), propagator 3.50 -> 1.79 ms, force bias 0.77 -> 0.52 ms; exchange 30.1 ->
// 24.0 ms.  N = 95, G = 471, 161 walkers, per block of ten steps: VHS 2.15 -> 1.23 ms,
// propagator 5.20 -> 1.25 ms.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "umma.cuh"

namespace afq {

enum { F64_REAL = 0, F64_COMPLEX = 1 };
enum { F64_B_N = 0, F64_B_K = 1 };  // B contiguous along n, or along k

struct F64Shape {
  int K;               // summed length
  int mt, nt, nz;      // tiles along rows and columns, batches (or K splits)
  int arow_step;       // rows of A per tile
  int a_batched;       // A's third coordinate follows the batch
  int brow_step;       // B_K: rows of B (columns of D) per tile, also the height of its box
  int ksplit;          // nz splits K into chunks of this length (0: no split)
  int stages;
  int epi_bytes;       // shared memory of the epilogue
  int* err;
};

template <class Epi>
struct F64Params {
  CUtensorMap ta, ta2, tb;
  F64Shape s;
  Epi epi;
};

// LIVE: brow_step may be less than BN
template <int FM_, int WN_, int NG_, int KIND_, int BMODE_, bool LIVE_ = false>
struct F64Tile {
  static constexpr int FM = FM_, WN = WN_, NG = NG_, KIND = KIND_, BMODE = BMODE_;
  static constexpr bool LIVE = LIVE_;
  static constexpr int BM = 32 * FM, GROUPS = WN * NG, BN = 16 * GROUPS;
  static constexpr int CW = 4 * WN;                     // consumer warps
  static constexpr int NT = 32 * (CW + 1);
  static constexpr uint32_t A_BYTES = BM * 16 * 8;      // one matrix, one stage
  static constexpr uint32_t B_BYTES = BN * 16 * 8;
  static constexpr uint32_t STAGE = A_BYTES * (KIND == F64_COMPLEX ? 2 : 1) + B_BYTES;
};

struct F64At {
  int mti, nti, z;
};

// Epi: template <class T> __device__ void tile(const F64At&, double2 (&acc)[FM][NG][2], int wm, int wn, ...)
template <class T, class Epi>
__global__ void __launch_bounds__(T::NT, 1) f64_gemm_kernel(const __grid_constant__ F64Params<Epi> P) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem =
      reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int ST = P.s.stages;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + size_t(ST) * T::STAGE);
  uint64_t* empty = full + ST;
  volatile int* abort_s = reinterpret_cast<volatile int*>(empty + ST);
  uint8_t* epi_smem = reinterpret_cast<uint8_t*>(full) + 256;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], T::CW);
    }
    *abort_s = 0;
    fence_barrier_init();
  }
  __syncthreads();
  const int tiles = P.s.mt * P.s.nt * P.s.nz;
  const uint32_t tx = T::LIVE ? T::STAGE - T::B_BYTES + P.s.brow_step * 128 : T::STAGE;  // bytes per stage
  auto locate = [&](int t) {
    F64At a;
    a.nti = t % P.s.nt;
    const int r = t / P.s.nt;
    a.mti = r % P.s.mt;
    a.z = r / P.s.mt;
    return a;
  };
  auto krange = [&](const F64At& a, int& k0, int& kt) {
    k0 = P.s.ksplit ? a.z * P.s.ksplit : 0;
    const int k1 = P.s.ksplit ? min(P.s.K, k0 + P.s.ksplit) : P.s.K;
    kt = (k1 - k0 + 15) >> 4;
  };

  if (warp == T::CW) {
    Ring ring{full, empty, ST};
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      const F64At a = locate(t);
      int k0, kt;
      krange(a, k0, kt);
      const int arow = a.mti * P.s.arow_step;
      const int zb = P.s.ksplit ? 0 : a.z;
      const int az = P.s.a_batched ? a.z : 0;
      const bool ok = ring_fill(ring, kt, abort_s, P.s.err, [&](int stage, int kb) {
        mbar_arrive_expect_tx(&full[stage], tx);
        uint8_t* sa = smem + stage * T::STAGE;
        const int k = k0 + kb * 16;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tma_load_3d(sa + h * (T::A_BYTES / 2), &P.ta, &full[stage], k + 8 * h, arow, az);
          if (T::KIND == F64_COMPLEX)
            tma_load_3d(sa + T::A_BYTES + h * (T::A_BYTES / 2), &P.ta2, &full[stage], k + 8 * h, arow, az);
        }
        uint8_t* sb = sa + T::STAGE - T::B_BYTES;
        if (T::BMODE == F64_B_K) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
            tma_load_3d(sb + h * (T::B_BYTES / 2), &P.tb, &full[stage], k + 8 * h, a.nti * P.s.brow_step, 0);
        } else {
          for (int q = 0; q < T::GROUPS; ++q)
            tma_load_3d(sb + q * 2048, &P.tb, &full[stage], (a.nti * T::GROUPS + q) * 16, k, zb);
        }
      });
      if (!ok) break;
    }
    ring_drain(ring, full);
  } else {
    const int wm = warp & 3, wn = warp >> 2;
    const int g = lane >> 2, t4 = lane & 3;
    // byte offsets of this lane's fragments inside a stage
    const uint32_t a_off = (wm * T::FM * 8 + g) * 64 + t4 * 16;
    const uint32_t b_off0 = T::BMODE == F64_B_N ? (2 * t4) * 128 + ((g ^ (2 * t4)) << 4) : (4 * (g >> 1) + (g & 1)) * 64 + t4 * 16;
    const uint32_t b_off1 = (2 * t4 + 1) * 128 + ((g ^ (2 * t4 + 1)) << 4);
    Ring ring{full, empty, ST};
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      const F64At at = locate(t);
      int k0, kt;
      krange(at, k0, kt);
      double acc[T::FM][T::NG][2][2];
#pragma unroll
      for (int i = 0; i < T::FM; ++i)
#pragma unroll
        for (int n = 0; n < T::NG; ++n)
          acc[i][n][0][0] = acc[i][n][0][1] = acc[i][n][1][0] = acc[i][n][1][1] = 0.0;
      // the K loop with the first LV of this warp's MMA tiles (eight columns each)
      auto kloop = [&](auto lv) {
        constexpr int LV = decltype(lv)::value;
#pragma unroll 1
        for (int kb = 0; kb < kt; ++kb) {
          mbar_wait_run_on(&full[ring.stage], ring.phase, abort_s, P.s.err);
          const uint8_t* sa = smem + ring.stage * T::STAGE;
          const uint8_t* sb = sa + T::STAGE - T::B_BYTES;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            // b[n][ks][j]: MMA tile j of group n, k step ks
            double b[T::NG][2][2];
#pragma unroll
            for (int n = 0; n < T::NG; ++n) {
              if (2 * n >= LV) continue;
              const int q = wn * T::NG + n;
              if (T::BMODE == F64_B_N) {
                const double2 u = *reinterpret_cast<const double2*>(sb + q * 2048 + h * 1024 + b_off0);
                const double2 v = *reinterpret_cast<const double2*>(sb + q * 2048 + h * 1024 + b_off1);
                b[n][0][0] = u.x; b[n][0][1] = u.y;
                b[n][1][0] = v.x; b[n][1][1] = v.y;
              } else {
                const bool half = 2 * n + 1 >= LV;
                const uint8_t* p = sb + h * (T::B_BYTES / 2) + q * 1024 + (half ? g * 64 + t4 * 16 : b_off0);
                const double2 u = *reinterpret_cast<const double2*>(p);
                b[n][0][0] = u.x; b[n][1][0] = u.y;
                if (!half) {
                  const double2 v = *reinterpret_cast<const double2*>(p + 128);
                  b[n][0][1] = v.x; b[n][1][1] = v.y;
                }
              }
            }
#pragma unroll
            for (int i = 0; i < T::FM; ++i) {
              if (LV == 0) continue;
              const double2 a = *reinterpret_cast<const double2*>(sa + h * (T::A_BYTES / 2) + a_off + i * 512);
#pragma unroll
              for (int n = 0; n < T::NG; ++n) {
                if (2 * n < LV) dmma_8x8x4(acc[i][n][0][0], acc[i][n][0][1], a.x, b[n][0][0]);
                if (2 * n + 1 < LV) dmma_8x8x4(acc[i][n][1][0], acc[i][n][1][1], a.x, b[n][0][1]);
              }
#pragma unroll
              for (int n = 0; n < T::NG; ++n) {
                if (2 * n < LV) dmma_8x8x4(acc[i][n][0][0], acc[i][n][0][1], a.y, b[n][1][0]);
                if (2 * n + 1 < LV) dmma_8x8x4(acc[i][n][1][0], acc[i][n][1][1], a.y, b[n][1][1]);
              }
            }
            if (T::KIND == F64_COMPLEX) {
#pragma unroll
              for (int i = 0; i < T::FM; ++i) {
                const double2 a = *reinterpret_cast<const double2*>(sa + T::A_BYTES + h * (T::A_BYTES / 2) +
                                                                    a_off + i * 512);
#pragma unroll
                for (int n = 0; n < T::NG; ++n) {
                  dmma_8x8x4(acc[i][n][0][0], acc[i][n][0][1], -a.x, b[n][0][1]);
                  dmma_8x8x4(acc[i][n][1][0], acc[i][n][1][1], a.x, b[n][0][0]);
                }
#pragma unroll
                for (int n = 0; n < T::NG; ++n) {
                  dmma_8x8x4(acc[i][n][0][0], acc[i][n][0][1], -a.y, b[n][1][1]);
                  dmma_8x8x4(acc[i][n][1][0], acc[i][n][1][1], a.y, b[n][1][0]);
                }
              }
            }
          }
          // every lane's reads of the stage complete before the TMA that refills it
          // (generic reads, async-proxy writes: without the fence short stages were
          // overwritten under a warp's last loads)
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[ring.stage]);
          ring.advance();
        }
      };
      if (!T::LIVE) {
        kloop(std::integral_constant<int, 2 * T::NG>{});
      } else {  // warp-uniform
        const int live = (P.s.brow_step + 7) / 8 - wn * 2 * T::NG;
        if (live >= 2 * T::NG)
          kloop(std::integral_constant<int, 2 * T::NG>{});
        else if (T::NG > 1 && live == 3)
          kloop(std::integral_constant<int, (T::NG > 1 ? 3 : 0)>{});
        else if (T::NG > 1 && live == 2)
          kloop(std::integral_constant<int, (T::NG > 1 ? 2 : 0)>{});
        else if (live == 1)
          kloop(std::integral_constant<int, 1>{});
        else
          kloop(std::integral_constant<int, 0>{});
      }
      P.epi.template tile<T>(at, acc, wm, wn, g, t4, epi_smem);
    }
  }
}

// Calls f(row, col, v) for the lane's accumulators of one tile: v holds the four
// consecutive columns col .. col + 3 (interleaved: two complex numbers), row and col relative
// to the tile.  (LIVE: see exch_stage.)
template <class T, class F>
__device__ __forceinline__ void f64_each(double (&acc)[T::FM][T::NG][2][2], int wm, int wn, int g, int t4,
                                         F&& f) {
#pragma unroll
  for (int i = 0; i < T::FM; ++i)
#pragma unroll
    for (int n = 0; n < T::NG; ++n) {
      const int row = (wm * T::FM + i) * 8 + g, c = (wn * T::NG + n) * 16 + 4 * t4;
      if (T::BMODE == F64_B_N)
        f(row, c, acc[i][n][0][0], acc[i][n][1][0], acc[i][n][0][1], acc[i][n][1][1]);
      else
        f(row, c, acc[i][n][0][0], acc[i][n][0][1], acc[i][n][1][0], acc[i][n][1][1]);
    }
}

// host side ------------------------------------------------------------------
// 3-D map of doubles: dims {x, y, z}, strides in doubles (even), box {bx, by, 1};
// swizzled for boxes of 16 doubles
int make_tmap_f64(CUtensorMap* map, const void* base, long long x, long long y, long long z,
                  long long ystride, long long zstride, int bx, int by);

constexpr size_t kF64SmemBudget = 227 * 1024;

// stages of a launch of `per` CTAs an SM
template <class T>
inline int f64_stages(size_t epi_bytes, int per = 1) {
  for (int st = 6; st >= 2; --st)
    if (1024 + st * size_t(T::STAGE) + 256 + epi_bytes <= kF64SmemBudget / per) return st;
  return 0;
}

template <class T, class Epi>
cudaError_t f64_launch(F64Params<Epi>& P, int ctas, cudaStream_t st) {
  if (P.s.stages == 0) P.s.stages = f64_stages<T>(P.s.epi_bytes);
  if (P.s.stages < 2) return cudaErrorInvalidValue;
  const size_t smem = 1024 + P.s.stages * size_t(T::STAGE) + 256 + P.s.epi_bytes;
  cudaError_t e = allow_smem(f64_gemm_kernel<T, Epi>, smem);
  if (e != cudaSuccess) return e;
  const long long tiles = (long long)P.s.mt * P.s.nt * P.s.nz;
  if (tiles >= (1LL << 31)) return cudaErrorInvalidValue;
  f64_gemm_kernel<T, Epi><<<(int)(tiles < ctas ? tiles : ctas), T::NT, smem, st>>>(P);
  return cudaGetLastError();
}

}  // namespace afq
