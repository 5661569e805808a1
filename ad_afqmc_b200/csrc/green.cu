// Overlap, half-rotated Green's function and one-body energy per walker.
//
// One CTA per (walker, spin sector).  For a walker W (N x No, complex) and
// a real trial C (N x No):
//   S     = C^T W                       (No x No)
//   det S , S^-1  by in-place Gauss-Jordan with partial pivoting
//            (pivot = first max of |re|+|im|, as LAPACK izamax)
//   Theta = W S^-1                      (N x No)  -> energy operand
//   G     = Theta^T                     (No x N)  -> force-bias operand
//   E1    = sum_ij G[i,j] rot_h1[i,j]
// Follows rhf._calc_green (wavefunctions.py:1089-1100), uhf._calc_green
// (:1289-1312), rhf/uhf overlaps (:1064-1074, :1259-1268) and the one-body
// part of the energies (:1128-1174, :1331-1363).  All arithmetic is FP64.
#include "common.cuh"
#include "gauss_jordan.cuh"
#include "ops.h"
#include "profile.cuh"

namespace afq {

namespace {

constexpr int kRowChunk = 32;

// asynchronous global -> shared copies (Ampere-style cp.async): the next
// chunk of walker rows streams in while the current one is multiplied
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// wait until at most one group (the newest) of this thread's copies is in flight
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// mode 0: the whole computation; 1: S = C^T W only, into a.sbuf; 2: Theta
// and its outputs from S^-1 in a.sbuf (the inverse and det by gj_kernel).
// T threads: one warp per column tile of 8 real columns (2 No of them), at least
// eight (see green_threads).
// What bounds it: the FP64 tensor cores and the instructions around them (18 us for
// S and 36 us for Theta of the former at N = 200, No = 40, 512 walkers).  The warp's tile of
// S^-1 is laid out once in registers for all rows of Theta, and the inner loops
// hold loads and MMAs only: entries beyond the matrices are read as they stand
// where they reach nothing that is stored.  S + Theta there 177 -> 125 us, at N = 300,
// No = 60 + 58, 1024 walkers 2.26 -> 1.72 ms, with every fragment rebuilt and
// range-checked for each MMA before.
template <int T>
__device__ __forceinline__ void green_body(const GreenArgs& a, int mode, int w, int sct) {
  extern __shared__ double2 sm[];
  const GreenSector& S_ = a.sec[sct];
  const int N = a.N, no = S_.no, tid = threadIdx.x;
  // row tiles of S and k-steps of Theta at the widest No of this T (green_threads)
  constexpr int MT = T == 256 ? 4 : (T == 320 ? 5 : (T == 384 ? 6 : 8));
  constexpr int KS = 4 * MT;

  double2* S = sm;                          // no*no
  double2* colk = S + no * no;              // 64
  // two buffers each of walker rows and trial rows (chunk c in buffer c & 1);
  // walker rows at a stride of sd doubles, sd = 4 (mod 16): the 8-byte
  // fragment loads of a warp (8 rows x 4 columns, or 4 rows x 8 columns) then
  // take the minimum two shared-memory wavefronts
  const int nc2_ = 2 * no;
  const int sd = nc2_ + ((20 - nc2_ % 16) % 16);
  const int sbuf_ = kRowChunk * (sd / 2);  // double2 per buffer
  double2* stage = colk + 64;                                            // 2 x sbuf_
  double* moc = reinterpret_cast<double*>(stage + 2 * sbuf_);             // 2 x kRowChunk*no
  double2* tstage = reinterpret_cast<double2*>(moc + 2 * kRowChunk * no);
  const int ts = no + 1;  // padded row stride of tstage (conflict-free column reads)
  __shared__ double red[2 * (T / 32)];
  __shared__ int perm[64];

  const double2* Wg =
      reinterpret_cast<const double2*>(S_.walk) + (long long)w * N * no;

  // ---- S = C^T W on the FP64 tensor cores ----------------------------------
  // As real matrices: S (No x 2No, (re, im) interleaved) = C^T (No x N) times
  // W (N x 2No, the complex walker viewed as doubles).  mma.m8n8k4 tiles: warp
  // w owns column tile w and every row tile, so each B fragment is
  // loaded once per k-step.  Rows of W and C are staged 32 at a time.
  const int warp = tid >> 5, lane = tid & 31;
  const int nc2 = 2 * no;
  const int mtiles = (no + 7) >> 3, ntiles = (nc2 + 7) >> 3;  // <= 8, <= 16
  const int nchunks = (N + kRowChunk - 1) / kRowChunk;
  // chunk c of the walker rows (and, with_mo, of the trial rows) into buffer c & 1
  auto load_chunk = [&](int c, bool with_mo) {
    const int p0 = c * kRowChunk, rows = min(kRowChunk, N - p0);
    double2* st = stage + (c & 1) * sbuf_;
    double* mc = moc + (c & 1) * kRowChunk * no;
    for (int e = tid; e < rows * no; e += T) {
      const int r = e / no;
      cp_async16(&st[r * (sd / 2) + (e - r * no)], &Wg[(long long)p0 * no + e]);
      if (with_mo) cp_async8(&mc[e], &S_.mo[(long long)p0 * no + e]);
    }
    cp_async_commit();
  };
  double2* sg = a.sbuf ? reinterpret_cast<double2*>(a.sbuf) + ((long long)sct * a.W + w) * a.sstride
                       : nullptr;
  const int npairs = no * no;
  if (mode != 2) {
  double sacc[MT][2];
#pragma unroll
  for (int mi = 0; mi < MT; ++mi) sacc[mi][0] = sacc[mi][1] = 0.0;
  load_chunk(0, true);
  for (int c = 0; c < nchunks; ++c) {
    const int p0 = c * kRowChunk, rows = min(kRowChunk, N - p0);
    if (c + 1 < nchunks) load_chunk(c + 1, true);
    else cp_async_commit();  // an empty group keeps the wait count uniform
    cp_async_wait1();
    __syncthreads();
    if (warp < ntiles) {  // warp-uniform
      // lane (r = lane / 4, q = lane % 4): A[m = 8 mi + r][k = q], B[k = q][n = 8 warp + r];
      // entries beyond No and 2 No (what follows in shared memory) only reach rows
      // and columns of S that are not stored
      const double* bp = reinterpret_cast<const double*>(stage + (c & 1) * sbuf_) + (lane & 3) * sd +
                         warp * 8 + (lane >> 2);
      const double* ap = moc + (c & 1) * kRowChunk * no + (lane & 3) * no + (lane >> 2);
      auto tiles = [&](auto count) {  // the first M row tiles
        constexpr int M = decltype(count)::value;
        const int full = rows & ~3;
#pragma unroll 2
        for (int kk = 0; kk < full; kk += 4) {
          const double b = bp[kk * sd];
          double afr[M];
#pragma unroll
          for (int mi = 0; mi < M; ++mi) afr[mi] = ap[kk * no + mi * 8];
#pragma unroll
          for (int mi = 0; mi < M; ++mi) dmma_8x8x4(sacc[mi][0], sacc[mi][1], afr[mi], b);
        }
        if (full < rows) {
          const bool kin = full + (lane & 3) < rows;
          const double b = kin ? bp[full * sd] : 0.0;
#pragma unroll
          for (int mi = 0; mi < M; ++mi)
            dmma_8x8x4(sacc[mi][0], sacc[mi][1], kin ? ap[full * no + mi * 8] : 0.0, b);
        }
      };
      // sectors and fragments smaller than the launch's widest work on fewer tiles
      if (mtiles <= 2)
        tiles(std::integral_constant<int, 2>{});
      else if (mtiles <= 4)
        tiles(std::integral_constant<int, 4>{});
      else
        tiles(std::integral_constant<int, MT>{});
    }
    __syncthreads();
  }
  if (warp < ntiles) {
#pragma unroll
    for (int mi = 0; mi < MT; ++mi) {
      const int i = mi * 8 + (lane >> 2), j = warp * 4 + (lane & 3);
      if (i < no && j < no) {
        const double2 v = make_double2(sacc[mi][0], sacc[mi][1]);
        if (mode == 1)
          sg[i * no + j] = v;
        else
          S[i * no + j] = v;
      }
    }
  }
  if (mode == 1) return;
  __syncthreads();
  }  // mode != 2
  if (mode == 2) {  // S^-1 from gj_kernel
    for (int e = tid; e < npairs; e += T) S[e] = sg[e];
    __syncthreads();
  } else {

  // ---- Gauss-Jordan inverse with partial pivoting, det ----------------------
  __shared__ double2 ipk_s;
  const double2 det = gauss_jordan_cta<T>(S, colk, perm, &ipk_s, no);
  if (tid == 0 && a.wscal) {
    a.wscal[(long long)w * 16 + 4 + 2 * sct] = det.x;
    a.wscal[(long long)w * 16 + 5 + 2 * sct] = det.y;
  }
  }  // mode 0: inverse in this CTA

  const bool need_theta = S_.theta || S_.gout || a.gpl || S_.rh1 || a.gplb[0] || S_.gtb[0];
  if (!need_theta) return;

  // ---- Theta = W S^-1, transposed copies, E1 --------------------------------
  double2 e1 = make_double2(0.0, 0.0);
  double* th = S_.theta ? S_.theta + (long long)w * 2 * no * S_.ldth : nullptr;
  double2* go = S_.gout ? reinterpret_cast<double2*>(S_.gout) + (long long)w * no * N : nullptr;
  double* gre = a.gpl ? a.gpl + (2LL * w) * a.ldg + S_.koff : nullptr;
  double* gim = a.gpl ? a.gpl + (2LL * w + 1) * a.ldg + S_.koff : nullptr;
  const bool gb = a.gplb[0] != nullptr;
  const bool tb = S_.gtb[0] != nullptr;
  load_chunk(0, false);
  // Theta rows (N x 2No real) = W rows (N x 2No) times the real form of
  // S^-1: R[2i][2j] = R[2i+1][2j+1] = Re s_ij, R[2i][2j+1] = Im s_ij,
  // R[2i+1][2j] = -Im s_ij.  A warp's column tile of it stays in registers for all rows.
  const int ksteps = (nc2 + 3) >> 2;
  double bfr[KS];
  {
    const int n = warp * 8 + (lane >> 2);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const int k = ks * 4 + (lane & 3);
      bfr[ks] = 0.0;
      if (k < nc2 && n < nc2) {
        const double2 sv = S[(k >> 1) * no + (n >> 1)];
        bfr[ks] = (k & 1) == 0 ? ((n & 1) == 0 ? sv.x : sv.y) : ((n & 1) == 0 ? -sv.y : sv.x);
      }
    }
  }
  for (int c = 0; c < nchunks; ++c) {
    const int p0 = c * kRowChunk, rows = min(kRowChunk, N - p0);
    // walker rows of the next chunk stream in while this one is processed
    if (c + 1 < nchunks) load_chunk(c + 1, false);
    else cp_async_commit();
    cp_async_wait1();
    __syncthreads();
    const double* stageD = reinterpret_cast<const double*>(stage + (c & 1) * sbuf_);
    if (warp < ntiles) {
      const int rtiles = (rows + 7) >> 3;  // <= 4
      double tacc[4][2];
#pragma unroll
      for (int ri = 0; ri < 4; ++ri) tacc[ri][0] = tacc[ri][1] = 0.0;
      // rows beyond the chunk's (left from another chunk) only reach rows not stored
      const double* ap = stageD + (lane >> 2) * sd + (lane & 3);
      if (rtiles == 4) {
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          if (ks >= ksteps) break;
          const bool kin = ks * 4 + (lane & 3) < nc2;
          double afr[4];
#pragma unroll
          for (int ri = 0; ri < 4; ++ri) afr[ri] = kin ? ap[ri * 8 * sd + ks * 4] : 0.0;
#pragma unroll
          for (int ri = 0; ri < 4; ++ri) dmma_8x8x4(tacc[ri][0], tacc[ri][1], afr[ri], bfr[ks]);
        }
      } else {
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          if (ks >= ksteps) break;
          const bool kin = ks * 4 + (lane & 3) < nc2;
#pragma unroll
          for (int ri = 0; ri < 3; ++ri)
            if (ri < rtiles)
              dmma_8x8x4(tacc[ri][0], tacc[ri][1], kin ? ap[ri * 8 * sd + ks * 4] : 0.0, bfr[ks]);
        }
      }
#pragma unroll
      for (int ri = 0; ri < 4; ++ri) {
        const int r = ri * 8 + (lane >> 2), j = warp * 4 + (lane & 3);
        if (r < rows && j < no) {
          const double2 sv = make_double2(tacc[ri][0], tacc[ri][1]);
          tstage[r * ts + j] = sv;
          if (S_.rh1) {
            const double h = S_.rh1[(long long)j * N + p0 + r];
            e1.x = fma(sv.x, h, e1.x);
            e1.y = fma(sv.y, h, e1.y);
          }
        }
      }
    }
    __syncthreads();
    if (th || go || gre || gb || tb) {
      for (int e = tid; e < rows * no; e += T) {
        const int j = rows == kRowChunk ? e / kRowChunk : e / rows, r = e - j * rows;
        const double2 v = tstage[r * ts + j];
        if (th) {
          th[2 * j * S_.ldth + p0 + r] = v.x;
          th[(2 * j + 1) * S_.ldth + p0 + r] = v.y;
        }
        if (go) go[(long long)j * N + p0 + r] = v;
        if (gre) {
          gre[(long long)j * N + p0 + r] = v.x;
          gim[(long long)j * N + p0 + r] = v.y;
        }
        if (gb) {
          const long long o = S_.koff + (long long)j * N + p0 + r;
          put_pieces(v.x, a.npc, a.gplb, (2LL * w) * a.ldgb + o);
          put_pieces(v.y, a.npc, a.gplb, (2LL * w + 1) * a.ldgb + o);
        }
        if (tb) {
          const long long rr = (long long)w * 2 * no + 2 * j;
          put_pieces(v.x, a.npc, S_.gtb, rr * S_.ldtb + p0 + r);
          put_pieces(v.y, a.npc, S_.gtb, (rr + 1) * S_.ldtb + p0 + r);
        }
      }
    }
    __syncthreads();
  }
  if (S_.rh1 && a.wscal) {
    const double ex = block_sum(e1.x, red);
    const double ey = block_sum(e1.y, red + T / 32);
    if (tid == 0) {
      a.wscal[(long long)w * 16 + 8 + 2 * sct] = ex;
      a.wscal[(long long)w * 16 + 9 + 2 * sct] = ey;
    }
  }
}

// Warp 0 of gj_kernel: the pivot among this lane's two candidate rows (lane,
// lane + 32) and the other lanes': the largest |re|+|im|, the lowest row
// among equal values (LAPACK izamax).  The keys hold the magnitude's bits above
// the row number: a non-negative double's bit pattern orders like its value, so
// the key order is the magnitude order except between values within 128 ulps of
// each other, which go to the lower row.  Non-candidates have key 0.  The maximum
// is two 32-bit warp reductions, the high words and then the low words under the
// highest; a 64-bit one by shuffles took 350 cycles a step.
__device__ __forceinline__ int gj_pivot(double2 v0, double2 v1, bool ok0, bool ok1, int lane) {
  auto key = [](double2 v, int row) -> unsigned long long {
    const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(v.x) + fabs(v.y));
    return (b & ~127ull) | 64ull | (unsigned long long)(63 - row);
  };
  unsigned long long k = ok0 ? key(v0, lane) : 0ull;
  const unsigned long long k1 = ok1 ? key(v1, lane + 32) : 0ull;
  k = k1 > k ? k1 : k;
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32) == hi ? (unsigned)k : 0u);
  return 63 - (int)(lo & 63u);
}

// Gauss-Jordan inverse and det of S = C^T W held in sbuf, one CTA per
// (walker, sector), in place in one shared-memory copy of S, in panels of four
// columns (partial pivoting, pivot = largest |re|+|im| in the column).
//  * Rows are never swapped: the pivot row r_k of step k stays in place and
//    the inverse is unscrambled once at the end, S^-1[i][r_k] = X[r_i][k].
//  * Pivot rows are scaled lazily: row r_k keeps its unscaled values, the factors
//    1 / p_k are applied where the row is used and at the end.
//  * Warp 0 runs a panel's steps on registers (lane l: rows l and l + 32 of the
//    four columns) without a block barrier and leaves each step's multipliers f_m
//    (the step's column before it) in P.
//  * Every other column then takes the four steps at once: s_m = a[r_m] / p_m with
//    the earlier steps applied to row r_m, a[i] -= f_m[i] s_m for i != r_m.  These
//    are the operations of one step after the other, in their order, so the
//    inverse has the same bits as without panels (the product of the four steps
//    applied as one matrix saves 10 us and rounds differently, which the
//    bf16 split of Theta then turns into differences of 1e-7 in a rare walker).
// What bounds it is the chain of pivots in warp 0 while the SM's other CTAs update.
// One barrier per column, with every step's column formed by warp 0 and the rest
// updated beside it, took 89 us at No = 40 and 512 walkers; this takes 67 us
// (No = 60, 58 and 1024 walkers: 940 -> 742 us; No = 39, 231 walkers: 59 -> 51 us).
// Panels of eight spill at 128 registers.
// Rows are stored with an odd stride (ld = no | 1 double2), so a warp reading a
// column hits distinct banks.  det = product of the pivots times the permutation's
// sign.  At most 64 rows (no <= 64, checked by the caller).
constexpr int kGjThreads = 128;
constexpr int kGjPanel = 4;

__device__ __forceinline__ double2 shfl2(double2 v, int lane) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}

// a b, rounded in one stated way wherever it stands: left to the compiler, the product
// that is fused in the imaginary part depends on the code around it
__device__ __forceinline__ double2 gj_mul(double2 a, double2 b) {
  return make_double2(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)), __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)));
}

__device__ __forceinline__ void gj_body(int W, int no0, int no1, double* sbuf, long long sstride,
                                        int bstride, double* wscal, int w, int sct) {
  extern __shared__ double2 gsm[];
  const int no = sct ? no1 : no0;
  const int ld = no | 1;
  const int nn = no * no;
  double2* const A = gsm;
  double2* const P = gsm + bstride;  // the panel: [64][kGjPanel]
  __shared__ int piv[64];
  __shared__ double2 ipks[64];  // 1 / pivot of each step (the lazy row scales)
  const int tid = threadIdx.x, lane = tid & 31;
  double2* g = reinterpret_cast<double2*>(sbuf) + ((long long)sct * W + w) * sstride;
  for (int e = tid; e < nn; e += kGjThreads) {
    const int i = e / no;
    A[i * ld + (e - i * no)] = g[e];
  }
  __syncthreads();

  const double2 zero = make_double2(0.0, 0.0);
  const bool in0 = lane < no, in1 = lane + 32 < no;
  bool used0 = false, used1 = false;  // warp 0: rows lane, lane + 32 already pivots
  double2 det = make_double2(1.0, 0.0);
  // trailing update: thread -> column jt of the no - b others, rows g0, g0 + RG, ...
  for (int k0 = 0; k0 < no; k0 += kGjPanel) {
    const int b = min(kGjPanel, no - k0);
    if (tid < 32) {
      double2 v0[kGjPanel], v1[kGjPanel];
#pragma unroll
      for (int c = 0; c < kGjPanel; ++c) {
        v0[c] = in0 && c < b ? A[lane * ld + k0 + c] : zero;
        v1[c] = in1 && c < b ? A[(lane + 32) * ld + k0 + c] : zero;
      }
#pragma unroll
      for (int m = 0; m < kGjPanel; ++m) {
        if (m < b) {
          const int rn = gj_pivot(v0[m], v1[m], in0 && !used0, in1 && !used1, lane);
          const bool hi = rn >= 32;
          const int owner = rn & 31;
          const double2 p = shfl2(hi ? v1[m] : v0[m], owner);
          const double inv = 1.0 / (p.x * p.x + p.y * p.y);
          const double2 ip = make_double2(p.x * inv, -p.y * inv);
          const bool mine0 = !hi && lane == owner, mine1 = hi && lane == owner;
          const double2 f0 = v0[m], f1 = v1[m];
          P[lane * kGjPanel + m] = f0;
          P[(lane + 32) * kGjPanel + m] = f1;
#pragma unroll
          for (int c = 0; c < kGjPanel; ++c) {
            if (c == m) continue;
            const double2 s = gj_mul(shfl2(hi ? v1[c] : v0[c], owner), ip);
            const double2 t0 = csub(v0[c], gj_mul(f0, s)), t1 = csub(v1[c], gj_mul(f1, s));
            v0[c] = mine0 ? v0[c] : t0;
            v1[c] = mine1 ? v1[c] : t1;
          }
          const double2 q0 = gj_mul(f0, ip), q1 = gj_mul(f1, ip);
          v0[m] = mine0 ? make_double2(1.0, 0.0) : make_double2(-q0.x, -q0.y);
          v1[m] = mine1 ? make_double2(1.0, 0.0) : make_double2(-q1.x, -q1.y);
          used0 |= mine0;
          used1 |= mine1;
          det = gj_mul(p, det);
          if (lane == 0) {
            piv[k0 + m] = rn;
            ipks[k0 + m] = ip;
          }
        }
      }
#pragma unroll
      for (int c = 0; c < kGjPanel; ++c) {
        if (c < b && in0) A[lane * ld + k0 + c] = v0[c];
        if (c < b && in1) A[(lane + 32) * ld + k0 + c] = v1[c];
      }
    }
    __syncthreads();
    const int cols = no - b;
    if (cols > 0) {
      // column tiles of at most kGjThreads columns never occur (no <= 64)
      const int rg = kGjThreads / cols, jt = tid % cols, r0 = tid / cols;
      const int j = jt < k0 ? jt : jt + b;
      int r[kGjPanel];
      double2 u[kGjPanel];  // the pivot rows' entries, then s_m
      if (r0 < rg) {
#pragma unroll
        for (int m = 0; m < kGjPanel; ++m) {
          r[m] = m < b ? piv[k0 + m] : 0;
          u[m] = m < b ? A[r[m] * ld + j] : zero;
        }
#pragma unroll
        for (int m = 0; m < kGjPanel; ++m)
          if (m < b) {
            u[m] = gj_mul(u[m], ipks[k0 + m]);
#pragma unroll
            for (int l = m + 1; l < kGjPanel; ++l)
              if (l < b) u[l] = csub(u[l], gj_mul(P[r[l] * kGjPanel + m], u[m]));
          }
      }
      __syncthreads();
      if (r0 < rg)
#pragma unroll 2
        for (int i = r0; i < no; i += rg) {
          double2 x = A[i * ld + j];
          const double2* pr = P + i * kGjPanel;
#pragma unroll
          for (int m = 0; m < kGjPanel; ++m)
            if (m < b) {
              const double2 t = csub(x, gj_mul(pr[m], u[m]));
              x = i == r[m] ? x : t;
            }
          A[i * ld + j] = x;
        }
      __syncthreads();
    }
  }
  // unscramble with the row scales: S^-1[i][r_k] = X[r_i][k] = A[r_i][k] / p_i
  for (int e = tid; e < nn; e += kGjThreads) {
    const int i = e / no, k = e - (e / no) * no;
    g[i * no + piv[k]] = gj_mul(ipks[i], A[piv[i] * ld + k]);
  }
  if (tid == 0) {
    // sign of the permutation k -> r_k: (-1)^(no - cycles)
    unsigned long long seen = 0ull;
    int cycles = 0;
    for (int s0 = 0; s0 < no; ++s0) {
      if (seen >> s0 & 1ull) continue;
      ++cycles;
      for (int t = s0; !(seen >> t & 1ull); t = piv[t]) seen |= 1ull << t;
    }
    if ((no - cycles) & 1) det = make_double2(-det.x, -det.y);
    if (wscal) {
      wscal[(long long)w * 16 + 4 + 2 * sct] = det.x;
      wscal[(long long)w * 16 + 5 + 2 * sct] = det.y;
    }
  }
}

template <int T>
__global__ void __launch_bounds__(T, T <= 320 ? 2 : 1) green_kernel(GreenArgs a, int mode) {
  green_body<T>(a, mode, blockIdx.x, blockIdx.y);
}

template <int T>
__global__ void __launch_bounds__(T, T <= 320 ? 2 : 1) green_kernel_grouped(const GreenArgs* A, BlockMap m, int mode) {
  int local;
  const GreenArgs& a = A[block_owner(m, blockIdx.x, local)];
  green_body<T>(a, mode, local % a.W, local / a.W);
}

// Threads of the S / Theta kernels: a warp for each of the (2 No + 7) / 8 column
// tiles, 8, 10, 12 or 16 of them.  With eight warps for ten tiles (No = 40) two
// warps worked twice as long as the rest: S + Theta 216 -> 177 us at N = 200,
// 512 walkers.
inline int green_threads(int nomax) {
  const int tiles = (2 * nomax + 7) / 8;
  return tiles <= 8 ? 256 : (tiles <= 10 ? 320 : (tiles <= 12 ? 384 : 512));
}

// calls f(kernel) for the kernel template's instance of `threads`
template <class F>
cudaError_t with_green_kernel(int threads, F&& f) {
  switch (threads) {
    case 256: return f(green_kernel<256>, green_kernel_grouped<256>);
    case 320: return f(green_kernel<320>, green_kernel_grouped<320>);
    case 384: return f(green_kernel<384>, green_kernel_grouped<384>);
    default: return f(green_kernel<512>, green_kernel_grouped<512>);
  }
}

__global__ void __launch_bounds__(kGjThreads, 4)
    gj_kernel(int W, int no0, int no1, double* sbuf, long long sstride, int bstride, double* wscal) {
  gj_body(W, no0, no1, sbuf, sstride, bstride, wscal, blockIdx.x, blockIdx.y);
}

__global__ void __launch_bounds__(kGjThreads, 4) gj_kernel_grouped(const GjArgs* A, BlockMap m) {
  int local;
  const GjArgs& a = A[block_owner(m, blockIdx.x, local)];
  gj_body(a.W, a.no0, a.no1, a.sbuf, a.sstride, a.bstride, a.wscal, local % a.W, local / a.W);
}

// one compiled copy for the solo and the grouped kernel (identical rounding)
__device__ __noinline__ void ovlp_body(int W, int ns, int mult, const double* wscal, double* out,
                                          int out_stride, int w) {
  if (w >= W) return;
  const double2 d0 = make_double2(wscal[(long long)w * 16 + 4], wscal[(long long)w * 16 + 5]);
  double2 o;
  if (ns == 1) {
    o = (mult == 2) ? cmul(d0, d0) : d0;
  } else {
    const double2 d1 = make_double2(wscal[(long long)w * 16 + 6], wscal[(long long)w * 16 + 7]);
    o = cmul(d0, d1);
  }
  out[(long long)w * out_stride] = o.x;
  out[(long long)w * out_stride + 1] = o.y;
}

__global__ void ovlp_combine_kernel(int W, int ns, int mult, const double* wscal, double* out,
                                    int out_stride) {
  ovlp_body(W, ns, mult, wscal, out, out_stride, blockIdx.x * blockDim.x + threadIdx.x);
}

__global__ void ovlp_combine_grouped(const OvlpArgs* A, BlockMap m) {
  int local;
  const OvlpArgs& a = A[block_owner(m, blockIdx.x, local)];
  ovlp_body(a.W, a.ns, a.mult, a.wscal, a.out, a.out_stride, local * blockDim.x + threadIdx.x);
}

}  // namespace

size_t green_smem_bytes(int nomax) {
  const int sdmax = 2 * nomax + ((20 - (2 * nomax) % 16) % 16);  // padded walker-row stride (doubles)
  return (size_t(nomax) * nomax + 64) * sizeof(double2) + 2 * size_t(kRowChunk) * sdmax * sizeof(double) +
         2 * size_t(kRowChunk) * nomax * sizeof(double) + size_t(kRowChunk) * (nomax + 1) * sizeof(double2);
}

// S with row stride nomax | 1 and a panel of four columns
size_t gj_smem_bytes(int nomax) {
  return (size_t(nomax) * (nomax | 1) + 64 * kGjPanel) * sizeof(double2);
}

cudaError_t launch_green_grouped(const GreenArgs* args, const BlockMap& m, int mode, int nomax,
                                 cudaStream_t st) {
  ProfScope ps(K_GREEN, st);
  const int threads = green_threads(nomax);
  const size_t smem = green_smem_bytes(nomax);
  return with_green_kernel(threads, [&](auto, auto kernel) {
    cudaError_t e = allow_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<m.start[m.n], threads, smem, st>>>(args, m, mode);
    return cudaGetLastError();
  });
}

cudaError_t launch_gj_grouped(const GjArgs* args, const BlockMap& m, size_t smem, cudaStream_t st) {
  cudaError_t e = allow_smem(gj_kernel_grouped, smem);
  if (e != cudaSuccess) return e;
  ProfScope ps(K_GREEN, st);
  gj_kernel_grouped<<<m.start[m.n], kGjThreads, smem, st>>>(args, m);
  return cudaGetLastError();
}

cudaError_t launch_ovlp_grouped(const OvlpArgs* args, const BlockMap& m, cudaStream_t st) {
  ProfScope ps(K_MISC, st);
  ovlp_combine_grouped<<<m.start[m.n], 256, 0, st>>>(args, m);
  return cudaGetLastError();
}

cudaError_t launch_green(const GreenArgs& a, cudaStream_t st) {
  int nomax = 0;
  for (int s = 0; s < a.ns; ++s) nomax = a.sec[s].no > nomax ? a.sec[s].no : nomax;
  const size_t smem = green_smem_bytes(nomax);
  const int threads = green_threads(nomax);
  dim3 grid(a.W, a.ns);
  ProfScope ps(K_GREEN, st);
  bool need_theta = a.gpl || a.gplb[0];
  for (int s = 0; s < a.ns; ++s)
    need_theta = need_theta || a.sec[s].theta || a.sec[s].gout || a.sec[s].rh1 || a.sec[s].gtb[0];
  return with_green_kernel(threads, [&](auto kernel, auto) {
    cudaError_t e = allow_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    if (!a.sbuf || !need_theta) {  // one kernel: S, its inverse and det, Theta and outputs
      kernel<<<grid, threads, smem, st>>>(a, 0);
      return cudaGetLastError();
    }
    // S into a.sbuf; its inverse and det; Theta and its outputs
    kernel<<<grid, threads, smem, st>>>(a, 1);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const int bstride = nomax * (nomax | 1);
    const size_t gsmem = gj_smem_bytes(nomax);
    if ((e = allow_smem(gj_kernel, gsmem)) != cudaSuccess) return e;
    gj_kernel<<<grid, kGjThreads, gsmem, st>>>(a.W, a.sec[0].no, a.ns > 1 ? a.sec[1].no : 0, a.sbuf,
                                               a.sstride, bstride, a.wscal);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    kernel<<<grid, threads, smem, st>>>(a, 2);
    return cudaGetLastError();
  });
}

cudaError_t launch_ovlp_combine(int W, int ns, int mult, const double* wscal, double* out,
                                int out_stride, cudaStream_t st) {
  ProfScope ps(K_MISC, st);
  ovlp_combine_kernel<<<(W + 255) / 256, 256, 0, st>>>(W, ns, mult, wscal, out, out_stride);
  return cudaGetLastError();
}

}  // namespace afq
