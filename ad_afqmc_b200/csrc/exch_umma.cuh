// Exchange energy on the tensor cores: f = RC . Theta per (Cholesky vectors x
// walkers) tile, reduced to tr f and sum f o f^T without leaving the SM
// (wavefunctions.py:1128-1174, 1331-1363).
//
// The tile is 128 rows (gpt Cholesky vectors of No rows) by BN columns (wpt
// walkers of 2 No columns).  Roles as in umma_gemm.cuh: a TMA producer warp, an
// MMA warp, eight epilogue warps behind one or two TMEM buffers and four reducing warps.  What sets it
// apart from the general GEMM:
//  * The shared-memory port (128 bytes per cycle) is what bounds it: an MMA of
//    128 x N x 16 reads 4096 + 32 N bytes of it, TMA writes the operands through it
//    and the epilogue stages f in it, and the MMAs have precedence.  So the
//    rot_chol pieces sit in TMEM where they fit (umma_exch_ts_kernel) while the
//    CTA walks the walkers: the MMAs read 32 N bytes and a tile streams its Theta
//    pieces only.
//  * Where they do not fit both operands stream, all CTAs on the same rot_chol
//    rows and neighbouring walkers.  The walkers go in chunks whose Theta pieces
//    stay in the L2 (without chunks, 1024 walkers at N = 300 re-read 157 MB of them
//    from HBM for each of 750 row tiles: 30 ms per spin, whatever the epilogue).
//  * Boxes hold the rows in use (gpt No, wpt 2 No), not the MMA's 128 x BN:
//    the MMA reads on into whatever follows, and those rows and columns of the
//    accumulator are never looked at.
//  * Eight epilogue warps share a tile (see exch_tile); its sums end in FP64 (exch_finish).
// Measured on a B200, two pieces, per launch, the general GEMM before -> this: N = 200,
// No = 40, G = 1000, W = 512 4.74 -> 2.45 ms; N = 300, No = 60, G = 1500, W = 1024 29.7 ->
// 23.8 ms; N = 250, No = 62, G = 1250, W = 256 4.98 -> 3.53 ms.
#pragma once

#include "layout.cuh"
#include "umma_gemm.cuh"

namespace afq {

struct ExchParams {
  CUtensorMap ta[3], tb[3];
  int npc;                 // bf16 pieces (2 or 3)
  int G, no, W, K;         // K = N
  int gpt, wpt, mt, nt;    // tiling
  int ncw;                 // walker tiles per L2 chunk
  int arows, brows;        // box rows of A (multiple of 8) and B (multiple of 8)
  int stages, gsub, wsub, lot;
  int ring;                // slots between the epilogue and the reducing warps (4 or 2)
  const bf16* a[2];        // row operand pieces (the TMEM kernel loads them itself), row stride lda
  long long lda;
  double* cout;            // (W, G) complex: tr f
  double* excout;          // (mt, W) complex: sum f o f^T
  int* err;
};

// float2 per staged row: the (re, im) pairs of wsub walkers, odd so that consecutive
// rows and consecutive pairs both spread over the banks
__host__ __device__ inline int exch_row_pairs(int no, int wsub) { return (no * wsub) | 1; }

// bytes behind the ring that an MMA over bn rows reads past a box of brows rows
__host__ __device__ inline size_t exch_overread(int bn, int brows) { return size_t(bn - brows) * 128; }

constexpr int kExchRing = 4;  // most walkers between the epilogue and the reducing warps

// What a launch needs besides the tiling.  ts: the row operand in TMEM.
struct ExchPlan {
  int ts, nbuf, lot;  // TMEM accumulator buffers; K blocks of the low piece that sit in TMEM
  int stages, gsub, wsub;  // Cholesky vectors and walkers staged at once
  int ring;
  size_t smem;
};
// ring of a walker's row chains (2 x float4) and diagonals (float2), and staging of the epilogue
__host__ __device__ inline size_t exch_epi_bytes(int no, int wsub, int gsub, int ring) {
  return (size_t(ring) * 128 * (2 * 16 + 8) + size_t(gsub) * no * exch_row_pairs(no, wsub) * 8 + 255) & ~size_t(255);
}

// Streaming kernel: [ring of A and B][barriers 256][sums][staging].
// TMEM kernel: [low-piece blocks of A that do not fit TMEM][ring of B][barriers
// 256][sums, staging].  An MMA reads 128 (A) or bn (B) rows from a box of
// fewer: what lies behind is the next box, or `over` bytes kept free.
inline ExchPlan exch_plan(int npc, int no, int K, const UExchTile& X, int arows, int brows,
                          int max_stages) {
  const int KB = (K + kUBK - 1) / kUBK, KS = (K + 15) / 16;
  const size_t a = size_t(arows) * 128, b = size_t(brows) * 128;
  const size_t fixed = 1024 + exch_overread(X.bn, brows) + 256;
  ExchPlan p{};
  const int cap = max_stages >= 2 ? max_stages : 6;
  // three stages hide the load latency behind a K block's MMAs; the whole tile
  // staged at once if it fits beside them (a pass less in the epilogue), else as
  // many of its walkers as fit, or, with one walker, Cholesky vectors.  (Several
  // walkers are never cut by vectors: the threads of the other rows would stand idle in
  // every pass.  Three pieces, N = 100, No = 8, 200 walkers, where three of 16 vectors
  // fit: 197 us an energy by vectors, 94 us by walkers.)
  auto fill = [&](size_t res, size_t stage) {
    const int most = X.wpt == 1 ? X.gpt : X.wpt;
    for (int ring = kExchRing; ring >= 2; ring >>= 1)
      for (int want = cap < 3 ? cap : 3; want >= 2; --want)
        for (int n = most; n >= 1; --n) {
          const int g = X.wpt == 1 ? n : X.gpt, w = X.wpt == 1 ? 1 : n;
          const size_t base = fixed + res + exch_epi_bytes(no, w, g, ring);
          if (base + want * stage > kUmmaSmemBudget) continue;
          const int st = int((kUmmaSmemBudget - base) / stage);
          p.stages = st > cap ? cap : st;
          p.gsub = g;
          p.wsub = w;
          p.ring = ring;
          p.smem = base + p.stages * stage;
          return true;
        }
    return false;
  };
  // two accumulator buffers if the high piece's K fits the columns beside them, else one
  for (p.nbuf = 2; npc == 2 && p.nbuf >= 1; --p.nbuf) {
    const int steps = (512 - p.nbuf * 2 * X.bn) / 8;
    if (steps < KS) continue;
    const int rest = steps - KS;
    p.lot = rest >= KS ? KB : rest / 4;  // whole 64-wide blocks
    p.ts = fill((KB - p.lot) * a, 2 * b);
    if (p.ts) return p;
  }
  p.ts = 0;
  fill(0, npc * (a + b));
  return p;
}

// the eight epilogue warps (four more reduce)
__device__ __forceinline__ void exch_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
constexpr int kExchThreads = 64 + 256 + 128;

// position of a tile: walker chunk [c0, c0 + width), row tile, walker tile;
// stepped without divisions (a 64-bit division costs the MMA thread 500 cycles)
struct ExchWalk {
  int c0, width, mti, nti;
};
__device__ __forceinline__ ExchWalk exch_locate(const ExchParams& P, int t) {
  ExchWalk w;
  const int per = P.mt * P.ncw, ch = t / per, rem = t - ch * per;
  w.c0 = ch * P.ncw;
  w.width = min(P.ncw, P.nt - w.c0);
  w.mti = w.width > 0 ? rem / w.width : 0;
  w.nti = w.c0 + rem - w.mti * w.width;
  return w;
}
__device__ __forceinline__ void exch_advance(const ExchParams& P, ExchWalk& w, int step) {
  w.nti += step;
  while (w.nti >= w.c0 + w.width) {
    w.nti -= w.width;
    if (++w.mti == P.mt) {  // next walker chunk: the overshoot carries over
      const int over = w.nti - w.c0;
      w.mti = 0;
      w.c0 += P.ncw;
      w.width = min(P.ncw, P.nt - w.c0);
      if (w.width <= 0) return;  // past the last tile
      w.nti = w.c0 + over;
    }
  }
}

// four consecutive fp32 columns of this thread's TMEM lane, issued without waiting
__device__ __forceinline__ void tmem_ld4_issue(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// no instruction: keeps every use of the registers behind the wait before it
__device__ __forceinline__ void tmem_tie(uint32_t (&r)[4], uint32_t (&q)[4]) {
  asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(q[0]), "+r"(q[1]),
                    "+r"(q[2]), "+r"(q[3]));
}

// Sums of FP32 values.  The FP64 unit waits for the tensor core while tcgen05.mma
// runs (110 to 170 cycles an instruction and scheduler, a dependent DADD 405, an FADD 14), so a
// lane adds its values up in FP32 with the rounding errors carried along twice
// (Knuth's two-sum): a + b + c holds about 70 bits of the sum, and becomes one FP64 number.
struct ExchSum {
  float a, b, c;
};
__device__ __forceinline__ float exch_two_sum(float& s, float x) {  // s += x, returns what was rounded off
  const float t = __fadd_rn(s, x), v = __fsub_rn(t, s);
  const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, v)), __fsub_rn(x, v));
  s = t;
  return e;
}
__device__ __forceinline__ void exch_add(ExchSum& s, float x) {
  s.c = __fadd_rn(s.c, exch_two_sum(s.b, exch_two_sum(s.a, x)));
}
__device__ __forceinline__ double exch_value(const ExchSum& s) { return (double)s.a + ((double)s.b + (double)s.c); }

// x of half the lanes (those with lane & o) exchanged for y of the others: lanes without
// the bit then hold the sum of two lanes' x, those with it of two lanes' y
__device__ __forceinline__ ExchSum exch_halve(const ExchSum& x, const ExchSum& y, int o) {
  const bool up = (threadIdx.x & o) != 0;
  ExchSum m = up ? y : x;
  const ExchSum t = up ? x : y;
  const float a = __shfl_xor_sync(0xffffffffu, t.a, o), b = __shfl_xor_sync(0xffffffffu, t.b, o),
              c = __shfl_xor_sync(0xffffffffu, t.c, o);
  exch_add(m, a);
  exch_add(m, b);
  exch_add(m, c);
  return m;
}

// One tile's epilogue by eight warps: f from the accumulators (both groups
// summed in FP32) to shared memory, then per row (g, i) and walker
// sum_j f[i][j] f[j][i] in four FP32 chains (j mod 4; the last no mod 4 terms in
// chain 0).  Half h of the warps moves the pairs j = 2h, 2h + 1 (mod 4) and runs
// chains 2h, 2h + 1 of all 128 rows.  The loops stay rolled: the warps share an
// instruction cache with the MMA warp, and a fully unrolled form with the row in
// registers ran slower.  A walker's chains (xs: [2 halves][128], re re im im) and
// diagonals (dg: [128]) go to the reducing warps through a ring of P.ring slots;
// `slot` counts them over the CTA's tiles.
// times the ring has gone round before this slot
__device__ __forceinline__ int exch_lap(const ExchParams& P, int slot) { return slot >> (P.ring == 4 ? 2 : 1); }

template <int BN>
__device__ __forceinline__ void exch_tile(const ExchParams& P, uint32_t taddr, uint64_t* release, int mti,
                                          int nti, int ew, int& slot, float2* Fs, float4* xsum, float2* diag,
                                          uint64_t* xempty, uint64_t* xfull, volatile int* abort_s) {
  const int lane = threadIdx.x & 31, h = ew >> 2, row = ((threadIdx.x >> 5) & 3) * 32 + lane;
  const int no = P.no, no4 = no & ~3;
  const int gl = row / no, i = row - gl * no;
  const int fs = exch_row_pairs(no, P.wsub);
  const bool one = P.wpt == 1;
  const int gcount = min(P.gpt, P.G - mti * P.gpt), wcount = min(P.wpt, P.W - nti * P.wpt);
  const int nall = one ? gcount : wcount, nsub = one ? P.gsub : P.wsub;
  for (int s = 0; s < nall; s += nsub) {  // Cholesky vectors (one walker) or walkers staged together
    const int n = min(nsub, nall - s);
    const bool last = s + nsub >= nall;
    const int gs = one ? s : 0, gn = one ? n : gcount, ws = one ? 0 : s, wn = one ? 1 : n;
    const bool mine = gl >= gs && gl < gs + gn;
    const int plo = ws * no, phi = (ws + wn) * no;  // (re, im) pairs of the row
    float2* const fr = Fs + (row - gs * no) * fs;
    constexpr int NCH = BN / 16, CU = NCH == 5 ? 5 : (NCH == 6 ? 3 : (NCH >= 4 ? 4 : NCH));
#pragma unroll 1
    for (int c = 0; c < NCH; c += CU) {
      if ((c + CU) * 8 <= plo || c * 8 >= phi) continue;
      uint32_t x[2 * CU][4], y[2 * CU][4];
#pragma unroll
      for (int k = 0; k < 2 * CU; ++k) {
        const uint32_t ta = taddr + c * 16 + k * 8 + 4 * h;
        tmem_ld4_issue(ta, x[k]);
        tmem_ld4_issue(ta + BN, y[k]);
      }
      tmem_wait_ld();
#pragma unroll
      for (int k = 0; k < 2 * CU; ++k) {
        tmem_tie(x[k], y[k]);
        const int pr = c * 8 + k * 4 + 2 * h;
        if (mine && pr >= plo && pr < phi)
          fr[pr - plo] = make_float2(__uint_as_float(x[k][0]) + __uint_as_float(y[k][0]),
                                     __uint_as_float(x[k][1]) + __uint_as_float(y[k][1]));
        if (mine && pr + 1 >= plo && pr + 1 < phi)
          fr[pr + 1 - plo] = make_float2(__uint_as_float(x[k][2]) + __uint_as_float(y[k][2]),
                                         __uint_as_float(x[k][3]) + __uint_as_float(y[k][3]));
      }
    }
    if (last) {  // the accumulators are in shared memory
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(release);
    }
    exch_sync();
    for (int wl = 0; wl < wn; ++wl) {
      const int q = slot & (P.ring - 1);
      if (!one || s == 0) mbar_wait_run_on(&xempty[q], (exch_lap(P, slot) & 1) ^ 1, abort_s, P.err);
      if (mine) {
        const float2* fc = Fs + (gl - gs) * no * fs + wl * no + i;
        const float2* fw = fr + wl * no;
        float ar0 = 0.f, ai0 = 0.f, ar1 = 0.f, ai1 = 0.f;
#pragma unroll 2
        for (int j = 2 * h; j < no4; j += 4) {
          const float2 a0 = fw[j], a1 = fw[j + 1], b0 = fc[j * fs], b1 = fc[(j + 1) * fs];
          ar0 = fmaf(a0.x, b0.x, fmaf(-a0.y, b0.y, ar0));
          ai0 = fmaf(a0.x, b0.y, fmaf(a0.y, b0.x, ai0));
          ar1 = fmaf(a1.x, b1.x, fmaf(-a1.y, b1.y, ar1));
          ai1 = fmaf(a1.x, b1.y, fmaf(a1.y, b1.x, ai1));
        }
        if (h == 0)
          for (int j = no4; j < no; ++j) {
            const float2 a = fw[j], b = fc[j * fs];
            ar0 = fmaf(a.x, b.x, fmaf(-a.y, b.y, ar0));
            ai0 = fmaf(a.x, b.y, fmaf(a.y, b.x, ai0));
          }
        xsum[q * 256 + h * 128 + row] = make_float4(ar0, ar1, ai0, ai1);
        if (h == 0) diag[q * 128 + row] = fw[i];
      }
      if (!one || last) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&xfull[q]);
        ++slot;
      }
    }
    exch_sync();
  }
}

// The same sums in FP64 throughout: a walker some of whose FP32 sums leave FP32's range (an
// overflowed row, an infinite or undefined one).  +-inf stays +-inf.
__device__ __noinline__ void exch_finish_f64(const ExchParams& P, int mti, int w, const float4* xs,
                                             const float2* dg) {
  const int lane = threadIdx.x & 31, no = P.no;
  const int g0 = mti * P.gpt, gcount = min(P.gpt, P.G - g0), rows = gcount * no;
  double x = 0.0, y = 0.0;
  for (int k = lane; k < rows; k += 32) {
    const float4 u = xs[k], v = xs[128 + k];
    x += ((double)u.x + (double)u.y) + ((double)v.x + (double)v.y);
    y += ((double)u.z + (double)u.w) + ((double)v.z + (double)v.w);
  }
  __syncwarp();
  x = warp_sum(x);
  y = warp_sum(y);
  if (lane == 0) {
    P.excout[2 * ((long long)mti * P.W + w)] = x;
    P.excout[2 * ((long long)mti * P.W + w) + 1] = y;
  }
  double* const c = P.cout + 2 * ((long long)w * P.G + g0);
  for (int g = lane; g < gcount; g += 32) {
    double cr = 0.0, ci = 0.0;
    for (int q = 0; q < no; ++q) {
      const float2 z = dg[g * no + q];
      cr += (double)z.x;
      ci += (double)z.y;
    }
    c[2 * g] = cr;
    c[2 * g + 1] = ci;
  }
}

// The reducing warps: a walker's chains and diagonals to its exchange partial and its
// Cholesky vectors' traces, FP64 numbers.  Four warps take the slots in turn, off the
// epilogue's path: the sums take longer than a tile.  The FP32 sums come first, so
// that the FP64 instructions of all of them overlap.
__device__ __forceinline__ void exch_finish(const ExchParams& P, int mti, int w, const float4* xs,
                                            const float2* dg, uint64_t* xempty, uint64_t* xfull, uint32_t parity,
                                            volatile int* abort_s) {
  const int lane = threadIdx.x & 31, no = P.no;
  const int g0 = mti * P.gpt, gcount = min(P.gpt, P.G - g0), rows = gcount * no;
  mbar_wait_run_on(xfull, parity, abort_s, P.err);
  const ExchSum zero = {0.f, 0.f, 0.f};
  ExchSum r = zero, i = zero;
#pragma unroll 1
  for (int k = 0; k < 4; ++k)
    if (lane + 32 * k < rows) {
      const float4 u = xs[lane + 32 * k], v = xs[128 + lane + 32 * k];
      exch_add(r, u.x);
      exch_add(i, u.z);
      exch_add(r, u.y);
      exch_add(i, u.w);
      exch_add(r, v.x);
      exch_add(i, v.z);
      exch_add(r, v.y);
      exch_add(i, v.w);
    }
  __syncwarp();
  const ExchSum m = exch_halve(r, i, 16);  // lanes 0-15: re, 16-31: im
  double x = exch_value(m);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  if ((lane & 15) == 0) P.excout[2 * ((long long)mti * P.W + w) + (lane >> 4)] = x;
  // traces: a lane each of up to 128 Cholesky vectors (no <= 14), or eight lanes each
  // of up to eight, four of them re and four im
  double* const c = P.cout + 2 * ((long long)w * P.G + g0);
  bool fin = isfinite(m.a);
  if (gcount > 8) {
#pragma unroll 1
    for (int gb = 0; gb < gcount; gb += 32) {
      const int g = gb + lane;
      ExchSum tr = zero, ti = zero;
      if (g < gcount)
#pragma unroll 1
        for (int q = 0; q < no; ++q) {
          const float2 z = dg[g * no + q];
          exch_add(tr, z.x);
          exch_add(ti, z.y);
        }
      __syncwarp();
      fin = fin && isfinite(tr.a) && isfinite(ti.a);
      if (g < gcount) *reinterpret_cast<double2*>(c + 2 * g) = make_double2(exch_value(tr), exch_value(ti));
    }
  } else {
#pragma unroll 1
    for (int gb = 0; gb < gcount; gb += 4) {
      const int g = gb + (lane >> 3);
      ExchSum tr = zero, ti = zero;
      if (g < gcount)
#pragma unroll 1
        for (int q = lane & 7; q < no; q += 8) {
          const float2 z = dg[g * no + q];
          exch_add(tr, z.x);
          exch_add(ti, z.y);
        }
      __syncwarp();
      const ExchSum mt = exch_halve(tr, ti, 4);
      fin = fin && isfinite(mt.a);
      double y = exch_value(mt);
      y += __shfl_xor_sync(0xffffffffu, y, 2);
      y += __shfl_xor_sync(0xffffffffu, y, 1);
      if (g < gcount && (lane & 3) == 0) c[2 * g + ((lane >> 2) & 1)] = y;
    }
  }
  if (!__all_sync(0xffffffffu, fin)) exch_finish_f64(P, mti, w, xs, dg);
  __syncwarp();
  if (lane == 0) mbar_arrive(xempty);
}

// The reducing warps' part of one tile: every P.ring-th slot each.
__device__ __forceinline__ void exch_reduce(const ExchParams& P, int mti, int nti, int rw, int& slot,
                                            const float4* xsum, const float2* diag, uint64_t* xempty,
                                            uint64_t* xfull, volatile int* abort_s) {
  const int w0 = nti * P.wpt, wcount = min(P.wpt, P.W - w0);
  for (int wl = 0; wl < wcount; ++wl, ++slot)
    if ((slot & (P.ring - 1)) == rw)
      exch_finish(P, mti, w0 + wl, xsum + rw * 256, diag + rw * 128, &xempty[rw], &xfull[rw],
                  exch_lap(P, slot) & 1, abort_s);
}

// Streaming form: three-piece operands, or K too long for TMEM.
template <int BN, int NPC>
__global__ void __launch_bounds__(kExchThreads, 1) umma_exch_kernel(const __grid_constant__ ExchParams P) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem =
      reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int ST = P.stages, no = P.no, KB = (P.K + kUBK - 1) / kUBK;
  const uint32_t a_bytes = P.arows * 128, b_bytes = P.brows * 128;
  const uint32_t stage_bytes = NPC * (a_bytes + b_bytes);
  uint8_t* ring = smem;
  uint64_t* full =
      reinterpret_cast<uint64_t*>(ring + size_t(ST) * stage_bytes + exch_overread(BN, P.brows));
  uint64_t* empty = full + ST;
  uint64_t* accf = empty + ST;
  uint64_t* acce = accf + 2;
  uint64_t* xfull = acce + 2;
  uint64_t* xempty = xfull + kExchRing;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xempty + kExchRing);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float4* xsum = reinterpret_cast<float4*>(reinterpret_cast<uint8_t*>(full) + 256);
  float2* diag = reinterpret_cast<float2*>(xsum + P.ring * 256);
  float2* Fs = diag + P.ring * 128;

  constexpr uint32_t kCols = umma_tmem_cols(BN, 2, 2);
  constexpr uint32_t acc_stride = 2 * BN;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], 8);
    }
    for (int b = 0; b < kExchRing; ++b) {
      mbar_init(&xfull[b], 8);
      mbar_init(&xempty[b], 1);
    }
    *abort_s = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tmem_slot;

  // tiles of this CTA: every gridDim-th
  const int T = P.mt * P.nt;  // < 2^31, checked on the host
  const int t_lo = blockIdx.x, t_step = gridDim.x;
  const int tail = (P.K - (KB - 1) * kUBK + 15) >> 4;  // 16-wide K steps with data in the last block

  Ring rg{full, empty, ST};
  if (warp == 0) {
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < T; t += t_step, exch_advance(P, wk, t_step)) {
      const int arow = wk.mti * P.gpt * no, brow = wk.nti * P.wpt * 2 * no;
      const bool ok = ring_fill(rg, KB, abort_s, P.err, [&](int stage, int kb) {
        mbar_arrive_expect_tx(&full[stage], stage_bytes);
        uint8_t* sa = ring + stage * stage_bytes;
        uint8_t* sb = sa + NPC * a_bytes;
        for (int i = 0; i < NPC; ++i)
          tma_load_3d(sa + i * a_bytes, &P.ta[i], &full[stage], kb * kUBK, arow, 0);
        for (int j = 0; j < NPC; ++j)
          tma_load_3d(sb + j * b_bytes, &P.tb[j], &full[stage], kb * kUBK, brow, 0);
      });
      if (!ok) break;
    }
    ring_drain(rg, full);
  } else if (warp == 1) {
    const uint32_t ring_base = su32(ring);
    int it = 0;
    for (int t = t_lo; t < T; t += t_step, ++it) {
      const int buf = it & 1;
      const bool ok = mbar_wait_or_abort(&acce[buf], ((it >> 1) & 1) ^ 1, abort_s, P.err);
      tc_fence_after();
      const uint32_t dt = tbase + buf * acc_stride;
      if (!ok) break;
      for (int kb = 0; kb < KB; ++kb) {
        mbar_wait_run_on(&full[rg.stage], rg.phase, abort_s, P.err);
        tc_fence_after();
        const uint32_t sa = ring_base + rg.stage * stage_bytes;
        if (elect_one()) {
          issue_pairs<BN, NPC>(dt, sa, sa + NPC * a_bytes, a_bytes, b_bytes, kb + 1 < KB ? 4 : tail, kb != 0);
          umma_commit(&empty[rg.stage]);
        }
        __syncwarp();
        rg.advance();
      }
      if (elect_one()) umma_commit(&accf[buf]);
      __syncwarp();
    }
    ring_drain(rg, empty);
  } else if (warp < 10) {
    const uint32_t lane_t = tbase + ((uint32_t)((warp & 3) * 32) << 16);
    int it = 0, slot = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < T; t += t_step, ++it, exch_advance(P, wk, t_step)) {
      const int buf = it & 1;
      mbar_wait_run_on(&accf[buf], (it >> 1) & 1, abort_s, P.err);
      tc_fence_after();
      exch_tile<BN>(P, lane_t + buf * acc_stride, &acce[buf], wk.mti, wk.nti, warp - 2, slot, Fs,
                    xsum, diag, xempty, xfull, abort_s);
    }
  } else {
    int slot = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < T; t += t_step, exch_advance(P, wk, t_step))
      exch_reduce(P, wk.mti, wk.nti, warp - 10, slot, xsum, diag, xempty, xfull, abort_s);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tbase, kCols);
  }
}

// MMA with the row operand in TMEM (128 lanes, two bf16 per column, eight
// columns per 16-wide K step)
__device__ __forceinline__ void umma_bf16_ts(uint32_t dtmem, uint32_t atmem, uint32_t blo,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 db;\n setp.ne.b32 p, %4, 0;\n"
      " mov.b64 db, {%2, %5};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n}" ::"r"(dtmem),
      "r"(atmem), "r"(blo), "r"(idesc), "r"(accumulate), "r"(kDescHi)
      : "memory");
}

// the products of one K block: (0,0) into group 0, (0,1) and (1,0) into group 1.
// ahi, alo: TMEM columns of the block's row pieces; asm_lo != 0: the low piece in
// shared memory instead
template <int BN, int NKS>
__device__ __forceinline__ void exch_issue_ts(uint32_t dt, uint32_t ahi, uint32_t alo, uint32_t asm_lo,
                                              uint32_t blo, uint32_t bs, uint32_t acc) {
  constexpr uint32_t idesc = instr_desc(kUBM, BN, 1);
#pragma unroll
  for (int ks = 0; ks < NKS; ++ks) umma_bf16_ts(dt, ahi + 8 * ks, blo + 2 * ks, idesc, ks ? 1u : acc);
#pragma unroll
  for (int ks = 0; ks < NKS; ++ks)
    umma_bf16_ts(dt + BN, ahi + 8 * ks, blo + bs + 2 * ks, idesc, ks ? 1u : acc);
  if (asm_lo == 0) {
#pragma unroll
    for (int ks = 0; ks < NKS; ++ks) umma_bf16_ts(dt + BN, alo + 8 * ks, blo + 2 * ks, idesc, 1u);
  } else {
#pragma unroll
    for (int ks = 0; ks < NKS; ++ks) umma_bf16_lo(dt + BN, asm_lo + 2 * ks, blo + 2 * ks, idesc, 1u);
  }
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint4& a, const uint4& b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(
                   taddr),
               "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
               : "memory");
}

// the first n of eight bf16 values, zeros in place of the others
__device__ __forceinline__ uint4 bf16_first(uint4 v, int n) {
  auto word = [n](uint32_t u, int i) {  // values 2 i (low half) and 2 i + 1
    return n >= 2 * i + 2 ? u : (n == 2 * i + 1 ? u & 0xffffu : 0u);
  };
  return make_uint4(word(v.x, 0), word(v.y, 1), word(v.z, 2), word(v.w, 3));
}

// Row operand in TMEM, two-piece operands.  The CTA walks a contiguous range of
// tiles, so its rot_chol rows change a few times in all; four epilogue warps
// write new ones to TMEM when they meet the first tile that needs them.  MMA
// operand reads then take 32 N bytes of shared memory instead of 4096 + 32 N,
// which leaves the port to the staging.  With BN = 128 there is room for one
// accumulator buffer only: the next tile's MMAs start when the epilogue has it
// staged.
template <int BN, int NBUF>
__global__ void __launch_bounds__(kExchThreads, 1)
    umma_exch_ts_kernel(const __grid_constant__ ExchParams P) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem =
      reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int ST = P.stages, no = P.no, KB = (P.K + kUBK - 1) / kUBK, KS = (P.K + 15) >> 4;
  const int lot = P.lot, nlo = KB - lot;
  const uint32_t a_bytes = P.arows * 128, b_bytes = P.brows * 128;
  const uint32_t stage_bytes = 2 * b_bytes;
  uint8_t* alo_s = smem;
  uint8_t* ring = smem + size_t(nlo) * a_bytes;
  uint64_t* full =
      reinterpret_cast<uint64_t*>(ring + size_t(ST) * stage_bytes + exch_overread(BN, P.brows));
  uint64_t* empty = full + ST;
  uint64_t* accf = empty + ST;  // per buffer: the tile's accumulators are complete
  uint64_t* acce = accf + 2;    // per buffer: they have been read
  uint64_t* afull = acce + 2;   // the row operand is in TMEM
  uint64_t* sfull = afull + 1;  // its shared-memory blocks have landed
  uint64_t* aempty = sfull + 1; // every MMA on the previous rows has finished
  uint64_t* xfull = aempty + 1; // ring of the row sums
  uint64_t* xempty = xfull + kExchRing;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xempty + kExchRing);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float4* xsum = reinterpret_cast<float4*>(reinterpret_cast<uint8_t*>(full) + 256);
  float2* diag = reinterpret_cast<float2*>(xsum + P.ring * 256);
  float2* Fs = diag + P.ring * 128;

  constexpr uint32_t kACol = NBUF * 2 * BN;  // first column of the row operand
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], 8);
    }
    for (int b = 0; b < kExchRing; ++b) {
      mbar_init(&xfull[b], 8);
      mbar_init(&xempty[b], 1);
    }
    mbar_init(afull, 4);
    mbar_init(sfull, 1);
    mbar_init(aempty, 1);
    *abort_s = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tmem_slot;

  const int T = P.mt * P.nt;
  const int t_lo = (int)((long long)T * blockIdx.x / gridDim.x);
  const int t_hi = (int)((long long)T * (blockIdx.x + 1) / gridDim.x);
  const int tail = (P.K - (KB - 1) * kUBK + 15) >> 4;

  Ring rg{full, empty, ST};
  if (warp == 0) {
    int have = -1;
    uint32_t aphase = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < t_hi; ++t, exch_advance(P, wk, 1)) {
      if (wk.mti != have) {
        // the blocks of the low piece that stay in shared memory
        if (!mbar_wait_or_abort(aempty, aphase ^ 1, abort_s, P.err)) break;
        if (nlo && elect_one()) {
          mbar_arrive_expect_tx(sfull, nlo * a_bytes);
          for (int k = 0; k < nlo; ++k)
            tma_load_3d(alo_s + k * a_bytes, &P.ta[1], sfull, (lot + k) * kUBK, wk.mti * P.gpt * no, 0);
        }
        __syncwarp();
        have = wk.mti;
        aphase ^= 1;
      }
      const int brow = wk.nti * P.wpt * 2 * no;
      const bool ok = ring_fill(rg, KB, abort_s, P.err, [&](int stage, int kb) {
        mbar_arrive_expect_tx(&full[stage], stage_bytes);
        uint8_t* sb = ring + stage * stage_bytes;
        tma_load_3d(sb, &P.tb[0], &full[stage], kb * kUBK, brow, 0);
        tma_load_3d(sb + b_bytes, &P.tb[1], &full[stage], kb * kUBK, brow, 0);
      });
      if (!ok) break;
    }
    ring_drain(rg, full);
    if (nlo && have >= 0) mbar_wait(sfull, aphase ^ 1);  // the low piece's last blocks have landed
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t ring_base = su32(ring), alo_base = su32(alo_s), bs = b_bytes >> 4;
    const uint32_t ahi_t = tbase + kACol, alo_t = ahi_t + 8 * KS;
    int have = -1, it = 0;
    uint32_t aphase = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < t_hi; ++t, ++it, exch_advance(P, wk, 1)) {
      if (wk.mti != have) {
        if (have >= 0 && elect_one()) umma_commit(aempty);  // every MMA on the previous rows
        __syncwarp();
        mbar_wait_run_on(afull, aphase, abort_s, P.err);
        if (nlo) mbar_wait_run_on(sfull, aphase, abort_s, P.err);
        tc_fence_after();
        aphase ^= 1;
        have = wk.mti;
      }
      const int buf = NBUF == 2 ? it & 1 : 0;
      const bool ok = mbar_wait_or_abort(&acce[buf], ((it / NBUF) & 1) ^ 1, abort_s, P.err);
      tc_fence_after();
      const uint32_t dt = tbase + buf * 2 * BN;
      if (!ok) break;
      for (int kb = 0; kb < KB; ++kb) {
        mbar_wait_run_on(&full[rg.stage], rg.phase, abort_s, P.err);
        tc_fence_after();
        const uint32_t blo = smem_desc_lo(ring_base + rg.stage * stage_bytes);
        const uint32_t ahi = ahi_t + kb * 32, alo = alo_t + kb * 32;
        const uint32_t as = kb < lot ? 0u : smem_desc_lo(alo_base + (kb - lot) * a_bytes);
        const uint32_t acc = kb != 0;
        const int nks = kb + 1 < KB ? 4 : tail;
        if (elect_one()) {
          if (nks == 4) exch_issue_ts<BN, 4>(dt, ahi, alo, as, blo, bs, acc);
          else if (nks == 3) exch_issue_ts<BN, 3>(dt, ahi, alo, as, blo, bs, acc);
          else if (nks == 2) exch_issue_ts<BN, 2>(dt, ahi, alo, as, blo, bs, acc);
          else exch_issue_ts<BN, 1>(dt, ahi, alo, as, blo, bs, acc);
          umma_commit(&empty[rg.stage]);
        }
        __syncwarp();
        rg.advance();
      }
      if (elect_one()) umma_commit(&accf[buf]);
      __syncwarp();
    }
    ring_drain(rg, empty);
  } else if (warp < 10) {
    const uint32_t lane_t = tbase + ((uint32_t)((warp & 3) * 32) << 16);
    int it = 0, have = -1, slot = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < t_hi; ++t, ++it, exch_advance(P, wk, 1)) {
      if (wk.mti != have) {
        // new rows: the previous tile's accumulators were complete, so no MMA
        // reads the old ones any more
        have = wk.mti;
        if (warp < 6) {
          const int row = (warp & 3) * 32 + lane;
          const long long r = (long long)have * P.gpt * no + row;
          const bool in = row < P.gpt * no && r < (long long)P.G * no;
          const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
          for (int pc = 0; pc < 2; ++pc) {
            const uint4* src = reinterpret_cast<const uint4*>(P.a[pc] + (in ? r : 0) * P.lda);
            const int steps = pc == 0 ? KS : min(KS, lot * 4);
            const uint32_t col = lane_t + kACol + (pc ? 8 * KS : 0);
            for (int k = 0; k < steps; ++k) {
              uint4 x = in ? src[2 * k] : zero, y = in ? src[2 * k + 1] : zero;
              if (16 * (k + 1) > P.K) {  // beyond K: whatever the rows' padding holds
                x = bf16_first(x, P.K - 16 * k);
                y = bf16_first(y, P.K - 16 * k - 8);
              }
              __syncwarp();
              tmem_st8(col + 8 * k, x, y);
            }
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(afull);
        }
        __syncwarp();
      }
      const int buf = NBUF == 2 ? it & 1 : 0;
      mbar_wait_run_on(&accf[buf], (it / NBUF) & 1, abort_s, P.err);
      tc_fence_after();
      exch_tile<BN>(P, lane_t + buf * 2 * BN, &acce[buf], wk.mti, wk.nti, warp - 2, slot, Fs,
                    xsum, diag, xempty, xfull, abort_s);
    }
  } else {
    int slot = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < t_hi; ++t, exch_advance(P, wk, 1))
      exch_reduce(P, wk.mti, wk.nti, warp - 10, slot, xsum, diag, xempty, xfull, abort_s);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tbase, 512);
  }
}

}  // namespace afq
