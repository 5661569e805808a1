// Exchange energy on the tensor cores: f = RC . Theta per (Cholesky vectors x
// walkers) tile, reduced to tr f and sum f o f^T without leaving the SM
// (wavefunctions.py:1128-1174, 1331-1363).
//
// The tile is 128 rows (gpt Cholesky vectors of No rows) by BN columns (wpt
// walkers of 2 No columns).  Roles as in umma_gemm.cuh: a TMA producer warp, an
// MMA warp, one epilogue warpgroup behind two TMEM buffers.  What sets it
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
//  * Eight epilogue warps share a tile (see exch_tile).
// Measured on a B200, two pieces, per launch: N = 200, No = 40, G = 1000, W = 512
// 4.74 -> 2.43 ms; N = 300, No = 60, G = 1500, W = 1024 29.7 -> 22.8 ms; N = 250,
// No = 62, G = 1250, W = 256 4.98 -> 3.47 ms.
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
  const bf16* a[2];        // row operand pieces (the TMEM kernel loads them itself), row stride lda
  long long lda;
  float4* cout;            // (W, G): tr f as pairs (re hi, re lo, im hi, im lo)
  float4* excout;          // (mt, W): sum f o f^T, the same
  int* err;
};

// float2 per staged row: the (re, im) pairs of wsub walkers, odd so that consecutive
// rows and consecutive pairs both spread over the banks
__host__ __device__ inline int exch_row_pairs(int no, int wsub) { return (no * wsub) | 1; }

// bytes behind the ring that an MMA over bn rows reads past a box of brows rows
__host__ __device__ inline size_t exch_overread(int bn, int brows) { return size_t(bn - brows) * 128; }

// What a launch needs besides the tiling.  ts: the row operand in TMEM.
struct ExchPlan {
  int ts, nbuf, lot;  // TMEM accumulator buffers; K blocks of the low piece that sit in TMEM
  int stages, gsub, wsub;  // Cholesky vectors and walkers staged at once
  size_t smem;
};
constexpr size_t kExchSums = 4 * 128 * (2 * 16 + 8);  // ring of row sums (2 x float4) and diagonals (float2)

// sums (several walkers per tile: a float4 for each and epilogue warp) and staging of the epilogue
__host__ __device__ inline size_t exch_epi_bytes(int no, int wpt, int wsub, int gsub) {
  return ((wpt == 1 ? kExchSums : size_t(wpt) * 8 * 16) + size_t(gsub) * no * exch_row_pairs(no, wsub) * 8 + 255) & ~size_t(255);
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
  ExchPlan p{0, 0, 0, 0, 0, 0, 0};
  const int cap = max_stages >= 2 ? max_stages : 6;
  // three stages hide the load latency behind a K block's MMAs; the whole tile
  // staged at once if it fits beside them (a pass less in the epilogue), else as
  // many of its walkers as fit, or, with one walker, Cholesky vectors.  (Several
  // walkers are never cut by vectors: the threads of the other rows would stand idle in
  // every pass.  Three pieces, N = 100, No = 8, 200 walkers, where three of 16 vectors
  // fit: 197 us an energy by vectors, 86 us by walkers.)
  auto fill = [&](size_t res, size_t stage) {
    const int most = X.wpt == 1 ? X.gpt : X.wpt;
    for (int want = cap < 3 ? cap : 3; want >= 2; --want)
      for (int n = most; n >= 1; --n) {
        const int g = X.wpt == 1 ? n : X.gpt, w = X.wpt == 1 ? 1 : n;
        const size_t base = fixed + res + exch_epi_bytes(no, X.wpt, w, g);
        if (base + want * stage > kUmmaSmemBudget) continue;
        const int st = int((kUmmaSmemBudget - base) / stage);
        p.stages = st > cap ? cap : st;
        p.gsub = g;
        p.wsub = w;
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
constexpr int kExchRing = 4;  // tiles between the epilogue and the reducing warps

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

// Sums of FP32 values as unevaluated pairs hi + lo (Knuth's two-sum; about 48
// bits).  A dependent DADD takes 400 cycles while tcgen05.mma runs (the FP64 unit
// waits for the tensor core), an FADD about 14; the consumer adds hi and lo in FP64.
struct ff {
  float hi, lo;
};
__device__ __forceinline__ ff ff_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ ff ff_add(ff a, ff b) {
  const ff s = ff_two_sum(a.hi, b.hi);
  const float e = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
  const float h = __fadd_rn(s.hi, e);
  return {h, __fsub_rn(e, __fsub_rn(h, s.hi))};
}
// sums of r and i over groups of WIDTH lanes, valid in the first lane of each
template <int WIDTH>
__device__ __forceinline__ void ff_lane_sum(ff& r, ff& i) {
#pragma unroll
  for (int o = WIDTH >> 1; o > 0; o >>= 1) {
    const ff a = {__shfl_down_sync(0xffffffffu, r.hi, o), __shfl_down_sync(0xffffffffu, r.lo, o)};
    const ff b = {__shfl_down_sync(0xffffffffu, i.hi, o), __shfl_down_sync(0xffffffffu, i.lo, o)};
    r = ff_add(r, a);
    i = ff_add(i, b);
  }
}
// (re, im) pairs of such sums as they are stored
__device__ __forceinline__ float4 ff_pack(ff r, ff i) { return make_float4(r.hi, r.lo, i.hi, i.lo); }

// One tile's epilogue by eight warps: f from the accumulators (both groups
// summed in FP32) to shared memory, then per row (g, i) and walker
// sum_j f[i][j] f[j][i] in four FP32 chains (j mod 4; the last no mod 4 terms in
// chain 0), combined as pairs.  Half h of the warps moves the pairs j = 2h, 2h + 1
// (mod 4) and runs chains 2h, 2h + 1 of all 128 rows.  The loops stay rolled: the
// warps share an instruction cache with the MMA warp, and a fully unrolled form
// with the row in registers ran slower.  Everything after the chains is summed
// in pairs in a fixed order, so results are reproducible.
// One walker per tile: the row sums (xs: [2 halves][128]) and diagonals (dg: [128])
// go to the reducing warps through a ring of kExchRing tiles; several: xs holds a
// partial per (walker, warp) and the tile is finished here.
template <int BN>
__device__ __forceinline__ void exch_tile(const ExchParams& P, uint32_t taddr, uint64_t* release, int mti,
                                          int nti, int ew, int it, float2* Fs, float4* xs, float2* dg,
                                          uint64_t* xempty, uint64_t* xfull, volatile int* abort_s) {
  const int lane = threadIdx.x & 31, h = ew >> 2, row = ((threadIdx.x >> 5) & 3) * 32 + lane;
  const int no = P.no, no4 = no & ~3;
  const int gl = row / no, i = row - gl * no;
  const int fs = exch_row_pairs(no, P.wsub);
  const bool one = P.wpt == 1;
  const int g0 = mti * P.gpt, w0 = nti * P.wpt;
  const int gcount = min(P.gpt, P.G - g0), wcount = min(P.wpt, P.W - w0);
  if (one) mbar_wait_or_abort(xempty, ((it / kExchRing) & 1) ^ 1, abort_s, P.err);
  const int nall = one ? gcount : wcount, nsub = one ? P.gsub : P.wsub;
  for (int s = 0; s < nall; s += nsub) {  // Cholesky vectors (one walker) or walkers staged together
    const int n = min(nsub, nall - s);
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
    if (s + nsub >= nall) {  // the accumulators are in shared memory
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(release);
    }
    exch_sync();
    for (int wl = 0; wl < wn; ++wl) {
      ff xr = {0.f, 0.f}, xi = {0.f, 0.f};
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
        xr = ff_two_sum(ar0, ar1);
        xi = ff_two_sum(ai0, ai1);
        if (one) {
          xs[h * 128 + row] = ff_pack(xr, xi);
          if (h == 0) dg[row] = fw[i];
        }
      }
      if (!one) {
        ff_lane_sum<32>(xr, xi);
        if (lane == 0) xs[(ws + wl) * 8 + ew] = ff_pack(xr, xi);
      }
    }
    if (!one) {
      // traces of several walkers: one thread per (Cholesky vector, walker)
      for (int e = ew * 32 + lane; e < gn * wn; e += 256) {
        const int wl = e / gn, g = e - wl * gn;
        const float2* d = Fs + g * no * fs + wl * no;
        ff cr = {0.f, 0.f}, ci = {0.f, 0.f};
        for (int r = 0; r < no; ++r) {
          const float2 z = d[r * fs + r];
          cr = ff_add(cr, {z.x, 0.f});
          ci = ff_add(ci, {z.y, 0.f});
        }
        P.cout[(long long)(w0 + ws + wl) * P.G + g0 + g] = ff_pack(cr, ci);
      }
    }
    exch_sync();
  }
  if (one && lane == 0) mbar_arrive(xfull);  // every row is written (the barrier above)
  if (!one) {
    for (int wl = ew * 32 + lane; wl < wcount; wl += 256) {
      ff xr = {0.f, 0.f}, xi = {0.f, 0.f};
      for (int k = 0; k < 8; ++k) {
        const float4 p = xs[wl * 8 + k];
        xr = ff_add(xr, {p.x, p.y});
        xi = ff_add(xi, {p.z, p.w});
      }
      P.excout[(long long)mti * P.W + w0 + wl] = ff_pack(xr, xi);
    }
  }
}

// The reducing warps (one walker per tile): a tile's row sums and diagonals to
// its exchange partial and its Cholesky vectors' traces.  Four warps take the tiles in
// turn, off the epilogue's path: the chain of pair additions takes longer than a
// tile.
__device__ __forceinline__ void exch_finish(const ExchParams& P, int mti, int nti, int it, const float4* xs,
                                            const float2* dg, uint64_t* xempty, uint64_t* xfull,
                                            volatile int* abort_s) {
  const int lane = threadIdx.x & 31, no = P.no;
  const int g0 = mti * P.gpt, gcount = min(P.gpt, P.G - g0), rows = gcount * no;
  mbar_wait_or_abort(xfull, (it / kExchRing) & 1, abort_s, P.err);
  ff r[4], i[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool in = lane + 32 * k < rows;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 u = in ? xs[lane + 32 * k] : z, v = in ? xs[128 + lane + 32 * k] : z;
    r[k] = ff_add({u.x, u.y}, {v.x, v.y});
    i[k] = ff_add({u.z, u.w}, {v.z, v.w});
  }
  ff xr = ff_add(ff_add(r[0], r[1]), ff_add(r[2], r[3]));
  ff xi = ff_add(ff_add(i[0], i[1]), ff_add(i[2], i[3]));
  ff_lane_sum<32>(xr, xi);
  if (lane == 0) P.excout[(long long)mti * P.W + nti] = ff_pack(xr, xi);
  for (int gb = 0; gb < gcount; gb += 4) {  // eight lanes per Cholesky vector
    const int g = gb + (lane >> 3);
    ff cr = {0.f, 0.f}, ci = {0.f, 0.f};
    if (g < gcount)
      for (int q = lane & 7; q < no; q += 8) {
        const float2 z = dg[g * no + q];
        cr = ff_add(cr, {z.x, 0.f});
        ci = ff_add(ci, {z.y, 0.f});
      }
    __syncwarp();
    ff_lane_sum<8>(cr, ci);
    if (g < gcount && (lane & 7) == 0) P.cout[(long long)nti * P.G + g0 + g] = ff_pack(cr, ci);
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(xempty);
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
  float2* diag = reinterpret_cast<float2*>(xsum + kExchRing * 256);
  float2* Fs = P.wpt == 1 ? diag + kExchRing * 128 : reinterpret_cast<float2*>(xsum + P.wpt * 8);

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

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < T; t += t_step, exch_advance(P, wk, t_step)) {
      const int arow = wk.mti * P.gpt * no, brow = wk.nti * P.wpt * 2 * no;
      for (int kb = 0; kb < KB; ++kb) {
        mbar_wait_or_abort(&empty[stage], phase ^ 1, abort_s, P.err);
        if (elect_one()) {
          mbar_arrive_expect_tx(&full[stage], stage_bytes);
          uint8_t* sa = ring + stage * stage_bytes;
          uint8_t* sb = sa + NPC * a_bytes;
          for (int i = 0; i < NPC; ++i)
            tma_load_3d(sa + i * a_bytes, &P.ta[i], &full[stage], kb * kUBK, arow, 0);
          for (int j = 0; j < NPC; ++j)
            tma_load_3d(sb + j * b_bytes, &P.tb[j], &full[stage], kb * kUBK, brow, 0);
        }
        __syncwarp();
        if (++stage == ST) { stage = 0; phase ^= 1; }
      }
    }
    // drain (bounded): every stage that was filled has been released
    for (int s = 0; s < ST; ++s) {
      mbar_wait_or_abort(&empty[stage], phase ^ 1, abort_s, P.err);
      if (++stage == ST) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    const uint32_t ring_base = su32(ring);
    int stage = 0, it = 0;
    uint32_t phase = 0;
    for (int t = t_lo; t < T; t += t_step, ++it) {
      const int buf = it & 1;
      mbar_wait_or_abort(&acce[buf], ((it >> 1) & 1) ^ 1, abort_s, P.err);
      tc_fence_after();
      const uint32_t dt = tbase + buf * acc_stride;
      for (int kb = 0; kb < KB; ++kb) {
        mbar_wait_or_abort(&full[stage], phase, abort_s, P.err);
        tc_fence_after();
        const uint32_t sa = ring_base + stage * stage_bytes;
        if (elect_one()) {
          issue_pairs<BN, NPC>(dt, sa, sa + NPC * a_bytes, a_bytes, b_bytes, kb + 1 < KB ? 4 : tail, kb != 0);
          umma_commit(&empty[stage]);
        }
        __syncwarp();
        if (++stage == ST) { stage = 0; phase ^= 1; }
      }
      if (elect_one()) umma_commit(&accf[buf]);
      __syncwarp();
    }
  } else if (warp < 10) {
    const uint32_t lane_t = tbase + ((uint32_t)((warp & 3) * 32) << 16);
    int it = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < T; t += t_step, ++it, exch_advance(P, wk, t_step)) {
      const int buf = it & 1;
      mbar_wait_or_abort(&accf[buf], (it >> 1) & 1, abort_s, P.err);
      tc_fence_after();
      exch_tile<BN>(P, lane_t + buf * acc_stride, &acce[buf], wk.mti, wk.nti, warp - 2, it, Fs, xsum + (P.wpt == 1 ? (it % kExchRing) * 256 : 0),
                    diag + (it % kExchRing) * 128, &xempty[it % kExchRing], &xfull[it % kExchRing], abort_s);
    }
  } else if (P.wpt == 1) {
    int it = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < T; t += t_step, ++it, exch_advance(P, wk, t_step)) {
      const int q = it % kExchRing;
      if (q == warp - 10)
        exch_finish(P, wk.mti, wk.nti, it, xsum + q * 256, diag + q * 128, &xempty[q], &xfull[q], abort_s);
    }
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
      "r"(atmem), "r"(blo), "r"(idesc), "r"(accumulate), "r"(0x40004040u)
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
  float2* diag = reinterpret_cast<float2*>(xsum + kExchRing * 256);
  float2* Fs = P.wpt == 1 ? diag + kExchRing * 128 : reinterpret_cast<float2*>(xsum + P.wpt * 8);

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

  if (warp == 0) {
    int stage = 0, have = -1;
    uint32_t phase = 0, aphase = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < t_hi; ++t, exch_advance(P, wk, 1)) {
      if (wk.mti != have) {
        // the blocks of the low piece that stay in shared memory
        mbar_wait_or_abort(aempty, aphase ^ 1, abort_s, P.err);
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
      for (int kb = 0; kb < KB; ++kb) {
        mbar_wait_or_abort(&empty[stage], phase ^ 1, abort_s, P.err);
        if (elect_one()) {
          mbar_arrive_expect_tx(&full[stage], stage_bytes);
          uint8_t* sb = ring + stage * stage_bytes;
          tma_load_3d(sb, &P.tb[0], &full[stage], kb * kUBK, brow, 0);
          tma_load_3d(sb + b_bytes, &P.tb[1], &full[stage], kb * kUBK, brow, 0);
        }
        __syncwarp();
        if (++stage == ST) { stage = 0; phase ^= 1; }
      }
    }
    // drain (bounded): every stage that was filled has been released, and
    // the low piece's last blocks have landed and been read
    for (int s = 0; s < ST; ++s) {
      mbar_wait_or_abort(&empty[stage], phase ^ 1, abort_s, P.err);
      if (++stage == ST) { stage = 0; phase ^= 1; }
    }
    mbar_wait_or_abort(aempty, aphase ^ 1, abort_s, P.err);
  } else if (warp == 1) {
    const uint32_t ring_base = su32(ring), alo_base = su32(alo_s), bs = b_bytes >> 4;
    const uint32_t ahi_t = tbase + kACol, alo_t = ahi_t + 8 * KS;
    int stage = 0, have = -1, it = 0;
    uint32_t phase = 0, aphase = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < t_hi; ++t, ++it, exch_advance(P, wk, 1)) {
      if (wk.mti != have) {
        if (have >= 0 && elect_one()) umma_commit(aempty);  // every MMA on the previous rows
        __syncwarp();
        mbar_wait_or_abort(afull, aphase, abort_s, P.err);
        if (nlo) mbar_wait_or_abort(sfull, aphase, abort_s, P.err);
        tc_fence_after();
        aphase ^= 1;
        have = wk.mti;
      }
      const int buf = NBUF == 2 ? it & 1 : 0;
      mbar_wait_or_abort(&acce[buf], ((it / NBUF) & 1) ^ 1, abort_s, P.err);
      tc_fence_after();
      const uint32_t dt = tbase + buf * 2 * BN;
      for (int kb = 0; kb < KB; ++kb) {
        mbar_wait_or_abort(&full[stage], phase, abort_s, P.err);
        tc_fence_after();
        const uint32_t blo = smem_desc_lo(ring_base + stage * stage_bytes);
        const uint32_t ahi = ahi_t + kb * 32, alo = alo_t + kb * 32;
        const uint32_t as = kb < lot ? 0u : smem_desc_lo(alo_base + (kb - lot) * a_bytes);
        const uint32_t acc = kb != 0;
        const int nks = kb + 1 < KB ? 4 : tail;
        if (elect_one()) {
          if (nks == 4) exch_issue_ts<BN, 4>(dt, ahi, alo, as, blo, bs, acc);
          else if (nks == 3) exch_issue_ts<BN, 3>(dt, ahi, alo, as, blo, bs, acc);
          else if (nks == 2) exch_issue_ts<BN, 2>(dt, ahi, alo, as, blo, bs, acc);
          else exch_issue_ts<BN, 1>(dt, ahi, alo, as, blo, bs, acc);
          umma_commit(&empty[stage]);
        }
        __syncwarp();
        if (++stage == ST) { stage = 0; phase ^= 1; }
      }
      if (elect_one()) umma_commit(&accf[buf]);
      __syncwarp();
    }
    if (have >= 0 && elect_one()) umma_commit(aempty);
    __syncwarp();
  } else if (warp < 10) {
    const uint32_t lane_t = tbase + ((uint32_t)((warp & 3) * 32) << 16);
    int it = 0, have = -1;
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
              const uint4 x = in ? src[2 * k] : zero, y = in ? src[2 * k + 1] : zero;
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
      mbar_wait_or_abort(&accf[buf], (it / NBUF) & 1, abort_s, P.err);
      tc_fence_after();
      exch_tile<BN>(P, lane_t + buf * 2 * BN, &acce[buf], wk.mti, wk.nti, warp - 2, it, Fs, xsum + (P.wpt == 1 ? (it % kExchRing) * 256 : 0),
                    diag + (it % kExchRing) * 128, &xempty[it % kExchRing], &xfull[it % kExchRing], abort_s);
    }
  } else if (P.wpt == 1) {
    int it = 0;
    ExchWalk wk = exch_locate(P, t_lo);
    for (int t = t_lo; t < t_hi; t += 1, ++it, exch_advance(P, wk, 1)) {
      const int q = it % kExchRing;
      if (q == warp - 10)
        exch_finish(P, wk.mti, wk.nti, it, xsum + q * 256, diag + q * 128, &xempty[q], &xfull[q], abort_s);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tbase, 512);
  }
}

}  // namespace afq
