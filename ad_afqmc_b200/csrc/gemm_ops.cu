// FP64 dense contractions of the phaseless step and of the local energy.
//
//  force bias   fb[w,g]   = mult * sum_k Gpl[(w,c),k] * RCcat[g,k]
//               (wavefunctions.py:1102-1126, 1314-1329)
//  field prep   x~ = x - fs, fs = -sqrt(dt)(i fb - mf), shift/fb terms
//               (propagation.py:295-301)
//  VHS          VHS[w] = i sqrt(dt) sum_g x~[w,g] L_g   (propagation.py:196-203)
//  propagator   y = e^{-dt h/2} w; y += sum_n VHS^n y / n!; w' = e^{-dt h/2} y
//               (propagation.py:154-176, 206-229)
//  exchange     f[g,w] = rot_chol[g] Theta_w ; c = tr f ; x = sum f o f^T
//               fused: f lives only in registers/shared memory
//               (wavefunctions.py:1128-1174, 1331-1363)
#include "common.cuh"
#include "f64_tma.cuh"
#include "ops.h"
#include "profile.cuh"

namespace afq {

int sm_count();

namespace {

// ---------------------------------------------------------------------------
// force bias: C[z] (2W x G) = Gpl (2W x Kfb) * RCcat^T, K split over z
// ---------------------------------------------------------------------------
struct FbEpi {
  double* C;
  long long ldc, zstride;
  int M, N;
  template <class T>
  __device__ void tile(const F64At& at, double (&acc)[T::FM][T::NG][2][2], int wm, int wn, int g, int t4,
                       uint8_t*) const {
    double* const Cz = C + at.z * zstride;
    f64_each<T>(acc, wm, wn, g, t4, [&](int r, int c, double v0, double v1, double v2, double v3) {
      const int m = at.mti * T::BM + r, n = at.nti * T::BN + c;
      if (m >= M) return;
      double* p = Cz + m * ldc + n;  // ldc even, n even: pairs are aligned, the pad column is never read
      if (n < N) *reinterpret_cast<double2*>(p) = make_double2(v0, v1);
      if (n + 2 < N) *reinterpret_cast<double2*>(p + 2) = make_double2(v2, v3);
    });
  }
};

// ---------------------------------------------------------------------------
// field preparation (one CTA per walker)
// ---------------------------------------------------------------------------
// one compiled copy for the solo and the grouped kernel (identical rounding)
// fbpart: split-K partial sums of the force bias, FP64 (FP64 path) or FP32
// (f32: the tensor-core path's FP32 accumulators, stored as they are)
__device__ __noinline__ void prep_body(int W, int G, long long Gpad, int splitk,
                                          const void* fbpart, int f32, double alpha, const double* fields,
                                          const double* mf, double sdt, double* xt, double* wscal,
                                          double* fb_out, int npc, bf16* xb0, bf16* xb1, bf16* xb2,
                                          long long ldxb, int w) {
  bf16* const xb[3] = {xb0, xb1, xb2};
  __shared__ double red[4 * 8];
  const int tid = threadIdx.x;
  const long long zs = 2LL * W * Gpad;
  double sr = 0, si = 0, br = 0, bi = 0;
  for (int g = tid; g < G; g += blockDim.x) {
    double fr = 0.0, fi = 0.0;
    if (f32) {
      const float* fp = static_cast<const float*>(fbpart);
      for (int z = 0; z < splitk; ++z) {
        fr += (double)fp[z * zs + (2LL * w) * Gpad + g];
        fi += (double)fp[z * zs + (2LL * w + 1) * Gpad + g];
      }
    } else {
      const double* dp = static_cast<const double*>(fbpart);
      for (int z = 0; z < splitk; ++z) {
        fr += dp[z * zs + (2LL * w) * Gpad + g];
        fi += dp[z * zs + (2LL * w + 1) * Gpad + g];
      }
    }
    fr *= alpha;
    fi *= alpha;
    if (fb_out) {
      fb_out[2 * ((long long)w * G + g)] = fr;
      fb_out[2 * ((long long)w * G + g) + 1] = fi;
    }
    if (fields) {
      const double mfr = mf[2 * g], mfi = mf[2 * g + 1];
      // field_shifts = -sqrt(dt) * (i*fb - mf_shifts)
      const double fsr = -sdt * (-fi - mfr);
      const double fsi = -sdt * (fr - mfi);
      const double x = fields[(long long)w * G + g];
      const double xr = x - fsr, xi = -fsi;  // shifted field
      sr += xr * mfr - xi * mfi;
      si += xr * mfi + xi * mfr;
      br += x * fsr - (fsr * fsr - fsi * fsi) / 2.0;
      bi += x * fsi - (2.0 * fsr * fsi) / 2.0;
      // VHS = i sqrt(dt) x~ L  ->  rows (w,0)=Re VHS, (w,1)=Im VHS
      if (xb0) {
        put_pieces(-sdt * xi, npc, xb, (2LL * w) * ldxb + g);
        put_pieces(sdt * xr, npc, xb, (2LL * w + 1) * ldxb + g);
      } else {
        xt[(2LL * w) * Gpad + g] = -sdt * xi;
        xt[(2LL * w + 1) * Gpad + g] = sdt * xr;
      }
    }
  }
  if (fields) {
    sr = block_sum(sr, red);
    si = block_sum(si, red + 8);
    br = block_sum(br, red + 16);
    bi = block_sum(bi, red + 24);
    if (tid == 0) {
      double* s = wscal + (long long)w * 16;
      s[0] = sr;
      s[1] = si;
      s[2] = br;
      s[3] = bi;
    }
  }
}

__global__ void __launch_bounds__(256) prep_kernel(int W, int G, long long Gpad, int splitk,
                                                   const void* fbpart, int f32, double alpha,
                                                   const double* fields, const double* mf,
                                                   double sdt, double* xt, double* wscal,
                                                   double* fb_out, int npc, bf16* xb0, bf16* xb1,
                                                   bf16* xb2, long long ldxb) {
  prep_body(W, G, Gpad, splitk, fbpart, f32, alpha, fields, mf, sdt, xt, wscal, fb_out, npc, xb0,
            xb1, xb2, ldxb, blockIdx.x);
}

__global__ void __launch_bounds__(256) prep_kernel_grouped(const PrepArgs* A, BlockMap m, int step) {
  int local;
  const PrepArgs& a = A[block_owner(m, blockIdx.x, local)];
  prep_body(a.W, a.G, a.Gpad, a.splitk, a.fbpart, a.f32, a.alpha, a.fields + (long long)step * a.field_step,
            a.mf, a.sdt, a.xt, a.wscal, nullptr, a.npc, a.xb[0], a.xb[1], a.xb[2], a.ldxb, local);
}

// ---------------------------------------------------------------------------
// VHS: C (2W x N*N) = Xt (2W x G) * chol (G x N*N), scattered to (W, N, 2Npad)
// ---------------------------------------------------------------------------
struct VhsEpi {
  double* vhs;
  int M, NN, N;
  long long Npad;
  template <class T>
  __device__ void tile(const F64At& at, double (&acc)[T::FM][T::NG][2][2], int wm, int wn, int g, int t4,
                       uint8_t*) const {
    const long long ld = 2 * Npad;
    const int n_ = N;
    f64_each<T>(acc, wm, wn, g, t4, [&](int row, int c, double v0, double v1, double v2, double v3) {
      const int m = at.mti * T::BM + row, n = at.nti * T::BN + c;
      if (m >= M || n >= NN) return;
      double* base = vhs + (long long)(m >> 1) * n_ * ld + (m & 1) * Npad;
      int p = n / n_, r = n - p * n_;
      const double v[4] = {v0, v1, v2, v3};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (n + q < NN) base[(long long)p * ld + r] = v[q];
        if (++r == n_) { r = 0; ++p; }
      }
    });
  }
};

// ---------------------------------------------------------------------------
// batched per-walker products of the one-body half-steps and the Taylor series
// (Horner: z_{n-1} = y + VHS z_n / n):  out = (yin) + scale * A B
// ---------------------------------------------------------------------------
struct PropEpi {
  double* out;
  const double* yin;  // nullptr: none
  double scale;
  int M, nc;
  template <class T>
  __device__ void tile(const F64At& at, double (&acc)[T::FM][T::NG][2][2], int wm, int wn, int g, int t4,
                       uint8_t*) const {
    const long long boff = (long long)at.z * M * nc;
    const double s = scale;
    const double* const y = yin ? yin + boff : nullptr;
    double* const o = out + boff;
    const int M_ = M, n_ = nc;
    f64_each<T>(acc, wm, wn, g, t4, [&](int row, int c, double v0, double v1, double v2, double v3) {
      const int m = at.mti * T::BM + row, n = at.nti * T::BN + c;
      if (m >= M_ || n >= n_) return;
      const long long e = (long long)m * n_ + n;
      double2 u = make_double2(s * v0, s * v1), w = make_double2(s * v2, s * v3);
      const bool two = n + 2 < n_;  // nc is even
      if (y) {
        const double2 y0 = *reinterpret_cast<const double2*>(y + e);
        u = make_double2(y0.x + u.x, y0.y + u.y);
        if (two) {
          const double2 y1 = *reinterpret_cast<const double2*>(y + e + 2);
          w = make_double2(y1.x + w.x, y1.y + w.y);
        }
      }
      *reinterpret_cast<double2*>(o + e) = u;
      if (two) *reinterpret_cast<double2*>(o + e + 2) = w;
    });
  }
};

template <class T>
__device__ __forceinline__ void f64_consumer_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(32 * T::CW) : "memory");
}

// The tile of f in shared memory: rows (Cholesky vector, i), a walker's 2 No columns
// one after the other; row stride BN + 2 doubles, so that 16-byte loads
// down a column (4 banks apart) and along a row are conflict-free.
template <class T>
__device__ __forceinline__ double* exch_stage(double (&acc)[T::FM][T::NG][2][2], int cols, int wm, int wn, int g,
                                              int t4, uint8_t* smem) {
  constexpr int CS = T::BN + 2;
  double* Ct = reinterpret_cast<double*>(smem);
#pragma unroll
  for (int n = 0; n < T::NG; ++n) {
    const int c0 = (wn * T::NG + n) * 16;
    if (c0 >= cols) continue;  // warp-uniform
    const bool half = cols - c0 <= 8;  // only the first MMA tile, its columns in order
    double* p = Ct + (wm * T::FM * 8 + g) * CS + c0 + (half ? 2 : 4) * t4;
#pragma unroll
    for (int i = 0; i < T::FM; ++i) {
      *reinterpret_cast<double2*>(p + i * 8 * CS) = make_double2(acc[i][n][0][0], acc[i][n][0][1]);
      if (!half) *reinterpret_cast<double2*>(p + i * 8 * CS + 2) = make_double2(acc[i][n][1][0], acc[i][n][1][1]);
    }
  }
  f64_consumer_sync<T>();
  return Ct;
}
template <class T>
inline size_t exch_stage_bytes(int extra) {
  return size_t(T::BM) * (T::BN + 2) * 8 + size_t(extra) * 8;
}

// ---------------------------------------------------------------------------
// fused exchange: tile = gpt Cholesky vectors x wpt walkers.  Per block (g, w):
// tr f and sum_ij f_ij f_ji = sum_i f_ii^2 + 2 sum_{i<j} f_ij f_ji.
// ---------------------------------------------------------------------------
struct ExchEpi {
  int G, no, W, gpt, wpt;
  double* cout;
  double* excout;
  template <class T>
  __device__ void tile(const F64At& at, double (&acc)[T::FM][T::NG][2][2], int wm, int wn, int g, int t4,
                       uint8_t* smem) const {
    constexpr int CS = T::BN + 2, CW = T::CW;
    const double* Ct = exch_stage<T>(acc, 2 * no * wpt, wm, wn, g, t4, smem);
    double4* blk = reinterpret_cast<double4*>(smem + size_t(T::BM) * CS * 8);  // [CW or more][block]
    const int g0 = at.mti * gpt, w0 = at.nti * wpt;
    const int gcount = min(gpt, G - g0), wcount = min(wpt, W - w0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nblk = gcount * wcount, parts = max(1, CW / nblk);
    // The lanes walk the triangle i <= j folded to a rectangle: row r holds the No - r
    // entries of row r and the r + 1 of row No - 1 - r (odd No: the middle row alone).
    const int len = no + 1, di = 32 * parts / len, dj = 32 * parts - di * len;
    for (int e = warp; e < nblk * parts; e += CW) {
      const int b = e / parts, part = e - b * parts;
      const int gl = b % gcount, wl = b / gcount;
      const double* F = Ct + (gl * CS + 2 * wl) * no;
      double er = 0, ei = 0, dr = 0, dgi = 0, cr = 0, ci = 0;
      int r = (part * 32 + lane) / len, q = part * 32 + lane - r * len;
      while (2 * r < no) {
        const bool second = q >= no - r;
        const int i = second ? no - 1 - r : r, j = second ? i + q - (no - r) : r + q;
        if (!second || 2 * r + 1 < no) {
          const double2 fij = *reinterpret_cast<const double2*>(F + i * CS + 2 * j);
          const double2 fji = *reinterpret_cast<const double2*>(F + j * CS + 2 * i);
          const double pr = fij.x * fji.x - fij.y * fji.y, pi = fij.x * fji.y + fij.y * fji.x;
          if (i == j) {
            dr += pr;
            dgi += pi;
            cr += fij.x;
            ci += fij.y;
          } else {
            er += pr;
            ei += pi;
          }
        }
        r += di;
        q += dj;
        if (q >= len) {
          q -= len;
          ++r;
        }
      }
      er = dr + 2.0 * er;
      ei = dgi + 2.0 * ei;
      // the four sums by one exchange of halves each: lane 8 q ends with the q-th
      const bool up = lane & 16, up8 = lane & 8;
      double a = up ? cr : er, b2 = up ? ci : ei;
      a += __shfl_xor_sync(0xffffffffu, up ? er : cr, 16);
      b2 += __shfl_xor_sync(0xffffffffu, up ? ei : ci, 16);
      double c = up8 ? b2 : a;
      c += __shfl_xor_sync(0xffffffffu, up8 ? a : b2, 8);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
      if ((lane & 7) == 0) reinterpret_cast<double*>(blk + e)[lane >> 3] = c;
    }
    f64_consumer_sync<T>();
    for (int b = threadIdx.x; b < nblk; b += 32 * CW) {
      double4 s = blk[b * parts];
      for (int q = 1; q < parts; ++q) {
        const double4 u = blk[b * parts + q];
        s.x += u.x; s.y += u.y; s.z += u.z; s.w += u.w;
      }
      const long long co = 2 * ((long long)(w0 + b / gcount) * G + g0 + b % gcount);
      cout[co] = s.z;
      cout[co + 1] = s.w;
    }
    for (int wl = CW - 1 - warp; wl < wcount; wl += CW) {  // a warp per walker
      const double4* u = blk + wl * gcount * parts;
      double sx = 0, sy = 0;
      for (int e = lane; e < gcount * parts; e += 32) {
        sx += u[e].x;
        sy += u[e].y;
      }
      sx = warp_sum(sx);
      sy = warp_sum(sy);
      if (lane == 0) {
        excout[2 * ((long long)at.mti * W + w0 + wl)] = sx;
        excout[2 * ((long long)at.mti * W + w0 + wl) + 1] = sy;
      }
    }
    f64_consumer_sync<T>();
  }
};

// ---------------------------------------------------------------------------
// LNO orbital energy (rhf_lno._calc_orbenergy, wavefunctions.py:6904-6923):
// f = RC[g] . Theta_vir per (Cholesky vector, walker), Theta's occupied rows
// zeroed beforehand (so only rot_chol's virtual columns contribute), staged
// in shared memory as in the exchange.  With m = sum_r p_r^T p_r (prjlo rows
// p_r): c = tr f, s1 = sum_r p_r f p_r^T (= sum f o m), s2 = sum_r (p_r f).(f
// p_r^T) (= sum (f f) o m); the tile's partial sum_g (2 c s1 - s2) per walker.
// ---------------------------------------------------------------------------
constexpr int kMaxLo = 8;

struct OrbEpi {
  int G, no, W, gpt, wpt, nlo;
  const double* prj;
  double* orbout;
  template <class T>
  __device__ void tile(const F64At& at, double (&acc)[T::FM][T::NG][2][2], int wm, int wn, int g, int t4,
                       uint8_t* smem) const {
    constexpr int CS = T::BN + 2, CW = T::CW;
    double* P = reinterpret_cast<double*>(smem) + T::BM * CS;  // nlo x no projector rows
    double2* blk = reinterpret_cast<double2*>(P + kMaxLo * 64);
    for (int e = threadIdx.x; e < nlo * no; e += 32 * CW) P[e] = prj[e];
    const double* Ct = exch_stage<T>(acc, 2 * no * wpt, wm, wn, g, t4, smem);
    const int g0 = at.mti * gpt, w0 = at.nti * wpt;
    const int gcount = min(gpt, G - g0), wcount = min(wpt, W - w0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nblk = gcount * wcount;
    for (int bi = warp; bi < nblk; bi += CW) {
      const int gl = bi % gcount, wl = bi / gcount;
      const double* F = Ct + (gl * CS + 2 * wl) * no;
      double cr = 0, ci = 0, ar = 0, ai = 0, br = 0, bi_ = 0;
      for (int k = lane; k < no; k += 32) {
        cr += F[k * CS + 2 * k];
        ci += F[k * CS + 2 * k + 1];
      }
      for (int r = 0; r < nlo; ++r) {
        const double* p = P + r * no;
        for (int k = lane; k < no; k += 32) {
          double ur = 0, ui = 0, vr = 0, vi = 0;  // u = (p f)[k], v = (f p^T)[k]
          for (int x = 0; x < no; ++x) {
            const double2 fu = *reinterpret_cast<const double2*>(F + x * CS + 2 * k);
            const double2 fv = *reinterpret_cast<const double2*>(F + k * CS + 2 * x);
            ur = fma(p[x], fu.x, ur);
            ui = fma(p[x], fu.y, ui);
            vr = fma(fv.x, p[x], vr);
            vi = fma(fv.y, p[x], vi);
          }
          ar = fma(ur, p[k], ar);
          ai = fma(ui, p[k], ai);
          br += ur * vr - ui * vi;
          bi_ += ur * vi + ui * vr;
        }
      }
      cr = warp_sum(cr);
      ci = warp_sum(ci);
      ar = warp_sum(ar);
      ai = warp_sum(ai);
      br = warp_sum(br);
      bi_ = warp_sum(bi_);
      if (lane == 0)  // 2 c s1 - s2
        blk[gl * wpt + wl] = make_double2(2.0 * (cr * ar - ci * ai) - br, 2.0 * (cr * ai + ci * ar) - bi_);
    }
    f64_consumer_sync<T>();
    for (int wl = threadIdx.x; wl < wcount; wl += 32 * CW) {
      double sx = 0, sy = 0;
      for (int gl = 0; gl < gcount; ++gl) {
        const double2 v = blk[gl * wpt + wl];
        sx += v.x;
        sy += v.y;
      }
      orbout[2 * ((long long)at.mti * W + w0 + wl)] = sx;
      orbout[2 * ((long long)at.mti * W + w0 + wl) + 1] = sy;
    }
    f64_consumer_sync<T>();
  }
};

// Theta (rows (walker, i, re/im) of N doubles at stride ld): columns p < No set to
// zero (the occupied block)
__global__ void theta_zero_occ_kernel(double* theta, long long rows, long long ld, int no) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < rows * no;
       e += (long long)gridDim.x * blockDim.x)
    theta[e / no * ld + e % no] = 0.0;
}

// orbital energy per walker: sum of the row-tile partials (one warp per walker)
__global__ void orb_combine_kernel(int W, int mt, const double* part, double* out) {
  const int lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= W) return;
  double xr = 0, xi = 0;
  for (int m = lane; m < mt; m += 32) {
    xr += part[2 * ((long long)m * W + w)];
    xi += part[2 * ((long long)m * W + w) + 1];
  }
  xr = warp_sum(xr);
  xi = warp_sum(xi);
  if (lane == 0) {
    out[2LL * w] = xr;
    out[2LL * w + 1] = xi;
  }
}

// ---------------------------------------------------------------------------
// local energy from the pieces (one warp per walker)
// ---------------------------------------------------------------------------
__global__ void energy_combine_kernel(int W, int G, int ns, int restricted, const double* scal,
                                      const double* c0, const double* c1, const double* x0,
                                      int mt0, const double* x1, int mt1, const double* wscal,
                                      double* eout, int eout_stride) {
  const int lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= W) return;
  double jr = 0, ji = 0, xr = 0, xi = 0;
  for (int g = lane; g < G; g += 32) {
    double2 a = reinterpret_cast<const double2*>(c0)[(long long)w * G + g];
    if (ns == 2) a = cadd(a, reinterpret_cast<const double2*>(c1)[(long long)w * G + g]);
    jr += a.x * a.x - a.y * a.y;
    ji += 2.0 * a.x * a.y;
  }
  for (int m = lane; m < mt0; m += 32) {
    const double2 x = reinterpret_cast<const double2*>(x0)[(long long)m * W + w];
    xr += x.x;
    xi += x.y;
  }
  if (ns == 2)
    for (int m = lane; m < mt1; m += 32) {
      const double2 x = reinterpret_cast<const double2*>(x1)[(long long)m * W + w];
      xr += x.x;
      xi += x.y;
    }
  jr = warp_sum(jr);
  ji = warp_sum(ji);
  xr = warp_sum(xr);
  xi = warp_sum(xi);
  if (lane == 0) {
    const double* s = wscal + (long long)w * 16;
    const double h0 = scal[0];
    double er, ei;
    if (restricted) {
      // 2 sum c^2 - exc + 2 E1 + h0
      er = 2.0 * jr - xr + 2.0 * s[8] + h0;
      ei = 2.0 * ji - xi + 2.0 * s[9];
    } else {
      // ((c_up + c_dn)^2 - exc_up - exc_dn) / 2 + E1_up + E1_dn + h0
      er = 0.5 * (jr - xr) + s[8] + s[10] + h0;
      ei = 0.5 * (ji - xi) + s[9] + s[11];
    }
    eout[(long long)w * eout_stride] = er;
    eout[(long long)w * eout_stride + 1] = ei;
  }
}

// Tile of the two plain contractions (force bias, VHS): from 128 x 128 (8 warps,
// 32 x 64 each) down to 32 x 32, whichever gives the shortest sum of waves; a tile
// costs its MMAs per warp (FM NG) and about 1.5 for its loads and stores.  A
// wave of big tiles that leaves SMs idle loses to more waves of smaller ones
// (N = 95, G = 471, 161 walkers, force bias: 64 x 64 tiles).
template <int BMODE, class F>
cudaError_t with_gemm_tile(long long M, long long N, int nz, F&& f) {
  const int fm[5] = {4, 2, 2, 1, 1}, ng[5] = {4, 4, 2, 2, 1}, sms = sm_count();
  int best = 0;
  double cost = 1e300;
  for (int i = 0; i < 5; ++i) {
    const long long tiles = ((M + 32 * fm[i] - 1) / (32 * fm[i])) * ((N + 32 * ng[i] - 1) / (32 * ng[i])) * nz;
    const double c = double((tiles + sms - 1) / sms) * (fm[i] * ng[i] + 1.5);
    if (c < cost - 1e-9) { cost = c; best = i; }
  }
  switch (best) {
    case 0: return f(F64Tile<4, 2, 4, F64_REAL, BMODE>());
    case 1: return f(F64Tile<2, 2, 4, F64_REAL, BMODE>());
    case 2: return f(F64Tile<2, 2, 2, F64_REAL, BMODE>());
    case 3: return f(F64Tile<1, 2, 2, F64_REAL, BMODE>());
    default: return f(F64Tile<1, 2, 1, F64_REAL, BMODE>());
  }
}

int* f64_err(const Layout& L, double* work) { return reinterpret_cast<int*>(work + L.w_misc); }

// CTAs for a persistent launch of a kernel of `threads` threads and tiles of
// shared memory `smem`: small tiles share an SM
int f64_ctas(int threads, size_t smem) {
  int per = (int)(kF64SmemBudget / (smem ? smem : 1));
  const int byt = 1024 / threads;
  if (per > byt) per = byt;
  return sm_count() * (per < 1 ? 1 : (per > 3 ? 3 : per));
}

struct PropCall {
  const double *a1, *a2;  // A (second: imaginary part), row stride lda, batch stride abs (0: shared)
  long long lda, abs;
  const double* b;        // (W, N, nc)
  double* out;
  const double* yin;
  double scale;
};

template <int FM, int WN, int KIND>
cudaError_t prop_run(const Layout& L, double* work, int nc, const PropCall& c, cudaStream_t st) {
  using T = F64Tile<FM, WN, 1, KIND, F64_B_N>;
  F64Params<PropEpi> P{};
  const int N = L.N, W = L.W;
  const int nb = c.abs ? W : 1;
  if (make_tmap_f64(&P.ta, c.a1, N, N, nb, c.lda, c.abs ? c.abs : c.lda * N, 8, T::BM) != AFQ_OK ||
      (KIND == F64_COMPLEX && make_tmap_f64(&P.ta2, c.a2, N, N, nb, c.lda, c.abs, 8, T::BM) != AFQ_OK) ||
      make_tmap_f64(&P.tb, c.b, nc, N, W, nc, (long long)N * nc, 16, 16) != AFQ_OK)
    return cudaErrorInvalidValue;
  P.s.K = N;
  P.s.mt = (N + T::BM - 1) / T::BM;
  P.s.nt = (nc + T::BN - 1) / T::BN;
  P.s.nz = W;
  P.s.arow_step = T::BM;
  P.s.a_batched = c.abs != 0;
  P.s.err = f64_err(L, work);
  P.epi = PropEpi{c.out, c.yin, c.scale, N, nc};
  // few warps: two or three CTAs an SM if each keeps three stages, so that one's
  // loads and stores run under another's MMAs (N = 34, No = 12, 10000 walkers, seven launches:
  // 1.56 ms with six stages and one CTA, 1.24 so; 1.26 with the cp.async kernel before)
  int per = T::CW <= 4 ? 3 : (T::CW <= 8 ? 2 : 1);
  while (per > 1 && f64_stages<T>(0, per) < 3) --per;
  P.s.stages = f64_stages<T>(0, per);
  const size_t smem = 1024 + P.s.stages * size_t(T::STAGE) + 256;
  ProfScope ps(K_PROP, st);
  return f64_launch<T>(P, f64_ctas(T::NT, smem), st);
}

// Tile of the per-walker products: 32 FM rows by 16 WN columns.  Every scheduler
// runs WN of the 4 WN consumer warps, 2 FM MMAs per K step each, so a tile costs
// FM WN and the launch ceil(tiles / SMs) of them; the choice with the least padding
// and the fullest last wave (N = 200, No = 40, 512 walkers: 7 x 5, 4 waves).
template <int KIND>
cudaError_t prop_gemm(const Layout& L, double* work, int nc, const PropCall& c, cudaStream_t st) {
  const int fms[6] = {1, 2, 3, 4, 5, 7};
  const int groups = (nc + 15) / 16, sms = sm_count();
  double best = 1e300;
  int bf = 1, bw = 1;
  for (int fm : fms)
    for (int wn = 1; wn <= 5; ++wn) {
      const long long tiles = (long long)((L.N + 32 * fm - 1) / (32 * fm)) * ((groups + wn - 1) / wn) * L.W;
      const double cost = double((tiles + sms - 1) / sms) * (fm * wn + 1.0) * (wn == 1 ? 1.3 : 1.0);
      if (cost < best - 1e-9) { best = cost; bf = fm; bw = wn; }
    }
#define AFQ_PROP_WN(FM)                                              \
  switch (bw) {                                                      \
    case 1: return prop_run<FM, 1, KIND>(L, work, nc, c, st);        \
    case 2: return prop_run<FM, 2, KIND>(L, work, nc, c, st);        \
    case 3: return prop_run<FM, 3, KIND>(L, work, nc, c, st);        \
    case 4: return prop_run<FM, 4, KIND>(L, work, nc, c, st);        \
    default: return prop_run<FM, 5, KIND>(L, work, nc, c, st);       \
  }
  switch (bf) {
    case 1: AFQ_PROP_WN(1)
    case 2: AFQ_PROP_WN(2)
    case 3: AFQ_PROP_WN(3)
    case 4: AFQ_PROP_WN(4)
    case 5: AFQ_PROP_WN(5)
    default: AFQ_PROP_WN(7)
  }
#undef AFQ_PROP_WN
}

// Exchange and orbital-energy tiles: 128 rows (gpt Cholesky vectors) and the 2 No columns
// of wpt walkers, which lie one after the other in Theta's rows; calls f with the tile type.
// The choice with the smallest ceil(tiles / SMs) times the tile's MMA tiles of eight columns
// (plus 2.2 for its share of A, its loads and barriers: the fit to No = 9 with 1 to 4 walkers);
// at most 512 (Cholesky vector, walker) blocks, whose sums sit in shared memory.
// 80 columns leave room for four operand stages; 96, with three, pay where they hold more
// of the walkers (No = 15, 16, 21 to 24); 112, in 28 warps, two walkers of No = 25 to 28 (N = 60,
// No = 26, 1024 walkers 2.87 -> 2.38 ms); 128, with two stages, only hold what needs them.
// With every walker padded to groups of 16 columns, at most four to a tile, No = 2, 4, 9, 10, 26
// took longer than the kernel before, whose tiles held whole walkers without
// padding (energies at N = 300, 1024 walkers, ms, that one, padded, now: No = 2 0.90, 1.24, 0.66;
// No = 9 5.95, 7.25, 4.32; No = 10 7.02, 8.42, 5.38; No = 20 25.6, 23.7, 20.3).
template <class F>
cudaError_t with_exch_tile(int no, int G, int W, int& wpt, F&& f) {
  const int gpt = 128 / no, most = 512 / gpt, sms = sm_count();
  const long long mt = (G + gpt - 1) / gpt;
  double best = 1e300;
  int bn = 128;
  wpt = 1;
  for (int b : {80, 96, 112})
    for (int n = 1; n <= most && 2 * no * n <= b && (b < 112 || (no >= 25 && no <= 28)); ++n) {
      const long long waves = (mt * ((W + n - 1) / n) + sms - 1) / sms;
      const double cost = double(waves) * ((2 * no * n + 7) / 8 + 2.2) * (b > 80 ? 1.05 : 1.0);
      if (cost < best - 1e-9) {
        best = cost;
        bn = b;
        wpt = n;
      }
    }
  switch (bn) {
    case 80: return f(F64Tile<4, 5, 1, F64_REAL, F64_B_K, true>());
    case 96: return f(F64Tile<4, 3, 2, F64_REAL, F64_B_K, true>());
    case 112: return f(F64Tile<4, 7, 1, F64_REAL, F64_B_K, true>());
    default: return f(F64Tile<4, 4, 2, F64_REAL, F64_B_K, true>());
  }
}

template <class T, class Epi>
cudaError_t exch_run(const Layout& L, const double* prep, double* work, int s, F64Params<Epi>& P, int wpt,
                     int extra, cudaStream_t st) {
  const int no = L.no[s], gpt = L.ex[s].gpt;
  const long long rows = (long long)L.W * 2 * no;
  if (make_tmap_f64(&P.ta, prep + L.p_rc[s], L.N, (long long)L.G * no, 1, L.Npad, L.Npad * L.G * no, 8, T::BM) !=
          AFQ_OK ||
      make_tmap_f64(&P.tb, work + L.w_theta[s], L.N, rows, 1, L.Npad, L.Npad * rows, 8, wpt * 2 * no) != AFQ_OK)
    return cudaErrorInvalidValue;
  P.s.K = L.N;
  P.s.mt = (L.G + gpt - 1) / gpt;
  P.s.nt = (L.W + wpt - 1) / wpt;
  P.s.nz = 1;
  P.s.arow_step = gpt * no;
  P.s.brow_step = wpt * 2 * no;
  P.s.err = f64_err(L, work);
  P.s.epi_bytes = (int)exch_stage_bytes<T>(extra);
  ProfScope ps(K_EXCH, st);
  return f64_launch<T>(P, sm_count(), st);
}

}  // namespace

cudaError_t launch_fb_gemm(const Layout& L, const double* prep, double* work, cudaStream_t st) {
  const int M = 2 * L.W, N = L.G;
  const long long K = L.Kfb_used;
  int kchunk = (int)((K + L.splitk - 1) / L.splitk);
  kchunk = (kchunk + 15) / 16 * 16;
  const int ks = (int)((K + kchunk - 1) / kchunk);
  double* part = work + L.w_fbpart;
  const long long zs = 2LL * L.W * L.Gpad;
  for (int z = ks; z < L.splitk; ++z) {  // splits without work: their partial sums are zero
    cudaError_t e = cudaMemsetAsync(part + z * zs, 0, zs * sizeof(double), st);
    if (e != cudaSuccess) return e;
  }
  return with_gemm_tile<F64_B_K>(M, N, ks, [&](auto tile) {
    using T = decltype(tile);
    F64Params<FbEpi> P{};
    if (make_tmap_f64(&P.ta, work + L.w_gpl, K, M, 1, L.Kfb, L.Kfb * M, 8, T::BM) != AFQ_OK ||
        make_tmap_f64(&P.tb, prep + L.p_rccat, K, N, 1, L.Kfb, L.Kfb * N, 8, T::BN) != AFQ_OK)
      return cudaErrorInvalidValue;
    P.s.K = (int)K;
    P.s.mt = (M + T::BM - 1) / T::BM;
    P.s.nt = (N + T::BN - 1) / T::BN;
    P.s.nz = ks;
    P.s.arow_step = T::BM;
    P.s.brow_step = T::BN;
    P.s.ksplit = kchunk;
    P.s.err = f64_err(L, work);
    P.epi = FbEpi{part, L.Gpad, zs, M, N};
    ProfScope ps(K_FB, st);
    return f64_launch<T>(P, sm_count(), st);
  });
}

cudaError_t launch_prep_grouped(const PrepArgs* args, const BlockMap& m, int step, cudaStream_t st) {
  ProfScope ps(K_PREP, st);
  prep_kernel_grouped<<<m.start[m.n], 256, 0, st>>>(args, m, step);
  return cudaGetLastError();
}

cudaError_t launch_prep(const Layout& L, const double* prep, double* work, const double* fields,
                        double dt, double* fb_out, cudaStream_t st) {
  ProfScope ps(K_PREP, st);
  bf16* xb[3] = {nullptr, nullptr, nullptr};
  if (L.mixed) piece_ptrs(work, L.v_xt, L.v_xt_ps, L.npc, xb);
  prep_kernel<<<L.W, 256, 0, st>>>(L.W, L.G, L.Gpad, L.splitk, work + L.w_fbpart, L.mixed ? 1 : 0,
                                   (double)L.mult, fields, prep + L.p_mf, sqrt(dt),
                                   L.mixed ? nullptr : work + L.w_xt, work + L.w_wscal, fb_out, L.npc, xb[0], xb[1],
                                   xb[2], L.Gb);
  return cudaGetLastError();
}

// Free propagation (propagation.py:338-376): VHS = i sqrt(dt) x L from the raw
// fields x, rows (w, 0) = Re = 0 and (w, 1) = Im = sqrt(dt) x of the VHS operand
__global__ void __launch_bounds__(256) free_fields_kernel(int G, long long Gpad, const double* fields,
                                                          double sdt, double* xt, int npc, bf16* xb0,
                                                          bf16* xb1, bf16* xb2, long long ldxb) {
  bf16* const xb[3] = {xb0, xb1, xb2};
  const int w = blockIdx.x;
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    const double x = fields[(long long)w * G + g];
    if (xb0) {
      put_pieces(0.0, npc, xb, (2LL * w) * ldxb + g);
      put_pieces(sdt * x, npc, xb, (2LL * w + 1) * ldxb + g);
    } else {
      xt[(2LL * w) * Gpad + g] = 0.0;
      xt[(2LL * w + 1) * Gpad + g] = sdt * x;
    }
  }
}

cudaError_t launch_free_fields(const Layout& L, double* work, const double* fields, double dt,
                               cudaStream_t st) {
  ProfScope ps(K_PREP, st);
  bf16* xb[3] = {nullptr, nullptr, nullptr};
  if (L.mixed) piece_ptrs(work, L.v_xt, L.v_xt_ps, L.npc, xb);
  free_fields_kernel<<<L.W, 256, 0, st>>>(L.G, L.Gpad, fields, sqrt(dt), L.mixed ? nullptr : work + L.w_xt, L.npc, xb[0],
                                          xb[1], xb[2], L.Gb);
  return cudaGetLastError();
}

cudaError_t launch_vhs_gemm(const Layout& L, const double* prep, double* work, cudaStream_t st) {
  const int M = 2 * L.W, NN = L.N * L.N, K = L.G;
  return with_gemm_tile<F64_B_N>(M, NN, 1, [&](auto tile) {
    using T = decltype(tile);
    F64Params<VhsEpi> P{};
    if (make_tmap_f64(&P.ta, work + L.w_xt, K, M, 1, L.Gpad, L.Gpad * M, 8, T::BM) != AFQ_OK ||
        make_tmap_f64(&P.tb, prep + L.p_chol, NN, K, 1, L.N2pad, L.N2pad * K, 16, 16) != AFQ_OK)
      return cudaErrorInvalidValue;
    P.s.K = K;
    P.s.mt = (M + T::BM - 1) / T::BM;
    P.s.nt = (NN + T::BN - 1) / T::BN;
    P.s.nz = 1;
    P.s.arow_step = T::BM;
    P.s.err = f64_err(L, work);
    P.epi = VhsEpi{work + L.w_vhs, M, NN, L.N, L.Npad};
    ProfScope ps(K_VHS, st);
    return f64_launch<T>(P, sm_count(), st);
  });
}

cudaError_t launch_propagate_walkers(const Layout& L, const double* prep, double* work,
                                     double* const walkers[2], int n_exp_terms,
                                     cudaStream_t st) {
  const int N = L.N;
  const long long vld = 2 * L.Npad;
  const double* vr = work + L.w_vhs;
  const double* vi = vr + L.Npad;
  for (int s = 0; s < L.np; ++s) {
    const int nc = 2 * L.no[s];
    double* wk = walkers[s];
    double* y = work + L.w_y;
    const double* e1 = prep + L.p_exph1[s];
    // y = e^{-dt h/2} w
    cudaError_t err = prop_gemm<F64_REAL>(L, work, nc, {e1, nullptr, L.Npad, 0, wk, y, nullptr, 1.0}, st);
    if (err != cudaSuccess) return err;
    // z_{n-1} = y + VHS z_n / n for n = T .. 1 (T = n_exp_terms - 1), z_T = y
    const double* src = y;
    double* bufs[2] = {work + L.w_ta, work + L.w_tb};
    for (int n = n_exp_terms - 1; n >= 1; --n) {
      double* dst = bufs[n & 1];
      err = prop_gemm<F64_COMPLEX>(L, work, nc, {vr, vi, vld, (long long)N * vld, src, dst, y, 1.0 / n}, st);
      if (err != cudaSuccess) return err;
      src = dst;
    }
    // w' = e^{-dt h/2} z_0
    err = prop_gemm<F64_REAL>(L, work, nc, {e1, nullptr, L.Npad, 0, src, wk, nullptr, 1.0}, st);
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

cudaError_t launch_exchange(const Layout& L, const double* prep, double* work, int s,
                            cudaStream_t st) {
  const int no = L.no[s], gpt = L.ex[s].gpt;
  int wpt;
  return with_exch_tile(no, L.G, L.W, wpt, [&](auto tile) {
    using T = decltype(tile);
    F64Params<ExchEpi> P{};
    P.epi = ExchEpi{L.G, no, L.W, gpt, wpt, work + L.w_c[s], work + L.w_exc[s]};
    return exch_run<T>(L, prep, work, s, P, wpt, 4 * (gpt * wpt + T::CW), st);
  });
}

cudaError_t launch_orbenergy(const Layout& L, const double* prep, double* work, const double* prj,
                             int nlo, double* out, cudaStream_t st) {
  if (nlo < 1 || nlo > kMaxLo || L.no[0] > 64) return cudaErrorInvalidValue;
  {
    ProfScope ps(K_MISC, st);
    theta_zero_occ_kernel<<<256, 256, 0, st>>>(work + L.w_theta[0], (long long)L.W * 2 * L.no[0], L.Npad, L.no[0]);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int no = L.no[0], gpt = L.ex[0].gpt;
  int wpt;
  e = with_exch_tile(no, L.G, L.W, wpt, [&](auto tile) {
    using T = decltype(tile);
    F64Params<OrbEpi> P{};
    P.epi = OrbEpi{L.G, no, L.W, gpt, wpt, nlo, prj, work + L.w_orb};
    return exch_run<T>(L, prep, work, 0, P, wpt, kMaxLo * 64 + 2 * gpt * wpt, st);
  });
  if (e != cudaSuccess) return e;
  const int wpb = 8;
  const int mt = (L.G + gpt - 1) / gpt;
  ProfScope ps(K_ECOMB, st);
  orb_combine_kernel<<<(L.W + wpb - 1) / wpb, 32 * wpb, 0, st>>>(L.W, mt, work + L.w_orb, out);
  return cudaGetLastError();
}

cudaError_t launch_energy_combine(const Layout& L, const double* prep, double* work, double* eout,
                                  int eout_stride, cudaStream_t st) {
  const int wpb = 8;
  ProfScope ps(K_ECOMB, st);
  energy_combine_kernel<<<(L.W + wpb - 1) / wpb, 32 * wpb, 0, st>>>(
      L.W, L.G, L.ns, L.restricted, prep + L.p_scal, work + L.w_c[0], L.ns == 2 ? work + L.w_c[1] : nullptr,
      work + L.w_exc[0], L.ex[0].mt, L.ns == 2 ? work + L.w_exc[1] : nullptr,
      L.ns == 2 ? L.ex[1].mt : 0, work + L.w_wscal, eout, eout_stride);
  return cudaGetLastError();
}

}  // namespace afq
