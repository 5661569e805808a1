// The FP64 phaseless step of small systems in one kernel (propagation.py:274-336).
//
// At N = 10, No = 5, G = 50 a step's arithmetic is a few microseconds of one SM
// per walker, but as separate launches (Green's function, force bias, field preparation, VHS,
// seven propagator products, overlaps) it is 14 of them at 2.5-20 us each, all
// latency.  Here one CTA carries one walker through the whole step in shared
// memory; only the weight update, which needs every walker's overlap, is a second
// launch.  Every operand a walker needs (chol, rot_chol) is read from L2 once per
// walker, so the rule below bounds that: beyond it the tensor-core launches, which
// share the reads among walkers, are faster.
// Measured (B200, recorded steps): see small_step_fits.
#include "common.cuh"
#include "gauss_jordan.cuh"
#include "ops.h"
#include "profile.cuh"

namespace afq {

int sm_count();

namespace {

constexpr int kSmallThreads = 256;

struct SmallArgs {
  int N, G, W, ns, mult, n_exp, have_green;
  int no[2], koff[2];
  const double* mo[2];
  const double* exph1[2];
  const double* rccat;
  const double* chol;
  const double* mf;
  const double* fields;
  double* walk[2];
  double* gpl;
  double* wscal;
  long long npad, n2pad, kfb;
  int kused;
  double sdt;
};

// shared memory in doubles: two walker buffers and the Horner term y (complex,
// both sectors), Green's function (planar), S, VHS, exp_h1, fields, partial sums
struct SmallSmem {
  long long w0, w1, y, gre, gim, s, colk, vhs, e, xr, xi, part, total;
};
__host__ __device__ inline SmallSmem small_smem(int N, int G, int no0, int no1, int ns) {
  SmallSmem m;
  long long o = 0;
  auto take = [&](long long n) {
    const long long r = o;
    o += (n + 1) & ~1LL;
    return r;
  };
  const long long k = (long long)N * (no0 + (ns == 2 ? no1 : 0));
  const int nm = no0 > no1 ? no0 : no1;
  m.w0 = take(2 * k);
  m.w1 = take(2 * k);
  m.y = take(2 * k);
  m.gre = take(k);
  m.gim = take(k);
  m.s = take(2LL * nm * nm);
  m.colk = take(128);
  m.vhs = take(2LL * N * N);
  m.e = take((long long)ns * N * N);
  m.xr = take(G);
  m.xi = take(G);
  m.part = take(2LL * kSmallThreads);
  m.total = o;
  return m;
}

// Theta^T of the walkers in `w` into gre/gim (rows (sector, i), N long) and the
// determinants, returned by thread 0
__device__ void small_green(const SmallArgs& a, const double2* w, double2* S, double2* colk, double* gre,
                            double* gim, int* perm, double2* ipk, double2 (&det)[2]) {
  const int N = a.N, tid = threadIdx.x;
  long long off = 0;
  for (int s = 0; s < a.ns; ++s) {
    const int no = a.no[s];
    const double2* W = w + off;
    for (int e = tid; e < no * no; e += kSmallThreads) {
      const int i = e / no, j = e - i * no;
      double2 v = make_double2(0.0, 0.0);
      for (int p = 0; p < N; ++p) {
        const double c = a.mo[s][p * no + i];
        const double2 x = W[p * no + j];
        v.x = fma(c, x.x, v.x);
        v.y = fma(c, x.y, v.y);
      }
      S[e] = v;
    }
    __syncthreads();
    det[s] = gauss_jordan_cta<kSmallThreads>(S, colk, perm, ipk, no);
    for (int e = tid; e < N * no; e += kSmallThreads) {
      const int i = e / N, p = e - i * N;
      double2 v = make_double2(0.0, 0.0);
      for (int j = 0; j < no; ++j) v = cadd(v, cmul(W[p * no + j], S[j * no + i]));
      gre[a.koff[s] + e] = v.x;
      gim[a.koff[s] + e] = v.y;
    }
    __syncthreads();
    off += (long long)N * no;
  }
}

__global__ void __launch_bounds__(kSmallThreads) small_step_kernel(const SmallArgs a) {
  extern __shared__ double sm[];
  __shared__ double red[4 * (kSmallThreads / 32)];
  __shared__ int perm[64];
  __shared__ double2 ipk;
  const int N = a.N, G = a.G, w = blockIdx.x, tid = threadIdx.x, NN = N * N;
  const SmallSmem m = small_smem(N, G, a.no[0], a.no[1], a.ns);
  double2* w0 = reinterpret_cast<double2*>(sm + m.w0);
  double2* w1 = reinterpret_cast<double2*>(sm + m.w1);
  double2* y = reinterpret_cast<double2*>(sm + m.y);
  double* gre = sm + m.gre;
  double* gim = sm + m.gim;
  double2* S = reinterpret_cast<double2*>(sm + m.s);
  double2* colk = reinterpret_cast<double2*>(sm + m.colk);
  double2* V = reinterpret_cast<double2*>(sm + m.vhs);
  double* E = sm + m.e;
  double* xr = sm + m.xr;
  double* xi = sm + m.xi;
  double2* part = reinterpret_cast<double2*>(sm + m.part);
  const int n0 = N * a.no[0], nt = n0 + (a.ns == 2 ? N * a.no[1] : 0);  // complex elements of the walker

  for (int e = tid; e < nt; e += kSmallThreads)
    w0[e] = e < n0 ? reinterpret_cast<const double2*>(a.walk[0])[(long long)w * n0 + e]
                   : reinterpret_cast<const double2*>(a.walk[1])[(long long)w * (nt - n0) + e - n0];
  for (int e = tid; e < a.ns * NN; e += kSmallThreads) {
    const int s = e / NN, r = (e - s * NN) / N, c = e - s * NN - r * N;
    E[e] = a.exph1[s][r * a.npad + c];
  }
  double* const Gre = a.gpl + (2LL * w) * a.kfb;
  double* const Gim = Gre + a.kfb;
  double2 det[2] = {make_double2(1.0, 0.0), make_double2(1.0, 0.0)};
  __syncthreads();
  if (a.have_green) {  // left by the previous step
    for (int e = tid; e < a.kused; e += kSmallThreads) {
      gre[e] = Gre[e];
      gim[e] = Gim[e];
    }
    __syncthreads();
  } else {
    small_green(a, w0, S, colk, gre, gim, perm, &ipk, det);
  }

  // ---- force bias, shifted fields: eight lanes per Cholesky vector ----------
  double sr = 0, si = 0, br = 0, bi = 0;
  for (int gb = 0; gb < G; gb += kSmallThreads / 8) {
    const int g = gb + (tid >> 3), l = tid & 7;
    double fr = 0.0, fi = 0.0;
    if (g < G) {
      const double* rc = a.rccat + g * a.kfb;
#pragma unroll 4
      for (int k = l; k < a.kused; k += 8) {
        const double c = rc[k];
        fr = fma(c, gre[k], fr);
        fi = fma(c, gim[k], fi);
      }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      fr += __shfl_down_sync(0xffffffffu, fr, o);
      fi += __shfl_down_sync(0xffffffffu, fi, o);
    }
    if (l == 0 && g < G) {
      fr *= a.mult;
      fi *= a.mult;
      const double mfr = a.mf[2 * g], mfi = a.mf[2 * g + 1];
      // field_shifts = -sqrt(dt) * (i*fb - mf_shifts)
      const double fsr = -a.sdt * (-fi - mfr), fsi = -a.sdt * (fr - mfi);
      const double x = a.fields[(long long)w * G + g];
      const double tr = x - fsr, ti = -fsi;  // shifted field
      sr += tr * mfr - ti * mfi;
      si += tr * mfi + ti * mfr;
      br += x * fsr - (fsr * fsr - fsi * fsi) / 2.0;
      bi += x * fsi - (2.0 * fsr * fsi) / 2.0;
      xr[g] = -a.sdt * ti;
      xi[g] = a.sdt * tr;
    }
  }
  sr = warp_sum(sr);
  si = warp_sum(si);
  br = warp_sum(br);
  bi = warp_sum(bi);
  if ((tid & 31) == 0) {
    double* r = red + 4 * (tid >> 5);
    r[0] = sr;
    r[1] = si;
    r[2] = br;
    r[3] = bi;
  }
  __syncthreads();
  if (tid < 4) {
    double s = 0.0;
    for (int q = 0; q < kSmallThreads / 32; ++q) s += red[4 * q + tid];
    a.wscal[(long long)w * 16 + tid] = s;
  }

  // ---- VHS = sum_g x_g L_g; small N: the Cholesky index split over the threads
  const int parts = NN < kSmallThreads ? kSmallThreads / NN : 1;
  if (parts > 1) {
    const int q = tid / NN, e = tid - q * NN;
    double vr = 0.0, vi = 0.0;
    if (q < parts) {
#pragma unroll 4
      for (int g = q; g < G; g += parts) {
        const double c = a.chol[g * a.n2pad + e];
        vr = fma(c, xr[g], vr);
        vi = fma(c, xi[g], vi);
      }
      part[tid] = make_double2(vr, vi);
    }
    __syncthreads();
    if (tid < NN) {
      double2 v = part[tid];
      for (int k = 1; k < parts; ++k) v = cadd(v, part[k * NN + tid]);
      V[tid] = v;
    }
  } else {
    for (int e = tid; e < NN; e += kSmallThreads) {
      double vr = 0.0, vi = 0.0;
#pragma unroll 8
      for (int g = 0; g < G; ++g) {
        const double c = a.chol[g * a.n2pad + e];
        vr = fma(c, xr[g], vr);
        vi = fma(c, xi[g], vi);
      }
      V[e] = make_double2(vr, vi);
    }
  }

  // ---- y = e^{-dt h/2} w; Horner; w' = e^{-dt h/2} z_0 -----------------------
  auto one_body = [&](const double2* src, double2* dst) {
    for (int e = tid; e < nt; e += kSmallThreads) {
      const int s = e >= n0, r = s ? e - n0 : e, no = a.no[s];
      const int p = r / no, j = r - p * no;
      const double* er = E + s * NN + p * N;
      const double2* x = src + (s ? n0 : 0) + j;
      double2 v = make_double2(0.0, 0.0);
#pragma unroll 4
      for (int k = 0; k < N; ++k) {
        v.x = fma(er[k], x[k * no].x, v.x);
        v.y = fma(er[k], x[k * no].y, v.y);
      }
      dst[e] = v;
    }
  };
  one_body(w0, y);
  __syncthreads();
  const double2* src = y;
  for (int n = a.n_exp - 1; n >= 1; --n) {
    double2* dst = (n & 1) ? w1 : w0;
    const double sc = 1.0 / n;
    for (int e = tid; e < nt; e += kSmallThreads) {
      const int s = e >= n0, r = s ? e - n0 : e, no = a.no[s];
      const int p = r / no, j = r - p * no;
      const double2* vr = V + p * N;
      const double2* x = src + (s ? n0 : 0) + j;
      double2 u = make_double2(0.0, 0.0), t = make_double2(0.0, 0.0);
#pragma unroll 4
      for (int k = 0; k < N; ++k) {
        const double2 c = vr[k], z = x[k * no];
        u.x = fma(c.x, z.x, u.x);
        u.y = fma(c.x, z.y, u.y);
        t.x = fma(c.y, z.y, t.x);
        t.y = fma(c.y, z.x, t.y);
      }
      const double2 y0 = y[e];
      dst[e] = make_double2(y0.x + sc * (u.x - t.x), y0.y + sc * (u.y + t.y));
    }
    __syncthreads();
    src = dst;
  }
  double2* fin = src == w1 ? w0 : w1;  // neither y nor the source
  one_body(src, fin);
  __syncthreads();
  for (int e = tid; e < nt; e += kSmallThreads) {
    if (e < n0)
      reinterpret_cast<double2*>(a.walk[0])[(long long)w * n0 + e] = fin[e];
    else
      reinterpret_cast<double2*>(a.walk[1])[(long long)w * (nt - n0) + e - n0] = fin[e];
  }

  // ---- new overlap and Green's function (the next step's force bias) --------
  small_green(a, fin, S, colk, gre, gim, perm, &ipk, det);
  for (int e = tid; e < a.kused; e += kSmallThreads) {
    Gre[e] = gre[e];
    Gim[e] = gim[e];
  }
  if (tid == 0) {
    const double2 o = a.ns == 2 ? cmul(det[0], det[1]) : (a.mult == 2 ? cmul(det[0], det[0]) : det[0]);
    double* s = a.wscal + (long long)w * 16;
    s[4] = det[0].x;
    s[5] = det[0].y;
    if (a.ns == 2) {
      s[6] = det[1].x;
      s[7] = det[1].y;
    }
    s[12] = o.x;
    s[13] = o.y;
  }
}

}  // namespace

// Where this kernel is the faster one.  Per walker it takes
//   5.1e-4 G N (N + 1.7 No) + No (4e-3 N No + 2) - 19 ns  (No: a sum over spins; 19 per spin)
// more than the tensor-core launches, a fit to both at N = 4 to 24, No = 1 to N, G = 2 N to 16 N and
// 20 to 10000 walkers (recorded steps); the launches cost some 18 us more whatever the
// walkers, and below one walker per SM a walker's own time counts.  With this rule no size of
// that range is slower than the launches it replaced, and the sizes together are within
// 0.5 % of always taking the faster one.  Recorded steps, us, this kernel / the launches: N = 6, No = 1,
// G = 12, 296 walkers 19 / 52, 10000 345 / 620; N = 20, No = 10, G = 160, 296 walkers 55 / 71, 10000
// 1.47 times the launches; N = 16, No = 16, G = 256, 4000 walkers 945 / 449; N = 24, No = 24,
// G = 384, 20 walkers 153 / 76.  (All of N <= 20 took this kernel before: N = 16, No = 16, G = 256,
// 4000 walkers 945 us, 513 before it existed.)
bool small_step_fits(const Layout& L) {
  if (L.mixed || L.N > 24) return false;
  double ns = 0.0;
  int no = 0;
  for (int s = 0; s < L.ns; ++s) {
    no += L.no[s];
    ns += L.no[s] * (4e-3 * L.N * L.no[s] + 2.0) - 19.0;
  }
  ns += 5.1e-4 * L.G * L.N * (L.N + 1.7 * no);
  const int w = L.W > sm_count() ? L.W : sm_count();
  if (ns * w >= 18000.0) return false;
  return small_smem(L.N, L.G, L.no[0], L.no[1], L.ns).total * sizeof(double) <= 200 * 1024;
}

cudaError_t launch_small_step(const Layout& L, const double* prep, double* work, double* const walkers[2],
                              const double* fields, double dt, int n_exp_terms, bool have_green,
                              cudaStream_t st) {
  SmallArgs a{};
  a.N = L.N;
  a.G = L.G;
  a.W = L.W;
  a.ns = L.ns;
  a.mult = L.mult;
  a.n_exp = n_exp_terms;
  a.have_green = have_green;
  for (int s = 0; s < L.ns; ++s) {
    a.no[s] = L.no[s];
    a.koff[s] = (int)L.koff[s];
    a.mo[s] = prep + L.p_mo[L.uhf_trial ? s : 0];
    a.exph1[s] = prep + L.p_exph1[s];
    a.walk[s] = walkers[s];
  }
  a.rccat = prep + L.p_rccat;
  a.chol = prep + L.p_chol;
  a.mf = prep + L.p_mf;
  a.fields = fields;
  a.gpl = work + L.w_gpl;
  a.wscal = work + L.w_wscal;
  a.npad = L.Npad;
  a.n2pad = L.N2pad;
  a.kfb = L.Kfb;
  a.kused = (int)L.Kfb_used;
  a.sdt = sqrt(dt);
  const size_t smem = small_smem(L.N, L.G, L.no[0], L.no[1], L.ns).total * sizeof(double);
  cudaError_t e = allow_smem(small_step_kernel, smem);
  if (e != cudaSuccess) return e;
  ProfScope ps(K_PROP, st);  // the whole step is counted as the propagator
  small_step_kernel<<<L.W, kSmallThreads, smem, st>>>(a);
  return cudaGetLastError();
}

}  // namespace afq
