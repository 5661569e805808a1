// Block-wide Gauss-Jordan inverse of a small complex matrix in shared memory.
#pragma once

#include "common.cuh"

namespace afq {

// Gauss-Jordan inverse with partial pivoting of the No x No complex S in
// shared memory, in place, by the whole CTA (T threads); returns det S in
// thread 0.
template <int T>
__device__ double2 gauss_jordan_cta(double2* S, double2* colk, int* perm, double2* ipk_s, int no) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int Q = (4096 + T - 1) / T;  // elements of a 64 x 64 S per thread
  const int npairs = no * no;
  // Each elimination step: warp 0 alone finds the pivot (first max of
  // |re|+|im| in column k, as LAPACK izamax), swaps it into row k, keeps
  // column k and scales row k by 1/p (= conj(p)/|p|^2); then every thread
  // updates its fixed elements.  Two block barriers per step.
  int my_i[Q], my_j[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int e = tid + q * T;
    my_i[q] = e < npairs ? e / no : -1;
    my_j[q] = e < npairs ? e - (e / no) * no : 0;
  }
  double2 det = make_double2(1.0, 0.0);
  for (int k = 0; k < no; ++k) {
    if (warp == 0) {
      double best = -1.0;
      int bi = k;
      for (int r = k + lane; r < no; r += 32) {
        const double2 v = S[r * no + k];
        const double m = fabs(v.x) + fabs(v.y);
        if (m > best) { best = m; bi = r; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      const int pv = bi;
      if (pv != k)
        for (int j = lane; j < no; j += 32) {
          const double2 t0 = S[k * no + j];
          S[k * no + j] = S[pv * no + j];
          S[pv * no + j] = t0;
        }
      __syncwarp();
      const double2 pk = S[k * no + k];
      const double inv = 1.0 / (pk.x * pk.x + pk.y * pk.y);
      const double2 ipk = make_double2(pk.x * inv, -pk.y * inv);
      for (int i = lane; i < no; i += 32) colk[i] = S[i * no + k];
      __syncwarp();
      for (int j = lane; j < no; j += 32) S[k * no + j] = (j == k) ? ipk : cmul(S[k * no + j], ipk);
      if (lane == 0) {
        perm[k] = pv;
        *ipk_s = ipk;
        det = cmul(det, pk);
        if (pv != k) det = make_double2(-det.x, -det.y);
      }
    }
    __syncthreads();
    const double2 ipk = *ipk_s;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int i = my_i[q], j = my_j[q];
      if (i < 0 || i == k) continue;
      const double2 f = colk[i];
      if (j == k) {
        const double2 t0 = cmul(f, ipk);
        S[i * no + j] = make_double2(-t0.x, -t0.y);
      } else {
        S[i * no + j] = csub(S[i * no + j], cmul(f, S[k * no + j]));
      }
    }
    __syncthreads();
  }
  // undo the row interchanges as column interchanges, last first (rows independent)
  for (int i = tid; i < no; i += T)
    for (int k = no - 1; k >= 0; --k) {
      const int pv = perm[k];
      if (pv != k) {
        const double2 t0 = S[i * no + k];
        S[i * no + k] = S[i * no + pv];
        S[i * no + pv] = t0;
      }
    }
  __syncthreads();
  return det;
}

}  // namespace afq
