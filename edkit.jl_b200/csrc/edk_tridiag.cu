// edk_tridiag.cu — the lowest eigenvalues of many symmetric tridiagonal
// matrices on the device: the convergence checks of the batched Lanczos
// (eigen(SymTridiagonal(α, β)), src/algorithms/TimeEvolution.jl:311-323) and
// the candidates of the block Lanczos's eigenvalue step.
//
// Bound by the serial chain of a Sturm count (one dependent FMA per row of
// T), so the chain is what the layout shortens: a block owns one matrix, its
// threads are split into groups, one group per wanted eigenvalue, and every
// thread of a group counts at its own shift, so one pass over T narrows the
// group's interval by the group's size + 1 (256 threads on one eigenvalue: 8
// bits a pass, seven passes from Gershgorin's interval to the last bit).  The
// count is the number of sign changes of p_i = (a_i - x) p_{i-1} -
// b_{i-1}^2 p_{i-2} (the leading minors), which needs no division; p is
// rescaled by a power of two every eight rows.  T is scaled to entries below
// one and an off-diagonal below eps is taken as eps (a change of T within its
// rounding), so p can neither vanish nor leave the range in eight rows.
//
// The host solved the same problems before, one after another, with QL sweeps
// over whole spectra while the GPU waited: 4.5 ms a check for 96 matrices of
// order 10 .. 130, 4.3 ms for 18 of order 10 .. 960.  Here: 21 us and 64 us,
// between two steps of the solver's own stream.
#include <algorithm>
#include <cmath>
#include <vector>

#include "edk_internal.cuh"

namespace edk {

namespace {

constexpr int kTriThreads = 256;
constexpr int kTriStage = 1024;  // rows of T held in shared memory at a time
constexpr int kTriGroups = 8;    // eigenvalues searched at once, at most

// p_{i-1}, p_i scaled by the power of two that brings the larger into [1, 2)
__device__ __forceinline__ void tri_rescale(double& p0, double& p1) {
  const int e0 = (__double2hiint(p0) >> 20) & 0x7ff, e1 = (__double2hiint(p1) >> 20) & 0x7ff;
  const int e = min(max(max(e0, e1), 1), 2045);
  const double s = __hiloint2double((2046 - e) << 20, 0);
  p0 *= s;
  p1 *= s;
}

// Lowest eigenvalues 0 .. nk-1 of T_q (diagonal alpha + q ld, off-diagonal
// beta + q ld, order nsteps[q], or nfix[q] if positive, or nall), ascending, into
// ev + q nk; NaN past the order.  Blocks along y share a matrix's eigenvalues.
// With CHECK: matrices whose done[q] is set are left alone, the new values
// are compared with the ones the previous check left in ev (seen[q] says there
// are some), done[q] becomes 1 when all nk moved by at most tol max(1, |x|),
// and *left counts the matrices still running.
template <bool CHECK>
__global__ void __launch_bounds__(kTriThreads) k_tri_lowest(
    const double* __restrict__ alpha, const double* __restrict__ beta, int64_t ld,
    const int* __restrict__ nsteps, const int* __restrict__ nfix, int nall, int nk, int groups,
    double* __restrict__ ev, double tol, int* __restrict__ seen, int* __restrict__ done,
    int* __restrict__ left) {
  __shared__ double s_a[kTriStage], s_b[kTriStage];
  __shared__ double s_lo[kTriGroups], s_hi[kTriGroups], s_red[2][kTriThreads / 32];
  __shared__ int s_nle[kTriGroups], s_conv, s_open;
  const int q = blockIdx.x, tid = threadIdx.x;
  if (CHECK && done[q]) return;
  const int n = nsteps ? nsteps[q] : (nfix && nfix[q] > 0 ? nfix[q] : nall);
  if (CHECK && n < nk) {
    if (tid == 0) atomicAdd(left, 1);
    return;
  }
  const double* a = alpha + (int64_t)q * ld;
  const double* b = beta + (int64_t)q * ld;
  // Gershgorin interval
  double lo = INFINITY, hi = -INFINITY;
  for (int i = tid; i < n; i += kTriThreads) {
    const double r = (i > 0 ? fabs(b[i - 1]) : 0.0) + (i + 1 < n ? fabs(b[i]) : 0.0);
    lo = fmin(lo, a[i] - r);
    hi = fmax(hi, a[i] + r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((tid & 31) == 0) {
    s_red[0][tid >> 5] = lo;
    s_red[1][tid >> 5] = hi;
  }
  if (tid == 0) s_conv = 1;
  __syncthreads();
  for (int w = 0; w < kTriThreads / 32; ++w) {
    lo = fmin(lo, s_red[0][w]);
    hi = fmax(hi, s_red[1][w]);
  }
  const double norm = fmax(fabs(lo), fabs(hi));
  // a power of two: scaling is exact.  A zero or non-finite T is not searched.
  const bool ok = n > 0 && norm > 1e-290 && norm < 1e290;
  const double up = ok ? scalbn(1.0, ilogb(norm) + 1) : 1.0, dn = 1.0 / up;
  const double wide = 4.0 * 2.220446049250313e-16;
  lo = lo * dn - wide;
  hi = hi * dn + wide;
  auto stage = [&](int c0) {
    const int c1 = min(n, c0 + kTriStage);
    for (int i = c0 + tid; i < c1; i += kTriThreads) {
      s_a[i - c0] = a[i] * dn;
      const double o = i > 0 ? fmax(fabs(b[i - 1] * dn), 0x1p-53) : 0.0;
      s_b[i - c0] = o * o;  // couples row i to row i - 1
    }
  };
  const bool whole = n <= kTriStage;
  if (ok && whole) {
    stage(0);
    __syncthreads();
  }
  const int G = kTriThreads / groups, g = tid / G, t = tid % G;
  const double step = 1.0 / (G + 1);
  for (int k0 = blockIdx.y * groups; k0 < nk; k0 += groups * gridDim.y) {
    const int k = k0 + g;
    const bool mine = ok && k < nk && k < n;
    if (t == 0) {
      s_lo[g] = lo;
      s_hi[g] = hi;
    }
    __syncthreads();
    for (int round = 0; ok && round < 64; ++round) {
      if (t == 0) s_nle[g] = 0;
      if (tid == 0) s_open = 0;
      __syncthreads();
      const double l = s_lo[g], h = s_hi[g];
      const double x = fma(h - l, (t + 1) * step, l);
      // sign changes of the leading minors = eigenvalues below x
      double p0 = 0.0, p1 = 1.0;
      int neg = 0;
      for (int c0 = 0; c0 < n; c0 += kTriStage) {
        if (!whole) {
          __syncthreads();
          stage(c0);
          __syncthreads();
        }
        const int cn = min(n - c0, kTriStage);
        int i = 0;
        for (; i + 8 <= cn; i += 8) {
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const double p2 = fma(s_a[i + u] - x, p1, -(s_b[i + u] * p0));
            neg += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
            p0 = p1;
            p1 = p2;
          }
          tri_rescale(p0, p1);
        }
        for (; i < cn; ++i) {
          const double p2 = fma(s_a[i] - x, p1, -(s_b[i] * p0));
          neg += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
          p0 = p1;
          p1 = p2;
        }
        tri_rescale(p0, p1);
      }
      if (mine && neg <= k) atomicAdd(&s_nle[g], 1);
      __syncthreads();
      if (t == 0 && mine) {
        const int c = s_nle[g];  // shifts at or below eigenvalue k
        const double nl = c > 0 ? fma(h - l, c * step, l) : l;
        const double nh = c < G ? fma(h - l, (c + 1) * step, l) : h;
        s_lo[g] = nl;
        s_hi[g] = nh;
        // down to the spacing of the entries of T (its rounding)
        if (nh - nl > 0x1p-54 && (nl > l || nh < h)) s_open = 1;
      }
      __syncthreads();
      if (!s_open) break;
      __syncthreads();  // s_open is read before the next round clears it
    }
    if (t == 0 && k < nk) {
      double w = NAN;
      if (mine) w = 0.5 * (s_lo[g] + s_hi[g]) * up;
      else if (n > k && norm <= 1e-290) w = 0.0;
      double* e = ev + (int64_t)q * nk + k;
      if (CHECK && !(fabs(w - *e) <= tol * fmax(1.0, fabs(w)))) s_conv = 0;
      *e = w;
    }
    __syncthreads();
  }
  if (CHECK && tid == 0) {
    const bool conv = seen[q] && s_conv;
    seen[q] = 1;
    if (conv) done[q] = 1;
    else atomicAdd(left, 1);
  }
}

// groups of threads per block: a power of two, one per eigenvalue up to eight
int tri_groups(int nk) {
  int g = 1;
  while (g < nk && g < kTriGroups) g *= 2;
  return g;
}

}  // namespace

edk_status tridiag_check_device(int nops, const double* alpha, const double* beta, int64_t ld,
                                const int* nsteps, int nk, double* ev, double tol, int* seen,
                                int* done, int* left, cudaStream_t st) {
  EDK_TRY_CUDA(cudaMemsetAsync(left, 0, sizeof(int), st));
  k_tri_lowest<true><<<nops, kTriThreads, 0, st>>>(alpha, beta, ld, nsteps, nullptr, 0, nk,
                                                   tri_groups(nk), ev, tol, seen, done, left);
  EDK_TRY_CUDA(cudaGetLastError());
  return EDK_OK;
}

edk_status tridiag_lowest_device(int nops, const double* alpha, const double* beta, int64_t ld,
                                 const int* nsteps, const int* nfix, int nall, int nk, double* ev,
                                 cudaStream_t st) {
  const int groups = tri_groups(nk);
  const dim3 grid((unsigned)nops, (unsigned)std::min(65535, (nk + groups - 1) / groups));
  k_tri_lowest<false><<<grid, kTriThreads, 0, st>>>(alpha, beta, ld, nsteps, nfix, nall, nk, groups,
                                                    ev, 0.0, nullptr, nullptr, nullptr);
  EDK_TRY_CUDA(cudaGetLastError());
  return EDK_OK;
}

// The eigenvectors of one tridiagonal matrix (order m, on the host) for nk
// ascending eigenvalues w, by inverse iteration: Q column-major m x nk, unit
// length, first component not negative.  Vectors whose eigenvalues lie within
// 1e-3 |T| of each other are kept orthogonal.  O(m nk) instead of the O(m^3)
// of a QL sweep with vectors.
void tridiag_vectors(int m, const double* a, const double* b, int nk, const double* w, double* Q) {
  double norm = 0.0;
  for (int i = 0; i < m; ++i)
    norm = std::max(norm, std::fabs(a[i]) + (i + 1 < m ? std::fabs(b[i]) : 0.0));
  const double eps = 2.220446049250313e-16, tiny = std::max(eps * norm, 1e-300);
  std::vector<double> d(m), u(m), u2(m), l(m);
  std::vector<char> swp(m);
  for (int k = 0; k < nk; ++k) {
    // T - w_k = P L U with partial pivoting (U has two superdiagonals)
    for (int i = 0; i < m; ++i) {
      d[i] = a[i] - w[k];
      u[i] = i + 1 < m ? b[i] : 0.0;
      u2[i] = 0.0;
    }
    for (int i = 0; i + 1 < m; ++i) {
      const double s = b[i];  // subdiagonal of row i + 1
      swp[i] = std::fabs(s) > std::fabs(d[i]);
      if (!swp[i]) {
        if (std::fabs(d[i]) < tiny) d[i] = d[i] < 0 ? -tiny : tiny;
        l[i] = s / d[i];
        d[i + 1] -= l[i] * u[i];
      } else {
        l[i] = d[i] / s;
        const double du = u[i], dn = d[i + 1], un = i + 2 < m ? u[i + 1] : 0.0;
        d[i] = s;
        u[i] = dn;
        u2[i] = un;
        d[i + 1] = du - l[i] * dn;
        if (i + 2 < m) u[i + 1] = -l[i] * un;
      }
    }
    if (std::fabs(d[m - 1]) < tiny) d[m - 1] = d[m - 1] < 0 ? -tiny : tiny;
    double* y = Q + (size_t)k * m;
    for (int i = 0; i < m; ++i) y[i] = 1.0 + 0.25 * ((i * 7 + k) % 5);
    for (int it = 0; it < 4; ++it) {
      if (it > 0) {  // the start already stands for L^{-1} P of some vector
        for (int i = 0; i + 1 < m; ++i) {
          if (swp[i]) std::swap(y[i], y[i + 1]);
          y[i + 1] -= l[i] * y[i];
        }
      }
      for (int i = m - 1; i >= 0; --i) {
        double v = y[i];
        if (i + 1 < m) v -= u[i] * y[i + 1];
        if (i + 2 < m) v -= u2[i] * y[i + 2];
        y[i] = v / d[i];
        if (std::fabs(y[i]) > 1e200)  // keep the solution in range
          for (int r = 0; r < m; ++r) y[r] *= 1e-200;
      }
      for (int c = k - 1; c >= 0 && std::fabs(w[k] - w[c]) <= 1e-3 * norm; --c) {
        const double* z = Q + (size_t)c * m;
        double dot = 0.0;
        for (int i = 0; i < m; ++i) dot += z[i] * y[i];
        for (int i = 0; i < m; ++i) y[i] -= dot * z[i];
      }
      double big = 0.0, n2 = 0.0;
      for (int i = 0; i < m; ++i) big = std::max(big, std::fabs(y[i]));
      const double sc = big > 0.0 ? 1.0 / big : 1.0;
      for (int i = 0; i < m; ++i) {
        y[i] *= sc;
        n2 += y[i] * y[i];
      }
      const double r = (y[0] < 0 ? -1.0 : 1.0) / std::sqrt(n2);
      for (int i = 0; i < m; ++i) y[i] *= r;
    }
  }
}

}  // namespace edk
