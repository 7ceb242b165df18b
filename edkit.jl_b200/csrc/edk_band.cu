// edk_band.cu — the eigenvalue step of the block Lanczos on the device: the
// lowest distinct eigenvalues of each operator's block-tridiagonal T (p x p
// Hermitian blocks A_j on the diagonal, B_j below it), found the way the host
// form in edk_block.cu finds them (band_lowest): candidates from a Lanczos on
// T with full re-orthogonalisation (classical Gram-Schmidt twice), each kept
// only when T has more eigenvalues in a small window around it than T-hat (T
// without its first block row and column) — the Cullum-Willoughby test
// generalised to blocks, with exact counts from block Sturm (inertia)
// sequences.  All operators' T run together: a Lanczos step is four
// launches over every operator, and every Sturm count is one thread block.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "edk_internal.cuh"

namespace edk {

namespace {

constexpr int kBandSteps = 1200;  // Lanczos steps on T at most (the host form's limit)

__device__ __forceinline__ double bwsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Shapes shared by the kernels: T_q has mq[q] blocks (at most mmax), rows
// n_q = p * mq[q] (at most nmax); A and B hold block j of operator q at
// (j nops + q) p^2 (B_0 unused), as the block Lanczos wrote its steps; V holds
// `vcols` columns of nmax rows per operator.
struct BandDims {
  int p, nops, mmax, vcols;
  int64_t nmax;
  __device__ size_t block(int q, int j) const { return ((size_t)j * nops + q) * p * p; }
};

// w = T v_k: a block takes G = blockDim.x / (3 p) block rows of operator q; of the
// 3 p threads of a block row, thread (t, a) multiplies row a of B_j, A_j or
// B_{j+1}^H (t = 0, 1, 2) by x_{j-1+t}, and the three sums meet in shared memory.
// Bound by the latency of the entries a thread walks, so three threads share a
// row and eight entries are in flight (p is a multiple of 8).
__global__ void k_band_mv(BandDims d, const double2* __restrict__ A, const double2* __restrict__ B,
                          const int* __restrict__ mq, const double2* __restrict__ V, int k,
                          double2* __restrict__ w, const int* __restrict__ stop) {
  extern __shared__ double2 sx_all[];  // per block row: x_{jb-1}, x_jb, x_{jb+1}, then the sums
  const int q = blockIdx.y, p = d.p;
  if (stop[q]) return;
  const int G = blockDim.x / (3 * p), m = mq[q];
  const int g = threadIdx.x / (3 * p), e = threadIdx.x - g * 3 * p, t = e / p, a = e - t * p;
  const int jb = blockIdx.x * G + g, jj = jb - 1 + t;
  double2* sx = sx_all + 3 * p * g;
  double2* sum = sx_all + 3 * p * (G + g);
  const bool in = jb < m && jj >= 0 && jj < m;
  sx[e] = in ? V[((size_t)q * d.vcols + k) * d.nmax + (size_t)jj * p + a] : make_double2(0.0, 0.0);
  __syncthreads();
  double yr = 0.0, yi = 0.0;
  if (in) {
    const double2* xs = sx + t * p;
    if (t < 2) {  // B_j x_{j-1}, A_j x_j
      const double2* M = (t == 0 ? B : A) + d.block(q, jb) + a;
#pragma unroll 8
      for (int c = 0; c < p; ++c) {
        const double2 v = M[(size_t)c * p], xc = xs[c];
        yr += v.x * xc.x - v.y * xc.y;
        yi += v.x * xc.y + v.y * xc.x;
      }
    } else {  // B_{j+1}^H x_{j+1}: conj(B(c, a)) x_c
      const double2* M = B + d.block(q, jb + 1) + (size_t)a * p;
#pragma unroll 8
      for (int c = 0; c < p; ++c) {
        const double2 v = M[c], xc = xs[c];
        yr += v.x * xc.x + v.y * xc.y;
        yi += v.x * xc.y - v.y * xc.x;
      }
    }
  }
  sum[e] = make_double2(yr, yi);
  __syncthreads();
  if (t != 1 || jb >= m) return;
  const double2 lo = sum[a], up = sum[2 * p + a];
  w[(size_t)q * d.nmax + (size_t)jb * p + a] = make_double2((yr + lo.x) + up.x, (yi + lo.y) + up.y);
}

// The step orthogonalises twice with two passes over V, as the batched Lanczos
// does (k_rdots2 in edk_batch.cu): V[:, k] arrives after one sweep, its second
// sweep shares the passes of the next vector's first.
//
// s[q][c] = V_q[:, c]^H V_q[:, k] and r[q][c] = V_q[:, c]^H w_q for c <= k: one
// warp per (column, operator)
__global__ void __launch_bounds__(256) k_band_dots(BandDims d, const int* __restrict__ nq,
                                                   const double2* __restrict__ V, int k,
                                                   const double2* __restrict__ w,
                                                   double2* __restrict__ s, double2* __restrict__ r,
                                                   const int* __restrict__ stop) {
  const int q = blockIdx.y;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (stop[q] || c > k) return;
  const int lane = threadIdx.x & 31;
  const int64_t n = nq[q];
  const double2* v = V + ((size_t)q * d.vcols + c) * d.nmax;
  const double2* u = V + ((size_t)q * d.vcols + k) * d.nmax;
  const double2* x = w + (size_t)q * d.nmax;
  double f[2][4] = {};  // two rows in flight; s, r (real and imaginary parts)
#pragma unroll 2
  for (int64_t i = lane; i < n; i += 64) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (i + 32 * e >= n) break;
      const double2 a = v[i + 32 * e], b = u[i + 32 * e], y = x[i + 32 * e];
      f[e][0] += a.x * b.x + a.y * b.y;
      f[e][1] += a.x * b.y - a.y * b.x;
      f[e][2] += a.x * y.x + a.y * y.y;
      f[e][3] += a.x * y.y - a.y * y.x;
    }
  }
  double t[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) t[e] = bwsum(f[0][e] + f[1][e]);
  if (lane == 0) {
    s[(size_t)q * d.vcols + c] = make_double2(t[0], t[1]);
    r[(size_t)q * d.vcols + c] = make_double2(t[2], t[3]);
  }
}

// With a^2 = s_k - sum |s_c|^2 and g = (r_k - s^H r) / a^2 (sums over c < k):
// V[:, k] = (V[:, k] - V s) / a, final, and w = (w - V r - g (V[:, k] - V s)) / a,
// alpha_k = Re(g - beta_{k-1} s_{k-1} / a).  A block takes 32 rows, its eight warps
// every eighth column each, and the warps' sums meet in shared memory; every block
// adds up a and g for itself.  (One thread per row leaves four blocks per operator
// at order 960 and a serial walk over all columns.)  18 operators, the run of order
// 960, up to 280 columns: two sweeps of their own took 2 x (11.8 + 12.3) us a
// step, this 13.3 + 12.4.
__global__ void __launch_bounds__(256) k_band_update(BandDims d, const int* __restrict__ nq,
                                                     double2* __restrict__ V, int k,
                                                     const double2* __restrict__ s,
                                                     const double2* __restrict__ r,
                                                     double2* __restrict__ w,
                                                     double* __restrict__ alpha,
                                                     const double* __restrict__ beta,
                                                     const int* __restrict__ stop) {
  __shared__ double2 sum[2][8][32];
  __shared__ double red[8][3];
  const int q = blockIdx.y;
  if (stop[q]) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * 32 + lane;
  const bool on = i < nq[q];
  const double2* sq = s + (size_t)q * d.vcols;
  const double2* rq = r + (size_t)q * d.vcols;
  double ss = 0.0, hx = 0.0, hy = 0.0;
  for (int c = threadIdx.x; c < k; c += 256) {
    const double2 a = sq[c], b = rq[c];
    ss += a.x * a.x + a.y * a.y;
    hx += a.x * b.x + a.y * b.y;
    hy += a.x * b.y - a.y * b.x;
  }
  ss = bwsum(ss);
  hx = bwsum(hx);
  hy = bwsum(hy);
  if (lane == 0) {
    red[warp][0] = ss;
    red[warp][1] = hx;
    red[warp][2] = hy;
  }
  double2* v = V + (size_t)q * d.vcols * d.nmax + (on ? i : 0);
  double2 as = make_double2(0.0, 0.0), ar = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int c = warp; c < k; c += 8) {
    const double2 x = v[(size_t)c * d.nmax], y = sq[c], z = rq[c];
    as.x += x.x * y.x - x.y * y.y;
    as.y += x.x * y.y + x.y * y.x;
    ar.x += x.x * z.x - x.y * z.y;
    ar.y += x.x * z.y + x.y * z.x;
  }
  sum[0][warp][lane] = as;
  sum[1][warp][lane] = ar;
  __syncthreads();
  if (warp != 0) return;
  ss = hx = hy = 0.0;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    ss += red[u][0];
    hx += red[u][1];
    hy += red[u][2];
  }
  const double2 uu = sq[k], uw = rq[k];
  double a2 = uu.x - ss;
  if (a2 < 1e-30 * uu.x) a2 = 1e-30 * uu.x;  // (NaN stays)
  const double inva = 1.0 / sqrt(a2), gx = (uw.x - hx) / a2, gy = (uw.y - hy) / a2;
  if (blockIdx.x == 0 && lane == 0)
    alpha[(size_t)q * d.vcols + k] =
        gx - (k > 0 ? beta[(size_t)q * d.vcols + k - 1] * sq[k - 1].x * inva : 0.0);
  if (!on) return;
#pragma unroll
  for (int u = 1; u < 8; ++u) {
    as.x += sum[0][u][lane].x;
    as.y += sum[0][u][lane].y;
    ar.x += sum[1][u][lane].x;
    ar.y += sum[1][u][lane].y;
  }
  double2* vk = v + (size_t)k * d.nmax;
  double2* wi = w + (size_t)q * d.nmax + i;
  const double2 t = *vk, y = *wi;
  const double2 p = make_double2(t.x - as.x, t.y - as.y);
  *vk = make_double2(p.x * inva, p.y * inva);
  *wi = make_double2((y.x - ar.x - (gx * p.x - gy * p.y)) * inva,
                     (y.y - ar.y - (gx * p.y + gy * p.x)) * inva);
}

// beta_k = |w| and v_{k+1} = w / beta, after one sweep (one block per operator); a
// negligible beta (the host form's rule b < 1e-12 max(1, |a|)) stops the operator
// with k + 1 steps, recorded in stop[q]
__global__ void __launch_bounds__(1024) k_band_next(BandDims d, const int* __restrict__ nq, int k,
                                                    const double2* __restrict__ w,
                                                    const double* __restrict__ alpha,
                                                    double* __restrict__ beta,
                                                    double2* __restrict__ V,
                                                    int* __restrict__ stop) {
  __shared__ double sh[32];
  const int q = blockIdx.x;
  if (stop[q]) return;
  const int64_t n = nq[q];
  const double2* x = w + (size_t)q * d.nmax;
  double t = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) t += x[i].x * x[i].x + x[i].y * x[i].y;
  t = bwsum(t);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
  __syncthreads();
  const double n2 = bwsum(sh[threadIdx.x & 31]);
  const double a = alpha[(size_t)q * d.vcols + k], b = sqrt(n2);
  const bool end = b < 1e-12 * fmax(1.0, fabs(a));
  if (threadIdx.x == 0) {
    beta[(size_t)q * d.vcols + k] = b;
    if (end) stop[q] = k + 1;
  }
  if (end || k + 1 >= d.vcols) return;
  const double sc = 1.0 / b;
  double2* v = V + ((size_t)q * d.vcols + k + 1) * d.nmax;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
    v[i] = make_double2(x[i].x * sc, x[i].y * sc);
}

// One Sturm count: the number of eigenvalues below sigma of the
// block-tridiagonal matrix of operator q's blocks j0 .. m-1, as the sign count
// of its block LDL^H factorisation: M_j = A_j - sigma - B_j X_{j-1},
// X_{j-1} = M_{j-1}^{-1} B_j^H, each M_j factorised without pivoting (a
// pivot below `tiny` in magnitude is replaced by +-tiny, as in the host
// form).  One block of 256 threads; shared memory M, L, X (p^2 each) and the
// pivots.
struct BandTask {
  double sigma, tiny;
  int q, j0;
};

__global__ void __launch_bounds__(256) k_band_sturm(BandDims d, const double2* __restrict__ A,
                                                    const double2* __restrict__ B,
                                                    const int* __restrict__ mq,
                                                    const BandTask* __restrict__ tasks,
                                                    int* __restrict__ counts) {
  extern __shared__ double2 sm[];
  const int p = d.p;
  const int pp = p * p;
  double2* M = sm;
  double2* L = sm + pp;
  double2* X = sm + 2 * pp;
  double* dg = reinterpret_cast<double*>(sm + 3 * pp);
  __shared__ int s_neg;
  const BandTask tk = tasks[blockIdx.x];
  const int q = tk.q, m = mq[q];
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid == 0) s_neg = 0;
  bool have_x = false;
  for (int j = tk.j0; j < m; ++j) {
    const double2* Aj = A + d.block(q, j);
    for (int e = tid; e < pp; e += nt) {
      double2 v = Aj[e];
      if (e % (p + 1) == 0) v.x -= tk.sigma;  // the diagonal entries a (p + 1)
      M[e] = v;
      if (have_x) L[e] = B[d.block(q, j) + e];  // B_j, staged
    }
    __syncthreads();
    if (have_x) {  // M -= B_j X
      for (int e = tid; e < pp; e += nt) {
        const int a = e % p, c = e / p;
        double sr = 0.0, si = 0.0;
        for (int t = 0; t < p; ++t) {
          const double2 b = L[a + t * p], x = X[t + c * p];
          sr += b.x * x.x - b.y * x.y;
          si += b.x * x.y + b.y * x.x;
        }
        M[e].x -= sr;
        M[e].y -= si;
      }
      __syncthreads();
    }
    // right-looking LDL^H on the lower triangle: L(i, k) for i > k, pivots dg
    for (int k = 0; k < p; ++k) {
      if (tid == 0) {
        double dk = M[k + k * p].x;
        if (fabs(dk) < tk.tiny) dk = dk < 0 ? -tk.tiny : tk.tiny;
        dg[k] = dk;
        if (dk < 0) ++s_neg;
      }
      __syncthreads();
      const double dk = dg[k];
      for (int i = k + 1 + tid; i < p; i += nt) {
        const double2 v = M[i + k * p];
        L[i + k * p] = make_double2(v.x / dk, v.y / dk);
      }
      __syncthreads();
      const int r = p - k - 1;
      for (int e = tid; e < r * r; e += nt) {
        const int i = k + 1 + e % r, jj = k + 1 + e / r;
        if (jj > i) continue;
        const double2 li = L[i + k * p], lj = L[jj + k * p];
        // M(i, jj) -= L(i, k) dk conj(L(jj, k))
        M[i + jj * p].x -= dk * (li.x * lj.x + li.y * lj.y);
        M[i + jj * p].y -= dk * (li.y * lj.x - li.x * lj.y);
      }
      __syncthreads();
    }
    if (j + 1 < m) {
      // X = M^{-1} B_{j+1}^H: column c (four lanes of one warp each, p a
      // multiple of 8 so a warp's columns are all inside or all outside)
      const double2* Bn = B + d.block(q, j + 1);
      const int c = tid >> 2, part = tid & 3;
      if (c < p) {
        double2* x = X + (size_t)c * p;
        for (int a = part; a < p; a += 4) {  // rhs(a) = conj(B(c, a))
          const double2 b = Bn[c + (size_t)a * p];
          x[a] = make_double2(b.x, -b.y);
        }
        __syncwarp();
        for (int a = 0; a < p; ++a) {  // L y = rhs (unit lower)
          double sr = 0.0, si = 0.0;
          for (int t = part; t < a; t += 4) {
            const double2 l = L[a + t * p], y = x[t];
            sr += l.x * y.x - l.y * y.y;
            si += l.x * y.y + l.y * y.x;
          }
          sr += __shfl_xor_sync(0xffffffffu, sr, 1);
          si += __shfl_xor_sync(0xffffffffu, si, 1);
          sr += __shfl_xor_sync(0xffffffffu, sr, 2);
          si += __shfl_xor_sync(0xffffffffu, si, 2);
          if (part == 0) x[a] = make_double2(x[a].x - sr, x[a].y - si);
          __syncwarp();
        }
        for (int a = part; a < p; a += 4) x[a] = make_double2(x[a].x / dg[a], x[a].y / dg[a]);
        __syncwarp();
        for (int a = p - 1; a >= 0; --a) {  // L^H z = y
          double sr = 0.0, si = 0.0;
          for (int t = a + 1 + part; t < p; t += 4) {
            const double2 l = L[t + a * p], y = x[t];  // conj(L(t, a)) y_t
            sr += l.x * y.x + l.y * y.y;
            si += l.x * y.y - l.y * y.x;
          }
          sr += __shfl_xor_sync(0xffffffffu, sr, 1);
          si += __shfl_xor_sync(0xffffffffu, si, 1);
          sr += __shfl_xor_sync(0xffffffffu, sr, 2);
          si += __shfl_xor_sync(0xffffffffu, si, 2);
          if (part == 0) x[a] = make_double2(x[a].x - sr, x[a].y - si);
          __syncwarp();
        }
      }
      __syncthreads();
      have_x = true;
    }
  }
  if (tid == 0) counts[blockIdx.x] = s_neg;
}

// The diagonal blocks of the steps since the last call, from[q] .. mq[q] - 1, as the
// kernels read them, in place: A[j][q] arrives as (V_j^H W)^T column-major, so A_j(r, c) =
// A[c + r p], and is made Hermitian.  diag[q] rises to the largest |A_j(a, a)| over all j,
// diag[nops + q] over j >= 1 (at least one), as the bits of non-negative doubles.
__global__ void __launch_bounds__(256) k_band_pack(BandDims d, double2* __restrict__ A,
                                                   const int* __restrict__ from,
                                                   const int* __restrict__ mq,
                                                   unsigned long long* __restrict__ diag) {
  const int q = blockIdx.y, j = from[q] + blockIdx.x, p = d.p;
  if (j >= mq[q]) return;
  double2* a = A + d.block(q, j);
  for (int e = threadIdx.x; e < p * p; e += blockDim.x) {
    const int r = e % p, c = e / p;
    if (r > c) continue;
    const double2 x = a[c + r * p], y = a[r + c * p];  // A(r, c), A(c, r)
    const double2 h = make_double2(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
    a[r + c * p] = h;
    if (r != c) {
      a[c + r * p] = make_double2(h.x, -h.y);
    } else {
      const unsigned long long v = (unsigned long long)__double_as_longlong(fmax(1.0, fabs(h.x)));
      atomicMax(diag + q, v);
      if (j >= 1) atomicMax(diag + d.nops + q, v);
    }
  }
}

}  // namespace

edk_status band_lowest_device(int p, int nev, const std::vector<int>& m, void* SA, const void* SB,
                              BandState& state, cudaStream_t st,
                              std::vector<std::vector<double>>& out) {
  const int nops = (int)m.size();
  out.assign(nops, std::vector<double>(nev, NAN));
  if (nops == 0) return EDK_OK;
  if (p < 8 || p > 64 || p % 8 != 0) {
    set_error("block eigenvalue step: block must be a multiple of 8 between 8 and 64");
    return EDK_INVALID_ARG;
  }
  BandDims d;
  d.p = p;
  d.nops = nops;
  d.mmax = std::max(1, *std::max_element(m.begin(), m.end()));
  d.nmax = (int64_t)p * d.mmax;
  const int kmax = (int)std::min<int64_t>(d.nmax, kBandSteps);
  d.vcols = kmax + 1;
  const size_t pp = (size_t)p * p;
  DevBuf V, w, s1, s2, alpha, beta, stop, nq, mqd, from;
  double2* dA = static_cast<double2*>(SA);
  const double2* dB = static_cast<const double2*>(SB);
  if (state.packed.empty()) {
    state.packed.assign(nops, 0);
    EDK_RETURN_IF(state.diag.alloc_async(2 * (size_t)nops * 8, st));
    EDK_TRY_CUDA(cudaMemsetAsync(state.diag.p, 0, 2 * (size_t)nops * 8, st));
  }
  std::vector<int> hn(nops);
  for (int q = 0; q < nops; ++q) hn[q] = p * m[q];
  EDK_RETURN_IF(V.alloc_async((size_t)nops * d.vcols * d.nmax * sizeof(double2), st));
  EDK_RETURN_IF(w.alloc_async((size_t)nops * d.nmax * sizeof(double2), st));
  EDK_RETURN_IF(s1.alloc_async((size_t)nops * d.vcols * sizeof(double2), st));
  EDK_RETURN_IF(s2.alloc_async((size_t)nops * d.vcols * sizeof(double2), st));
  EDK_RETURN_IF(alpha.alloc_async((size_t)nops * d.vcols * sizeof(double), st));
  EDK_RETURN_IF(beta.alloc_async((size_t)nops * d.vcols * sizeof(double), st));
  EDK_RETURN_IF(stop.alloc_async((size_t)nops * sizeof(int), st));
  EDK_RETURN_IF(nq.alloc_async((size_t)nops * sizeof(int), st));
  EDK_RETURN_IF(mqd.alloc_async((size_t)nops * sizeof(int), st));
  EDK_TRY_CUDA(cudaMemcpyAsync(nq.p, hn.data(), nops * sizeof(int), cudaMemcpyHostToDevice, st));
  EDK_TRY_CUDA(cudaMemcpyAsync(mqd.p, m.data(), nops * sizeof(int), cudaMemcpyHostToDevice, st));
  EDK_RETURN_IF(from.alloc_async((size_t)nops * sizeof(int), st));
  EDK_TRY_CUDA(cudaMemcpyAsync(from.p, state.packed.data(), nops * sizeof(int),
                               cudaMemcpyHostToDevice, st));
  int fresh = 0;
  for (int q = 0; q < nops; ++q) fresh = std::max(fresh, m[q] - state.packed[q]);
  if (fresh > 0) {
    k_band_pack<<<dim3(fresh, nops), 256, 0, st>>>(d, dA, from.as<int>(), mqd.as<int>(),
                                                   state.diag.as<unsigned long long>());
    EDK_TRY_CUDA(cudaGetLastError());
  }
  std::vector<double> hmax(2 * (size_t)nops);
  EDK_TRY_CUDA(cudaMemcpyAsync(hmax.data(), state.diag.p, hmax.size() * 8, cudaMemcpyDeviceToHost, st));
  EDK_TRY_CUDA(cudaMemsetAsync(stop.p, 0, nops * sizeof(int), st));
  EDK_TRY_CUDA(cudaMemsetAsync(V.p, 0, (size_t)nops * d.vcols * d.nmax * sizeof(double2), st));
  // start vectors: the host form's seeded sequence, normalised, in column 0
  {
    std::vector<double2> v0((size_t)nops * d.nmax, make_double2(0.0, 0.0));
    for (int q = 0; q < nops; ++q) {
      uint64_t s = 0x12345678abcdefull;
      auto rnd = [&]() {
        s ^= s << 13;
        s ^= s >> 7;
        s ^= s << 17;
        return ((s >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
      };
      double nr = 0.0;
      double2* v = v0.data() + (size_t)q * d.nmax;
      for (int i = 0; i < hn[q]; ++i) {
        const double re = rnd(), im = rnd();
        v[i] = make_double2(re, im);
        nr += re * re + im * im;
      }
      nr = std::sqrt(nr);
      for (int i = 0; i < hn[q]; ++i) v[i] = make_double2(v[i].x / nr, v[i].y / nr);
      EDK_TRY_CUDA(cudaMemcpyAsync(V.as<double2>() + (size_t)q * d.vcols * d.nmax, v,
                                   (size_t)d.nmax * sizeof(double2), cudaMemcpyHostToDevice, st));
    }
    EDK_TRY_CUDA(cudaStreamSynchronize(st));
  }
  state.packed = m;
  // Lanczos on every T in lockstep; the host looks every 10 steps (and at
  // each operator's own last step), as the host form does
  std::vector<std::vector<double>> prev(nops), cand(nops);
  std::vector<int> finished(nops, 0), hstop(nops, 0);
  // the lowest nk eigenvalues of each Lanczos matrix, on the device
  // (edk_tridiag.cu): nev + 4 candidates, more only once values merge
  int nk = nev + 4;
  DevBuf evd;
  EDK_RETURN_IF(evd.alloc_async((size_t)nops * nk * sizeof(double), st));
  std::vector<double> hev((size_t)nops * nk);
  const unsigned rows = (unsigned)((d.nmax + 31) / 32);
  const int G = std::max(1, 64 / p);  // block rows per block of k_band_mv
  int left = nops;
  for (int k = 0; k < kmax && left > 0; ++k) {
    k_band_mv<<<dim3((d.mmax + G - 1) / G, nops), 3 * G * p, 6 * G * p * sizeof(double2), st>>>(
        d, dA, dB, mqd.as<int>(), V.as<double2>(), k, w.as<double2>(),
        stop.as<int>());
    k_band_dots<<<dim3((k + 8) / 8, nops), 256, 0, st>>>(d, nq.as<int>(), V.as<double2>(), k,
                                                        w.as<double2>(), s1.as<double2>(),
                                                        s2.as<double2>(), stop.as<int>());
    k_band_update<<<dim3(rows, nops), 256, 0, st>>>(d, nq.as<int>(), V.as<double2>(), k,
                                                    s1.as<double2>(), s2.as<double2>(),
                                                    w.as<double2>(), alpha.as<double>(),
                                                    beta.as<double>(), stop.as<int>());
    k_band_next<<<nops, 1024, 0, st>>>(d, nq.as<int>(), k, w.as<double2>(), alpha.as<double>(),
                                       beta.as<double>(), V.as<double2>(), stop.as<int>());
    EDK_TRY_CUDA(cudaGetLastError());
    bool look = (k + 1) % 10 == 0 || k + 1 == kmax;
    for (int q = 0; q < nops && !look; ++q)
      look = !finished[q] && k + 1 == std::min(hn[q], kBandSteps);
    if (!look) continue;
    // (repeated with twice as many values while one matrix has too few
    // distinct ones among them)
    std::vector<std::vector<double>> dist(nops);
    for (bool again = true; again;) {
      again = false;
      EDK_RETURN_IF(tridiag_lowest_device(nops, alpha.as<double>(), beta.as<double>(), d.vcols,
                                          nullptr, stop.as<int>(), k + 1, nk, evd.as<double>(), st));
      EDK_TRY_CUDA(cudaMemcpyAsync(hev.data(), evd.p, hev.size() * sizeof(double),
                                   cudaMemcpyDeviceToHost, st));
      EDK_TRY_CUDA(cudaMemcpyAsync(hstop.data(), stop.p, nops * sizeof(int),
                                   cudaMemcpyDeviceToHost, st));
      EDK_TRY_CUDA(cudaStreamSynchronize(st));
      for (int q = 0; q < nops; ++q) {
        if (finished[q]) continue;
        const int mm = hstop[q] > 0 ? hstop[q] : k + 1;
        std::vector<double>& dd = dist[q];  // distinct values: closer than 1e-12 relative merge
        dd.clear();
        for (int t = 0; t < std::min(nk, mm); ++t) {
          const double x = hev[(size_t)q * nk + t];
          if (dd.empty() || x - dd.back() > 1e-12 * std::max(1.0, std::fabs(x))) dd.push_back(x);
        }
        again = again || ((int)dd.size() < nev + 4 && nk < mm);
      }
      if (again) {
        nk = std::min(2 * nk, k + 1);
        EDK_RETURN_IF(evd.alloc_async((size_t)nops * nk * sizeof(double), st));
        hev.resize((size_t)nops * nk);
      }
    }
    bool changed = false;
    for (int q = 0; q < nops; ++q) {
      if (finished[q]) continue;
      const int own = std::min(hn[q], kBandSteps);
      const bool last = hstop[q] > 0 || k + 1 >= own;
      if (!last && (k + 1) % 10 != 0) continue;
      const std::vector<double>& dd = dist[q];
      bool conv = last;
      if (!conv && (int)dd.size() >= nev + 4 && (int)prev[q].size() >= nev + 4) {
        conv = true;
        for (int t = 0; t < nev + 4; ++t)
          if (std::fabs(dd[t] - prev[q][t]) > 1e-13 * std::max(1.0, std::fabs(dd[0]))) conv = false;
      }
      prev[q] = dd;
      if (conv) {
        cand[q].assign(dd.begin(), dd.begin() + std::min<size_t>(dd.size(), nev + 4));
        finished[q] = 1;
        --left;
        if (hstop[q] == 0) {
          hstop[q] = k + 1;
          changed = true;
        }
      }
    }
    if (changed)
      EDK_TRY_CUDA(cudaMemcpyAsync(stop.p, hstop.data(), nops * sizeof(int), cudaMemcpyHostToDevice, st));
  }
  for (int q = 0; q < nops; ++q)
    if (!finished[q]) cand[q] = prev[q].size() > (size_t)nev + 4
                                    ? std::vector<double>(prev[q].begin(), prev[q].begin() + nev + 4)
                                    : prev[q];
  // Sturm counts at both edges of every candidate cluster, for T and T-hat
  struct Cluster { int q; double lo, hi, dl; };
  std::vector<Cluster> cl;
  std::vector<BandTask> tasks;
  for (int q = 0; q < nops; ++q) {
    double tiny[2];
    for (int j0 = 0; j0 < 2; ++j0)
      tiny[j0] = 1e-300 + 1e-15 * std::max(1.0, hmax[(size_t)j0 * nops + q]);
    const std::vector<double>& c = cand[q];
    for (size_t i = 0; i < c.size();) {
      const double lo = c[i], dl = 1e-10 * std::max(1.0, std::fabs(lo));
      double hi = lo;
      size_t e = i + 1;
      while (e < c.size() && c[e] - hi <= dl) hi = c[e++];
      cl.push_back({q, lo, hi, dl});
      for (int j0 = 0; j0 < (m[q] > 1 ? 2 : 1); ++j0) {
        tasks.push_back({hi + dl, tiny[j0], q, j0});
        tasks.push_back({lo - dl, tiny[j0], q, j0});
      }
      i = e;
    }
  }
  std::vector<int> hc(tasks.size(), 0);
  if (!tasks.empty()) {
    DevBuf dt, dc;
    EDK_RETURN_IF(dt.alloc_async(tasks.size() * sizeof(BandTask), st));
    EDK_RETURN_IF(dc.alloc_async(tasks.size() * sizeof(int), st));
    EDK_TRY_CUDA(cudaMemcpyAsync(dt.p, tasks.data(), tasks.size() * sizeof(BandTask),
                                 cudaMemcpyHostToDevice, st));
    const size_t smem = 3 * pp * sizeof(double2) + p * sizeof(double);
    // the largest block's size (p = 64), the same from every calling thread
    EDK_TRY_CUDA(cudaFuncSetAttribute(k_band_sturm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(3 * 64 * 64 * sizeof(double2) + 64 * sizeof(double))));
    k_band_sturm<<<(unsigned)tasks.size(), 256, smem, st>>>(d, dA, dB,
                                                             mqd.as<int>(), dt.as<BandTask>(),
                                                             dc.as<int>());
    EDK_TRY_CUDA(cudaGetLastError());
    EDK_TRY_CUDA(cudaMemcpyAsync(hc.data(), dc.p, hc.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
    EDK_TRY_CUDA(cudaStreamSynchronize(st));
  }
  // keep a cluster when T has more eigenvalues in its window than T-hat
  std::vector<int> got(nops, 0);
  size_t t = 0;
  for (const Cluster& c : cl) {
    const int q = c.q;
    const int nt = hc[t] - hc[t + 1];
    const int nh = m[q] > 1 ? hc[t + 2] - hc[t + 3] : 0;
    t += m[q] > 1 ? 4 : 2;
    if (got[q] < nev && nt - nh >= 1) out[q][got[q]++] = c.lo;
  }
  return EDK_OK;
}

}  // namespace edk
