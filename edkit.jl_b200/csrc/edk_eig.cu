// edk_eig.cu — eigenvalues of a dense Hermitian matrix that fits the shared memory
// of all SMs, 1,808 rows real, 1,205 complex (the Gram matrices of ent_spec /
// ent_S, src/Schmidt.jl:84-165): Householder tridiagonalisation there, then the
// multi-section Sturm kernel (edk_tridiag.cu) for all eigenvalues at once.
//
// A tridiagonalisation is n dependent steps of one matrix-vector product and one
// rank-two update, so it is bound by what a step cannot overlap: a product needs
// the reflector, the reflector the column the last update left.  The matrix
// (8 MB at n = 1,024) stays in shared memory, columns dealt out cyclically to the
// blocks of one cooperative launch, one block per SM, one warp per column; both
// triangles are held, so each block multiplies and updates its own columns in
// one pass.  One grid barrier per step is left: before it a block publishes its
// entries of p = tau A v and the owner of the next column that column; after it
// every block forms w, the updated next column and its reflector for itself
// (n / 256 elements a thread) instead of waiting for the owner.
//   Gram matrix of 1,024 rows, real: cuSOLVER 11.3 ms (28 launches of the
//   reduction 9.3 ms, divide and conquer 2.0 ms), here 4.7 + 0.2 ms.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "edk_internal.cuh"

namespace edk {

namespace {

constexpr int kEigThreads = 256;
constexpr unsigned kEigPolls = 1u << 22;  // of a barrier, a second or two

__device__ __forceinline__ double cj(double a) { return a; }
__device__ __forceinline__ double2 cj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double mulx(double a, double b) { return a * b; }
__device__ __forceinline__ double2 mulx(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double mulx(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double2 mulx(double2 a, double2 b, double2 c) {  // a b + c
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ double neg(double a) { return -a; }
__device__ __forceinline__ double2 neg(double2 a) { return make_double2(-a.x, -a.y); }
__device__ __forceinline__ double scale(double a, double s) { return a * s; }
__device__ __forceinline__ double2 scale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double re(double a) { return a; }
__device__ __forceinline__ double re(double2 a) { return a.x; }
__device__ __forceinline__ double im(double) { return 0.0; }
__device__ __forceinline__ double im(double2 a) { return a.y; }
__device__ __forceinline__ void mk(double& o, double r, double) { o = r; }
__device__ __forceinline__ void mk(double2& o, double r, double i) { o = make_double2(r, i); }
__device__ __forceinline__ double wred(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double2 wred(double2 v) { return make_double2(wred(v.x), wred(v.y)); }
__device__ __forceinline__ double ldc(const double* p) { return __ldcg(p); }
__device__ __forceinline__ double2 ldc(const double2* p) { return __ldcg(p); }

// sum over the block, to every thread; `sh` alternates between two halves, so
// one __syncthreads is enough
template <class T>
__device__ __forceinline__ T bred(T v, T* sh) {
  v = wred(v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  T t = sh[0];
#pragma unroll
  for (int k = 1; k < kEigThreads / 32; ++k) {
    T o = sh[k];
    mk(t, re(t) + re(o), im(t) + im(o));
  }
  return t;
}

// d[n], e[n-1] of T = Q^H A Q for the Hermitian A whose lower triangle is in G
// (column-major, ld n).  pbuf, cbuf: 2 n each; bar zeroed; *err: 1 a barrier ran
// out of polls, 2 A is not finite.
template <class T>
__global__ void __launch_bounds__(kEigThreads, 1) k_tridiagonalise(
    int n, const T* __restrict__ G, double* __restrict__ d, double* __restrict__ e, T* pbuf,
    T* cbuf, unsigned* bar, int* err, unsigned polls_max) {
  extern __shared__ __align__(16) unsigned char raw[];
  T* v = reinterpret_cast<T*>(raw);  // v_k, zero up to row k
  T* w = v + n;                      // w_k
  T* u = w + n;                      // the next column, then v_{k+1}
  T* cols = u + n;
  __shared__ T sh[2][kEigThreads / 32];
  __shared__ double s_max[kEigThreads / 32];
  __shared__ int s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = blockIdx.x, nb = gridDim.x;
  const int ncl = (n - b + nb - 1) / nb;  // own columns b, b + nb, ...
  // scale to a largest diagonal entry in [1, 2): a Gram matrix's largest entry
  double mx = 0.0;
  for (int r = tid; r < n; r += kEigThreads) {
    const double x = fabs(re(G[(size_t)r * n + r]));
    mx = x > mx || x != x ? x : mx;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double x = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = x > mx || x != x ? x : mx;
  }
  if (lane == 0) s_max[warp] = mx;
  if (tid == 0) s_fail = 0;
  __syncthreads();
  for (int k = 0; k < kEigThreads / 32; ++k) mx = s_max[k] > mx || s_max[k] != s_max[k] ? s_max[k] : mx;
  if (!(mx <= 1e300)) {  // every block sees the same entries
    if (b == 0 && tid == 0) *err = 2;
    return;
  }
  const double up = mx > 1e-300 ? scalbn(1.0, ilogb(mx)) : 1.0, dn = 1.0 / up;
  for (int i = 0; i < ncl; ++i) {
    const int c = b + nb * i;
    for (int r = tid; r < n; r += kEigThreads) {
      const T a = r >= c ? G[(size_t)c * n + r] : cj(G[(size_t)r * n + c]);
      cols[(size_t)i * n + r] = scale(a, dn);
    }
  }
  for (int r = tid; r < n; r += kEigThreads) {
    u[r] = scale(G[r], dn);
    mk(v[r], 0.0, 0.0);
    mk(w[r], 0.0, 0.0);
  }
  __syncthreads();
  if (b == 0 && tid == 0) d[0] = re(u[0]) * up;
  if (n == 1) return;
  int half = 0;
  unsigned target = 0;
  for (int k = -1; k <= n - 2; ++k) {
    T tau;
    if (k >= 0) {
      // ---- step k's product is published: w_k and the updated column k + 1
      __syncthreads();
      if (tid == 0) {
        target += nb;
        __threadfence();
        atomicAdd(bar, 1u);
        unsigned polls = 0, seen;
        do {
          asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
        } while (seen < target && ++polls < polls_max);
        if (seen < target) {
          s_fail = 1;
          *err = 1;
        }
      }
      __syncthreads();
      if (s_fail) return;
      const T* p = pbuf + (size_t)(k & 1) * n;
      const T* cn = cbuf + (size_t)(k & 1) * n;
      // p[] carries tau A v; its own tau travels in p[k] (below the active rows)
      tau = ldc(p + k);
      T dot;
      mk(dot, 0.0, 0.0);
      for (int r = k + 1 + tid; r < n; r += kEigThreads) {
        const T x = ldc(p + r);
        w[r] = x;
        u[r] = ldc(cn + r);
        dot = mulx(cj(x), v[r], dot);
      }
      dot = bred(dot, sh[half ^= 1]);
      const T a2 = scale(mulx(tau, dot), -0.5);  // w = p - tau / 2 (p^H v) v
      for (int r = k + 1 + tid; r < n; r += kEigThreads) w[r] = mulx(a2, v[r], w[r]);
      __syncthreads();
      const T wc = neg(cj(w[k + 1])), vc = neg(cj(v[k + 1]));
      for (int r = k + 1 + tid; r < n; r += kEigThreads)
        u[r] = mulx(w[r], vc, mulx(v[r], wc, u[r]));
      __syncthreads();
      if (b == 0 && tid == 0) d[k + 1] = re(u[k + 1]) * up;
      if (k == n - 2) break;
    }
    // ---- reflector of column j = k + 1: u[j+1 ..] = beta e_1 after it
    const int j = k + 1;
    double s = 0.0;
    for (int r = j + 2 + tid; r < n; r += kEigThreads) s += re(u[r]) * re(u[r]) + im(u[r]) * im(u[r]);
    T st;
    mk(st, s, 0.0);
    s = re(bred(st, sh[half ^= 1]));
    const T alpha = u[j + 1];
    const double ar = re(alpha), ai = im(alpha);
    double beta, inv_r = 0.0, inv_i = 0.0;
    T taun;
    // (a column below 1e-140 of the matrix, whose squares leave the range of doubles, is
    // dropped: its reflector would not be unitary in what bits are left, and it meets
    // entries of size one)
    if (s > 0.0 && ar * ar + ai * ai + s > 1e-280) {
      beta = -copysign(sqrt(ar * ar + ai * ai + s), ar);
      mk(taun, (beta - ar) / beta, -ai / beta);
      const double q = (ar - beta) * (ar - beta) + ai * ai;
      inv_r = (ar - beta) / q;
      inv_i = -ai / q;
    } else {  // nothing to eliminate, or nothing that counts (a phase of beta does not move eigenvalues)
      beta = sqrt(ar * ar + ai * ai);
      mk(taun, 0.0, 0.0);
    }
    __syncthreads();  // alpha is read
    T inv;
    mk(inv, inv_r, inv_i);
    for (int r = j + 1 + tid; r < n; r += kEigThreads) {
      if (r == j + 1) mk(u[r], 1.0, 0.0);
      else u[r] = mulx(u[r], inv);
    }
    if (b == 0 && tid == 0) e[j] = beta * up;
    __syncthreads();
    // ---- own columns past j: the update of step k and the product with v_j
    T* pn = pbuf + (size_t)(j & 1) * n;
    T* cnx = cbuf + (size_t)(j & 1) * n;
    if (b == 0 && tid == 0) pn[j] = taun;
    for (int i = warp; i < ncl; i += kEigThreads / 32) {
      const int c = b + nb * i;
      if (c <= j) continue;
      T* a = cols + (size_t)i * n;
      const T wc = neg(cj(w[c])), vc = neg(cj(v[c]));
      T s1;
      mk(s1, 0.0, 0.0);
      for (int r = j + 1 + lane; r < n; r += 32) {
        const T x = mulx(w[r], vc, mulx(v[r], wc, a[r]));
        a[r] = x;
        s1 = mulx(cj(x), u[r], s1);
        if (c == j + 1) cnx[r] = x;
      }
      s1 = wred(s1);
      if (lane == 0) pn[c] = mulx(taun, s1);
    }
    __syncthreads();
    T* t = v;  // v_j takes over; its rows up to j are never read again
    v = u;
    u = t;
  }
}

template <class T>
size_t eig_smem(int n, int nb) {
  return (size_t)((n + nb - 1) / nb + 3) * n * sizeof(T);
}

template <class T>
edk_status eig_run(int n, const void* G, double* W, cudaStream_t st) {
  int dev = 0, nsm = 0, optin = 0;
  EDK_TRY_CUDA(cudaGetDevice(&dev));
  EDK_TRY_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  EDK_TRY_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  // a warp per column while there are blocks for it (fewer blocks meet sooner)
  int nb = std::max(1, std::min(nsm, (n + 7) / 8));
  const size_t smem = eig_smem<T>(n, nb);
  if (smem + 1024 > (size_t)optin) return EDK_UNSUPPORTED;
  // the device's limit rather than this call's size: threads with different
  // sizes would take the attribute from one another between here and the launch
  EDK_TRY_CUDA(cudaFuncSetAttribute(k_tridiagonalise<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    optin - 1024));
  DevBuf buf;
  const size_t vb = 2 * (size_t)n * sizeof(T);
  EDK_RETURN_IF(buf.alloc_async(2 * vb + 2 * (size_t)n * 8 + 16, st));
  T* pbuf = buf.as<T>();
  T* cbuf = pbuf + 2 * n;
  double* d = reinterpret_cast<double*>(cbuf + 2 * n);
  double* e = d + n;
  unsigned* bar = reinterpret_cast<unsigned*>(e + n);
  int* err = reinterpret_cast<int*>(bar + 1);
  EDK_TRY_CUDA(cudaMemsetAsync(bar, 0, 8, st));
  const T* g = static_cast<const T*>(G);
  unsigned polls = kEigPolls;  // (fewer in the test of a barrier that gives up)
  if (const char* p = std::getenv("EDK_EIG_POLLS"))
    polls = (unsigned)std::min<unsigned long>(std::strtoul(p, nullptr, 10), kEigPolls);
  void* args[] = {&n, &g, &d, &e, &pbuf, &cbuf, &bar, &err, &polls};
  if (cudaLaunchCooperativeKernel((const void*)k_tridiagonalise<T>, dim3(nb), dim3(kEigThreads),
                                  args, smem, st) != cudaSuccess) {
    cudaGetLastError();  // blocks that are not resident together here (a share of the SMs)
    return EDK_UNSUPPORTED;
  }
  EDK_RETURN_IF(tridiag_lowest_device(1, d, e, n, nullptr, nullptr, n, n, W, st));
  int h = 0;
  EDK_TRY_CUDA(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st));
  EDK_TRY_CUDA(cudaStreamSynchronize(st));
  return h == 0 ? EDK_OK : EDK_UNSUPPORTED;  // out of polls, or not finite
}

}  // namespace

// All eigenvalues, ascending, of the Hermitian n x n matrix whose lower triangle
// is in G (column-major, real or interleaved complex; left as it is) into W, both
// on the device.  EDK_UNSUPPORTED: too large for the SMs' shared memory, not finite, or
// the blocks could not be launched together or wait for each other; the caller has
// another solver for those.
edk_status hermitian_eigvals(bool cx, int n, const void* G, double* W, cudaStream_t st) {
  return cx ? eig_run<double2>(n, G, W, st) : eig_run<double>(n, G, W, st);
}

}  // namespace edk
