// edk_pauli.cu — products on the full space (TensorBasis) with operators that
// are no flip-flop chains (transverse fields, XY and DM couplings, any local
// terms): the operator as a sum of Pauli strings.
//
// Every local matrix is a sum of products X^x Z^z (a Walsh-Hadamard transform
// of its entries M[c ^ x][c] over c), so row i of H x is
//   y_i = d_i x_i + sum_x conj(sum_z v_{x,z} (-1)^{|i & z|}) x_{i ^ x},
// the colmn! loop (src/Operator.jl:417-465) without digits, columns or target
// search: one gather per distinct flip mask x and one sign per string.
//
// The gathers are what bounds it, so a block takes 256 RPT consecutive rows and
// keeps their x in shared memory: flips of the low bits stay inside the tile
// (an XOR of the index: no bank conflicts), the others read whole lines of
// another tile, RPT of them in flight per thread.  Plain flips (one real value,
// no sign) sit in the kernel's parameters.  Transverse-field Ising
// chain, L = 20, real: 87 us as general rows, 17 us here (cold L2; L1 65% busy).
#include <algorithm>
#include <type_traits>

#include "edk_rows.cuh"

namespace edk {

namespace {

constexpr int kPauliThreads = 256;

// diagonal of row state s: bond families by popcounts, the rest as z strings
__device__ __forceinline__ double pauli_diag(const OpDev& op, const PauliDev& pd, int L,
                                             uint32_t mask, uint32_t s) {
  double d = 0.0;
  for (int f = 0; f < op.nfam; ++f) {
    const FamDev* F = op.fam + f;
    const uint32_t X = s, Y = rotl_L(s, F->d, L, mask), V = (uint32_t)F->valid;
    d += F->dval[0].x * __popc(~X & ~Y & V) + F->dval[1].x * __popc(~X & Y & V) +
         F->dval[2].x * __popc(X & ~Y & V) + F->dval[3].x * __popc(X & Y & V);
  }
  for (int q = 0; q < pd.ndiag; ++q) {
    const double v = __ldg(&pd.diag[q].v.x);
    d += (__popc(s & __ldg(&pd.diag[q].z)) & 1) ? -v : v;
  }
  return d;
}

// y(:, k) (+)= H x(:, k), k = blockIdx.y; with `step` the input starts at
// column *step of x, and a set *done skips the product (batched Lanczos).  The
// first nlow plain flips stay inside a tile.  FULL: every tile is full (D is a
// power of two, so a tile that is not is the only one, and its flips stay in it).
template <class VT, int RPT, bool FULL>
__global__ void __launch_bounds__(kPauliThreads, 4) k_apply_pauli(
    OpDev op, PauliDev pd, PauliFlips fl, int nlow, int L, uint32_t mask, int64_t D,
    const VT* __restrict__ x, VT* __restrict__ y, int64_t ldx, int64_t ldy, int accumulate,
    const int* __restrict__ step, const int* __restrict__ done) {
  using A = typename VTraits<VT>::A;
  constexpr bool CX = VTraits<VT>::cx;
  constexpr uint32_t R = kPauliThreads * RPT;
  __shared__ VT sx[R];
  if (done && *done) return;
  const VT* xk = x + (step ? (int64_t)*step * ldx : 0) + (int64_t)blockIdx.y * ldx;
  VT* yk = y + (int64_t)blockIdx.y * ldy;
  const uint32_t base = blockIdx.x * R, t = threadIdx.x;
  const uint32_t rows = FULL ? R : (uint32_t)D;  // rows of this tile
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const uint32_t l = t + r * kPauliThreads;
    if (FULL || l < rows) sx[l] = xk[base + l];
  }
  __syncthreads();
  Cx<A> acc[RPT];
#pragma unroll
  for (int r = 0; r < RPT; ++r) acc[r] = Cx<A>{0, 0};
  auto add = [&](int r, A v, Cx<A> xv) {
    acc[r].r = fma_(v, xv.r, acc[r].r);
    if constexpr (CX) acc[r].i = fma_(v, xv.i, acc[r].i);
  };
  for (int f = 0; f < nlow; ++f) {
    const uint32_t lx = t ^ fl.x[f];  // rows of a thread differ in the bits above t's
    const A v = (A)fl.v[f];
#pragma unroll
    for (int r = 0; r < RPT; ++r)
      if (FULL || t + r * kPauliThreads < rows) add(r, v, ldout(sx + (lx ^ (r * kPauliThreads))));
  }
  if constexpr (FULL) {
    for (int f = nlow; f < fl.n; ++f) {
      const VT* xo = xk + ((base + t) ^ fl.x[f]);  // flips below R are not here: rows follow
      const A v = (A)fl.v[f];
      Cx<A> xv[RPT];
      const uint32_t low = fl.x[f] & (R - 1);
#pragma unroll
      for (int r = 0; r < RPT; ++r)
        xv[r] = low < kPauliThreads ? ldv(xo + r * kPauliThreads)
                                    : ldv(xk + ((base + t + r * kPauliThreads) ^ fl.x[f]));
#pragma unroll
      for (int r = 0; r < RPT; ++r) add(r, v, xv[r]);
    }
  }
  for (int g = 0; g < pd.ngroup; ++g) {
    const uint32_t xm = __ldg(&pd.group[g].x);
    const int s0 = __ldg(&pd.group[g].s0), s1 = __ldg(&pd.group[g].s1);
    const bool empty = __ldg(&pd.group[g].empty) != 0;
    A cr[RPT], ci[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) cr[r] = ci[r] = 0;
    for (int q = s0; q < s1; ++q) {
      const uint32_t z = __ldg(&pd.str[q].z);
      const A vr = (A)__ldg(&pd.str[q].v.x), vi = (A)__ldg(&pd.str[q].v.y);
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const bool neg = __popc((base + t + r * kPauliThreads) & z) & 1;
        cr[r] += neg ? -vr : vr;
        if constexpr (CX) ci[r] += neg ? -vi : vi;
      }
    }
    auto take = [&](int r) {
      const uint32_t l = t + r * kPauliThreads;
      const Cx<A> xv = xm < R ? ldout(sx + (l ^ xm)) : ldv(xk + ((base + l) ^ xm));
      acc[r].r = fma_(cr[r], xv.r, acc[r].r);
      if constexpr (CX) {
        acc[r].r = fma_(ci[r], xv.i, acc[r].r);
        acc[r].i = fma_(-ci[r], xv.r, fma_(cr[r], xv.i, acc[r].i));
      }
    };
    if (empty) {  // no element, no read: an infinity or NaN there is not this row's
#pragma unroll
      for (int r = 0; r < RPT; ++r)
        if ((FULL || t + r * kPauliThreads < rows) && !(cr[r] == 0 && (!CX || ci[r] == 0))) take(r);
    } else {  // (a test per row would keep its gathers from being in flight together)
#pragma unroll
      for (int r = 0; r < RPT; ++r)
        if (FULL || t + r * kPauliThreads < rows) take(r);
    }
  }
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const uint32_t l = t + r * kPauliThreads;
    if (!FULL && l >= rows) continue;
    const A d = (A)pauli_diag(op, pd, L, mask, base + l);
    const Cx<A> xi = ldout(sx + l);
    Cx<A> out{fma_(d, xi.r, acc[r].r), (A)0};
    if constexpr (CX) out.i = fma_(d, xi.i, acc[r].i);
    VT* yo = yk + base + l;
    if (accumulate) {
      const Cx<A> o = ldout(yo);
      out.r += o.r;
      out.i += o.i;
    }
    stv(yo, out);
  }
}

template <class VT>
edk_status launch_pauli(const edk_operator* op, const void* x, void* y, int64_t nvec, int64_t ldx,
                        int64_t ldy, int accumulate, cudaStream_t st, const int* step,
                        const int* done) {
  const BasisDev& b = op->b->dev;
  const VT* X = static_cast<const VT*>(x);
  VT* Y = static_cast<VT*>(y);
  // eight rows a thread once that leaves two blocks for every SM (4,096
  // rows), two below: small spaces need the blocks more than the wide tile
  // (four for double complex, whose eight rows do not fit the registers)
  constexpr int W = sizeof(VT) == 16 ? 4 : 8;
  const bool wide = b.D >= (int64_t)b.sms * 4096;
  const int64_t R = kPauliThreads * (wide ? W : 2);
  int nlow = 0;  // flips in ascending order
  while (nlow < op->pauli_flips.n && op->pauli_flips.x[nlow] < R) ++nlow;
  for (int64_t k0 = 0; k0 < nvec; k0 += 65535) {
    const int64_t nk = std::min<int64_t>(nvec - k0, 65535);
    const dim3 grid((unsigned)((b.D + R - 1) / R), (unsigned)nk);
    auto go = [&](auto kern) {
      kern<<<grid, kPauliThreads, 0, st>>>(op->dev, op->pauli, op->pauli_flips, nlow, b.L,
                                           (uint32_t)b.maskL, b.D, X + k0 * ldx, Y + k0 * ldy, ldx,
                                           ldy, accumulate, step, done);
    };
    if (wide) go(k_apply_pauli<VT, W, true>);
    else if (b.D >= R) go(k_apply_pauli<VT, 2, true>);
    else go(k_apply_pauli<VT, 2, false>);
    EDK_TRY_CUDA(cudaGetLastError());
  }
  return EDK_OK;
}

}  // namespace

edk_status apply_pauli(const edk_operator* op, int dtype, const void* x, void* y, int64_t nvec,
                       int64_t ldx, int64_t ldy, int accumulate, cudaStream_t st, const int* step,
                       const int* done) {
  switch (dtype) {
    case EDK_F64: return launch_pauli<double>(op, x, y, nvec, ldx, ldy, accumulate, st, step, done);
    case EDK_C128: return launch_pauli<double2>(op, x, y, nvec, ldx, ldy, accumulate, st, step, done);
    case EDK_F32: return launch_pauli<float>(op, x, y, nvec, ldx, ldy, accumulate, st, step, done);
    case EDK_C64: return launch_pauli<float2>(op, x, y, nvec, ldx, ldy, accumulate, st, step, done);
  }
  set_error("apply: unknown dtype");
  return EDK_INVALID_ARG;
}

}  // namespace edk
