// edk_apply.cu — matrix-free H * x on the device.
//
// Reference semantics (src/Operator.jl:399-465): for every basis state j and
// every local term, each nonzero M[r, c] of the local column c = digits of j on
// the term's sites produces the target state s' (digits rewritten to r) and
//     H[pos, j] += M[r, c] * C(s') * R[pos] / R[j],    (C, pos) = index(b, s').
//
// Row-gather form (the default).  When every local term is Hermitian and the
// operator is invariant under the basis symmetries, H is Hermitian and
//     y[i] = sum_{nonzeros of column i}  conj(H[pos, i]) * x[pos],
// so one thread owns one output row: no atomics, no private copies, a
// deterministic summation order.  The column-scatter form (atomics) is kept
// for operators that are not Hermitian in the sector.
//
// Terms are compiled for the device into
//   * bond families: 2-site terms (i, i+d mod L) that share one 4x4 matrix,
//     evaluated on whole bit planes (X = s, Y = rotl(s, d), local column
//     c = 2X+Y), so the diagonal is four popcounts and the off-diagonal hits
//     are the set bits of one mask;
//   * generic terms: per-term local column, CSC list of XOR masks.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <memory>
#include <type_traits>

#include "edk_spmm.cuh"

namespace edk {

// y(:, k) (+)= H x(:, k); blockIdx.y = k.  TPR lanes share a row.
template <int BK, class S, class VT, bool GATHER, int TPR>
__global__ void __launch_bounds__(256) k_apply(BasisDev b, OpDev op, const VT* __restrict__ x,
                                               VT* __restrict__ y, int64_t ldx, int64_t ldy,
                                               int accumulate) {
  __shared__ uint32_t s_binom[(BK == BK_PROJ_RANK) ? 32 * 33 : 1];
  if constexpr (BK == BK_PROJ_RANK) {
    fill_binom32(s_binom);
    __syncthreads();
  }
  const VT* xk = x + (int64_t)blockIdx.y * ldx;
  VT* yk = y + (int64_t)blockIdx.y * ldy;
  constexpr int RPB = 256 / TPR;
  for (int64_t i0 = (int64_t)blockIdx.x * RPB; i0 < b.D; i0 += (int64_t)gridDim.x * RPB) {
    const int64_t i = i0 + threadIdx.x / TPR;
    if constexpr (TPR == 1) {
      if (i < b.D) gen_row<BK, S, VT, GATHER>(b, op, i, xk, yk, accumulate, s_binom);
    } else {
      gen_row<BK, S, VT, GATHER, TPR>(b, op, i < b.D ? i : b.D - 1, xk, yk, accumulate, s_binom,
                                      threadIdx.x % TPR, i < b.D);
    }
  }
}

// Lanes per row of the general gather kernel.  A row is a serial chain of
// lookups, so a small sector with one lane per row leaves most of the GPU
// idle: lanes share a row while the rows times the lanes still fit two rounds
// of the resident threads (2,048 per SM).  Symmetry groups, whose lookup is the
// longest, take sixteen or four lanes, the others eight.
// (k, p, z) group sector of L = 22, some 8,360 rows, real vector: 621 us with
// one lane per row and every group element stepped through the generators, 45
// us with eight lanes and rotations read off a doubled word, 22 us with sixteen
// lanes and rotations compared at the zero-run tops (runs_arg32).
template <int BK> constexpr int many_lanes() { return BK == BK_ABELIAN ? 16 : 8; }
template <int BK> constexpr int few_lanes() { return BK == BK_ABELIAN ? 4 : 1; }
bool lanes_fit(const BasisDev& b, int64_t rows, int lanes) {
  return rows * lanes <= (int64_t)2 * b.sms * 2048;
}

// Resident blocks per SM asked of the compiler: the rank-search kernels are
// latency bound and fit 32 registers (8 blocks of 256 threads fill every warp
// slot) for real and single-precision complex vectors, or single precision
// when the sector has a phase or a parity; double complex on the hashed kinds
// with a phase or a parity fits 48 (5 blocks instead of 4 at 56: 25 sites, 697
// blocks, 64 -> 58 us, and no second wave); the others keep the compiler's choice.
template <int BK, class VT>
constexpr int ff_min_blocks() {
  constexpr bool single = std::is_same<VT, float>::value || std::is_same<VT, float2>::value;
  if ((BK == BK_TRANS0_RANK && !std::is_same<VT, double2>::value) ||
      ((BK == BK_TRANS_RANK || BK == BK_TRANSPAR_RANK) && single))
    return 8;
  return (BK == BK_TRANS || BK == BK_TRANSPAR) && std::is_same<VT, double2>::value ? 5 : 1;
}

template <int BK, class VT, int TPS>
__global__ void __launch_bounds__(256, ff_min_blocks<BK, VT>())
    k_apply_ff(BasisDev b, OpDev op, FFParams ff,
                                                  const VT* __restrict__ x, VT* __restrict__ y,
                                                  int64_t ldx, int64_t ldy, int accumulate,
                                                  int64_t tile0) {
  ff_tile<BK, VT, TPS>(b, op, ff, (tile0 + blockIdx.x) * (256 / TPS),
                       x + (int64_t)blockIdx.y * ldx, y + (int64_t)blockIdx.y * ldy, accumulate);
}

namespace {

int apply_grid(int64_t D) {
  int64_t g = (D + 255) / 256;
  if (g < 1) g = 1;
  if (g > 148 * 64) g = 148 * 64;
  return (int)g;
}

template <class VT, int TPS>
edk_status launch_apply_ff(const BasisDev& b, const OpDev& op, const FFParams& ff, const void* x,
                           void* y, int64_t nvec, int64_t ldx, int64_t ldy, int accumulate,
                           cudaStream_t st, int64_t row0 = 0, int64_t row1 = -1) {
  const VT* X = static_cast<const VT*>(x);
  VT* Y = static_cast<VT*>(y);
  constexpr int RT = 256 / TPS;
  if (row1 < 0) row1 = b.D;
  const int64_t tile0 = row0 / RT, tile1 = (row1 + RT - 1) / RT;
  if (tile1 <= tile0) return EDK_OK;
  for (int64_t k0 = 0; k0 < nvec; k0 += 65535) {
    int64_t nk = std::min<int64_t>(nvec - k0, 65535);
    dim3 grid((unsigned)(tile1 - tile0), (unsigned)nk);
    const VT* Xk = X + k0 * ldx;
    VT* Yk = Y + k0 * ldy;
#define EDK_FF(BK)                                                                         \
  case BK:                                                                                 \
    k_apply_ff<BK, VT, TPS><<<grid, 256, 0, st>>>(b, op, ff, Xk, Yk, ldx, ldy, accumulate, \
                                                  tile0);                                     \
    break;
    const int kind = b.search != 2 ? b.bk
                     : (b.bk == BK_TRANS0 ? (int)BK_TRANS0_RANK
                        : (b.bk == BK_TRANS ? (int)BK_TRANS_RANK
                           : (b.bk == BK_TRANSPAR ? (int)BK_TRANSPAR_RANK : b.bk)));
    switch (kind) {
      EDK_FF(BK_TENSOR)
      EDK_FF(BK_PROJ_RANK)
      EDK_FF(BK_PROJ_HASH)
      EDK_FF(BK_TRANS0)
      EDK_FF(BK_TRANS0_RANK)
      EDK_FF(BK_TRANS_RANK)
      EDK_FF(BK_TRANSPAR_RANK)
      EDK_FF(BK_TRANS)
      EDK_FF(BK_TRANSPAR)
      default:
        set_error("apply: fast path not available for this basis");
        return EDK_INVALID_ARG;
    }
#undef EDK_FF
    EDK_TRY_CUDA(cudaGetLastError());
  }
  return EDK_OK;
}

template <class VT, bool GATHER>
edk_status launch_apply(const BasisDev& b, const OpDev& op, const void* x, void* y, int64_t nvec,
                        int64_t ldx, int64_t ldy, int accumulate, cudaStream_t st) {
  const VT* X = static_cast<const VT*>(x);
  VT* Y = static_cast<VT*>(y);
  bool wide = b.L > 32;
  for (int64_t k0 = 0; k0 < nvec; k0 += 65535) {
    int64_t nk = std::min<int64_t>(nvec - k0, 65535);
    const VT* Xk = X + k0 * ldx;
    VT* Yk = Y + k0 * ldy;
    const int64_t rows = b.D * nk;
#define EDK_APPLY_T(BK, S, T)                                                                  \
  k_apply<BK, S, VT, GATHER, GATHER ? (T) : 1>                                                 \
      <<<dim3(apply_grid(b.D * (GATHER ? (T) : 1)), (unsigned)nk), 256, 0, st>>>(              \
          b, op, Xk, Yk, ldx, ldy, accumulate);
#define EDK_APPLY_S(BK, S)                                                                     \
  if (GATHER && lanes_fit(b, rows, many_lanes<BK>())) { EDK_APPLY_T(BK, S, many_lanes<BK>()) }    \
  else if (GATHER && lanes_fit(b, rows, few_lanes<BK>())) { EDK_APPLY_T(BK, S, few_lanes<BK>()) } \
  else { EDK_APPLY_T(BK, S, 1) }
#define EDK_APPLY(BK)                       \
  case BK:                                  \
    if (wide) { EDK_APPLY_S(BK, uint64_t) } \
    else { EDK_APPLY_S(BK, uint32_t) }      \
    break;
    switch (b.bk) {
      EDK_APPLY(BK_TENSOR)
      EDK_APPLY(BK_PROJ_RANK)
      EDK_APPLY(BK_PROJ_HASH)
      EDK_APPLY(BK_TRANS0)
      EDK_APPLY(BK_TRANS)
      EDK_APPLY(BK_TRANSPAR)
      EDK_APPLY(BK_ABELIAN)
      default:
        set_error("apply: unknown basis lookup kind");
        return EDK_INVALID_ARG;
    }
#undef EDK_APPLY
#undef EDK_APPLY_S
#undef EDK_APPLY_T
    EDK_TRY_CUDA(cudaGetLastError());
  }
  return EDK_OK;
}

size_t dtype_size(int dtype) {
  switch (dtype) {
    case EDK_F64: return 8;
    case EDK_C128: return 16;
    case EDK_F32: return 4;
    case EDK_C64: return 8;
  }
  return 0;
}

}  // namespace

namespace {

// column-major (ld) <-> row-major (p) blocks through 32 x 32 shared-memory
// tiles, coalesced on both sides; the reverse direction can accumulate
template <class VT>
__global__ void k_cols_to_rows_t(const VT* __restrict__ src, int64_t ld, int64_t D, int p,
                                 VT* __restrict__ dst) {
  __shared__ VT tile[32][33];
  const int64_t i0 = (int64_t)blockIdx.x * 32;
  const int c0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int64_t i = i0 + threadIdx.x;
    const int c = c0 + k;
    if (i < D && c < p) tile[k][threadIdx.x] = src[(int64_t)c * ld + i];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int64_t i = i0 + k;
    const int c = c0 + threadIdx.x;
    if (i < D && c < p) dst[i * p + c] = tile[threadIdx.x][k];
  }
}

template <class VT>
__global__ void k_rows_to_cols_t(const VT* __restrict__ src, int64_t D, int p,
                                 VT* __restrict__ dst, int64_t ld, int accumulate) {
  using A = typename VTraits<VT>::A;
  __shared__ VT tile[32][33];
  const int64_t i0 = (int64_t)blockIdx.x * 32;
  const int c0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int64_t i = i0 + k;
    const int c = c0 + threadIdx.x;
    if (i < D && c < p) tile[k][threadIdx.x] = src[i * p + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int64_t i = i0 + threadIdx.x;
    const int c = c0 + k;
    if (i < D && c < p) {
      VT* d = dst + (int64_t)c * ld + i;
      if (accumulate) {
        const Cx<A> a = ldout(d), v = ldout(&tile[threadIdx.x][k]);
        stv(d, Cx<A>{a.r + v.r, a.i + v.i});
      } else {
        *d = tile[threadIdx.x][k];
      }
    }
  }
}

template <class VT>
edk_status apply_block_t(edk_operator* op, const void* x, void* y, int64_t nvec, int64_t ldx,
                         int64_t ldy, int accumulate, cudaStream_t st, int bk, int64_t slots) {
  const int64_t D = op->b->D;
  const int pmax = 64;
  const int pc0 = (int)std::min<int64_t>(nvec, pmax);
  const size_t need = (size_t)D * pc0 * sizeof(VT);
  if (op->bx.bytes < need) EDK_RETURN_IF(op->bx.alloc(need));
  if (op->by.bytes < need) EDK_RETURN_IF(op->by.alloc(need));
  VT* bx = op->bx.as<VT>();
  VT* by = op->by.as<VT>();
  const VT* X = static_cast<const VT*>(x);
  VT* Y = static_cast<VT*>(y);
  for (int64_t k0 = 0; k0 < nvec; k0 += pmax) {
    const int pc = (int)std::min<int64_t>(nvec - k0, pmax);
    const dim3 tb(32, 8), tg((unsigned)((D + 31) / 32), (unsigned)((pc + 31) / 32));
    k_cols_to_rows_t<VT><<<tg, tb, 0, st>>>(X + k0 * ldx, ldx, D, pc, bx);
    EDK_TRY_CUDA(cudaGetLastError());
    EDK_RETURN_IF(launch_spmm<VT>(op->bop.as<SpmmOp>(), 1, bk, slots, D, pc, bx, by, 0, st));
    k_rows_to_cols_t<VT><<<tg, tb, 0, st>>>(by, D, pc, Y + k0 * ldy, ldy, accumulate);
    EDK_TRY_CUDA(cudaGetLastError());
  }
  return EDK_OK;
}

// Several right-hand sides on the row-gather paths: one SpMM over row-major
// copies of at most 64 columns at a time, so every hit is located once for
// all of them (false: not applicable, the caller uses the column kernels).
bool block_apply_ok(const edk_operator* op, int64_t nvec) {
  return nvec >= 4 && op->gather && (op->sell_ok || (op->ff_ok && op->use_ff && op->b->dev.L <= 32));
}

edk_status apply_block(edk_operator* op, int dtype, const void* x, void* y, int64_t nvec,
                       int64_t ldx, int64_t ldy, int accumulate, cudaStream_t st) {
  SpmmOp h;
  int bk;
  int64_t slots;
  spmm_describe(op, h, bk, slots);
  std::vector<unsigned char> bytes(sizeof(SpmmOp));
  std::memcpy(bytes.data(), &h, sizeof(SpmmOp));
  if (op->bop_host != bytes || !op->bop.p) {
    if (!op->bop.p) EDK_RETURN_IF(op->bop.alloc(sizeof(SpmmOp)));
    op->bop_host = bytes;
    EDK_TRY_CUDA(cudaMemcpyAsync(op->bop.p, op->bop_host.data(), sizeof(SpmmOp),
                                 cudaMemcpyHostToDevice, st));
  }
  switch (dtype) {
    case EDK_F64: return apply_block_t<double>(op, x, y, nvec, ldx, ldy, accumulate, st, bk, slots);
    case EDK_C128: return apply_block_t<double2>(op, x, y, nvec, ldx, ldy, accumulate, st, bk, slots);
    case EDK_F32: return apply_block_t<float>(op, x, y, nvec, ldx, ldy, accumulate, st, bk, slots);
    case EDK_C64: return apply_block_t<float2>(op, x, y, nvec, ldx, ldy, accumulate, st, bk, slots);
  }
  set_error("apply: unknown dtype");
  return EDK_INVALID_ARG;
}

}  // namespace

edk_status apply_device(edk_operator* op, int dtype, const void* x, void* y, int64_t nvec,
                        int64_t ldx, int64_t ldy, int accumulate, cudaStream_t st) {
  const BasisDev& b = op->b->dev;
  if (nvec <= 0 || b.D == 0) return EDK_OK;
  EDK_RETURN_IF(check_basis_dev(b));
  if (!op->gather && !accumulate) {
    // column scatter accumulates with atomics: start from zero
    size_t es = dtype_size(dtype);
    EDK_TRY_CUDA(cudaMemset2DAsync(y, ldy * es, 0, b.D * es, nvec, st));
  }
  bool sc = !op->gather;
  // automatic choice: the SpMM for a block of columns unless the operator is
  // materialised or runs on a row plan (both stream one column faster than
  // the SpMM locates hits once for all of them)
  if (block_apply_ok(op, nvec) &&
      (op->use_block > 0 || (op->use_block < 0 && !op->sell_ok && !plan_applies(op))))
    return apply_block(op, dtype, x, y, nvec, ldx, ldy, accumulate, st);
  if (op->sell_ok && !sc) return apply_sell(op, dtype, x, y, nvec, ldx, ldy, accumulate, st);
  if (op->ff_ok && !sc && op->use_ff) {
    if (plan_applies(op)) return apply_plan(op, dtype, x, y, nvec, ldx, ldy, accumulate, st, 0, -1);
    const FFParams& ff = *reinterpret_cast<const FFParams*>(op->ff_params.data());
#define EDK_FF_TPS(VT)                                                                          \
  switch (op->tps) {                                                                            \
    case 2: return launch_apply_ff<VT, 2>(b, op->dev, ff, x, y, nvec, ldx, ldy, accumulate, st); \
    case 4: return launch_apply_ff<VT, 4>(b, op->dev, ff, x, y, nvec, ldx, ldy, accumulate, st); \
    default: return launch_apply_ff<VT, 1>(b, op->dev, ff, x, y, nvec, ldx, ldy, accumulate, st); \
  }
    switch (dtype) {
      case EDK_F64: EDK_FF_TPS(double)
      case EDK_C128: EDK_FF_TPS(double2)
      case EDK_F32: EDK_FF_TPS(float)
      case EDK_C64: EDK_FF_TPS(float2)
    }
#undef EDK_FF_TPS
  }
  if (op->pauli_ok && op->use_ff) return apply_pauli(op, dtype, x, y, nvec, ldx, ldy, accumulate, st);
  switch (dtype) {
    case EDK_F64:
      return sc ? launch_apply<double, false>(b, op->dev, x, y, nvec, ldx, ldy, 1, st)
                : launch_apply<double, true>(b, op->dev, x, y, nvec, ldx, ldy, accumulate, st);
    case EDK_C128:
      return sc ? launch_apply<double2, false>(b, op->dev, x, y, nvec, ldx, ldy, 1, st)
                : launch_apply<double2, true>(b, op->dev, x, y, nvec, ldx, ldy, accumulate, st);
    case EDK_F32:
      return sc ? launch_apply<float, false>(b, op->dev, x, y, nvec, ldx, ldy, 1, st)
                : launch_apply<float, true>(b, op->dev, x, y, nvec, ldx, ldy, accumulate, st);
    case EDK_C64:
      return sc ? launch_apply<float2, false>(b, op->dev, x, y, nvec, ldx, ldy, 1, st)
                : launch_apply<float2, true>(b, op->dev, x, y, nvec, ldx, ldy, accumulate, st);
  }
  set_error("apply: unknown dtype");
  return EDK_INVALID_ARG;
}

// ---------------------------------------------------------------------------
// Operator compilation (host)
// ---------------------------------------------------------------------------
namespace {

struct HostTerm {
  std::vector<int> sites;           // 1-based
  int dim = 0;
  std::vector<double> re, im;       // dense, row-major M[r*dim + c]
};

double term_scale(const HostTerm& t) {
  double m = 0;
  for (size_t q = 0; q < t.re.size(); ++q) m = std::max(m, std::hypot(t.re[q], t.im[q]));
  return m;
}

bool term_hermitian(const HostTerm& t) {
  double tol = 1e-12 * std::max(1.0, term_scale(t));
  for (int r = 0; r < t.dim; ++r)
    for (int c = 0; c < t.dim; ++c) {
      double dr = t.re[r * t.dim + c] - t.re[c * t.dim + r];
      double di = t.im[r * t.dim + c] + t.im[c * t.dim + r];
      if (std::hypot(dr, di) > tol) return false;
    }
  return true;
}

// Canonical form: sites sorted ascending, tensor factors permuted to match.
HostTerm canonical(const HostTerm& t) {
  int ns = (int)t.sites.size();
  std::vector<int> order(ns);
  for (int k = 0; k < ns; ++k) order[k] = k;
  std::sort(order.begin(), order.end(), [&](int a, int b) { return t.sites[a] < t.sites[b]; });
  HostTerm o;
  o.dim = t.dim;
  o.sites.resize(ns);
  for (int k = 0; k < ns; ++k) o.sites[k] = t.sites[order[k]];
  o.re.assign(t.re.size(), 0.0);
  o.im.assign(t.im.size(), 0.0);
  // new local index bit (ns-1-k) holds old factor order[k] whose bit is (ns-1-order[k])
  auto remap = [&](int idx) {
    int out = 0;
    for (int k = 0; k < ns; ++k) {
      int bit = (idx >> (ns - 1 - order[k])) & 1;
      out |= bit << (ns - 1 - k);
    }
    return out;
  };
  for (int r = 0; r < t.dim; ++r)
    for (int c = 0; c < t.dim; ++c) {
      int nr = remap(r), nc = remap(c);
      o.re[nr * t.dim + nc] = t.re[r * t.dim + c];
      o.im[nr * t.dim + nc] = t.im[r * t.dim + c];
    }
  return o;
}

using TermMap = std::map<std::vector<int>, std::pair<std::vector<double>, std::vector<double>>>;

void add_term(TermMap& m, const HostTerm& t) {
  HostTerm c = canonical(t);
  auto it = m.find(c.sites);
  if (it == m.end()) {
    m[c.sites] = {c.re, c.im};
  } else {
    for (size_t q = 0; q < c.re.size(); ++q) {
      it->second.first[q] += c.re[q];
      it->second.second[q] += c.im[q];
    }
  }
}

// Is sum_t M_t invariant under (site permutation perm, inversion flags inv)?
bool invariant(const std::vector<HostTerm>& terms, const std::vector<int>& perm,
               const std::vector<uint8_t>& inv) {
  TermMap a, b;
  double scale = 0;
  for (auto& t : terms) {
    add_term(a, t);
    scale = std::max(scale, term_scale(t));
    HostTerm g;
    g.dim = t.dim;
    int ns = (int)t.sites.size();
    g.sites.resize(ns);
    int fmask = 0;
    for (int k = 0; k < ns; ++k) {
      g.sites[k] = perm[t.sites[k] - 1];
      if (inv[g.sites[k] - 1]) fmask |= 1 << (ns - 1 - k);
    }
    g.re.resize(t.re.size());
    g.im.resize(t.im.size());
    for (int r = 0; r < t.dim; ++r)
      for (int c = 0; c < t.dim; ++c) {
        g.re[(r ^ fmask) * t.dim + (c ^ fmask)] = t.re[r * t.dim + c];
        g.im[(r ^ fmask) * t.dim + (c ^ fmask)] = t.im[r * t.dim + c];
      }
    add_term(b, g);
  }
  double tol = 1e-12 * std::max(1.0, scale);
  auto cmp = [&](const TermMap& x, const TermMap& y) {
    for (auto& kv : x) {
      auto it = y.find(kv.first);
      for (size_t q = 0; q < kv.second.first.size(); ++q) {
        double yr = (it == y.end()) ? 0.0 : it->second.first[q];
        double yi = (it == y.end()) ? 0.0 : it->second.second[q];
        if (std::hypot(kv.second.first[q] - yr, kv.second.second[q] - yi) > tol) return false;
      }
    }
    return true;
  };
  return cmp(a, b) && cmp(b, a);
}

uint32_t site_mask(const HostTerm& h, int L, int c) {
  const int ns = (int)h.sites.size();
  uint32_t m = 0;
  for (int k = 0; k < ns; ++k)
    if ((c >> (ns - 1 - k)) & 1) m |= 1u << (L - h.sites[k]);
  return m;
}

// True when the strings of every flip mask give the matrix elements back: to a few
// roundings of the entries they are made of, in both widths and in the kernel's order
// of summation, and exactly zero where no term has an entry (the kernel reads the
// vector at nonzeros only, as the row kernel does, so an infinity or NaN stays in
// the rows that have an element with it).  An entry of at least a hundredth of the
// largest one beside it may carry that one's rounding.  (1.7, 0.3) as 1.0 +- 0.7
// passes; 1e10 and 1e-10 in one matrix, or three couplings that cancel only up to
// rounding, do not.  `empty`: the flip masks that have no entry for some pattern.
using PauliSum = std::map<std::pair<uint32_t, uint32_t>, std::pair<double, double>>;
bool strings_give_entries(const std::vector<HostTerm>& terms, const std::vector<char>& in_family,
                          int L, const PauliSum& sum, std::set<uint32_t>& empty) {
  constexpr int kBits = 10;  // patterns are enumerated over at most 2^10
  constexpr double e64 = 2.220446049250313e-16, e32 = 1.1920928955078125e-07;
  struct Part { const HostTerm* t; int x; };
  std::map<uint32_t, std::vector<Part>> parts;
  for (size_t q = 0; q < terms.size(); ++q) {
    const HostTerm& h = terms[q];
    for (int x = 0; x < h.dim; ++x) {
      bool any = false;
      for (int c = 0; c < h.dim && !any; ++c) {
        const double re = h.re[(c ^ x) * h.dim + c], im = h.im[(c ^ x) * h.dim + c];
        any = !(re == 0.0 && im == 0.0);
      }
      if (any && !(x == 0 && in_family[q])) parts[site_mask(h, L, x)].push_back({&h, x});
    }
  }
  // scale: the entries at this pattern, big: the largest over all patterns
  auto near = [](double got, double want, double scale, double big, double eps) {
    if (scale == 0.0) return got == 0.0;
    if (scale >= 0.01 * big) scale = std::max(scale, 0.25 * big);
    return std::fabs(got - want) <= 8.0 * eps * scale;
  };
  auto walsh = [](const HostTerm& h, int x, int z, double& vr, double& vi) {
    vr = vi = 0.0;
    for (int c = 0; c < h.dim; ++c) {
      const double sg = (__builtin_popcount(c & z) & 1) ? -1.0 : 1.0;
      vr += sg * h.re[(c ^ x) * h.dim + c];
      vi += sg * h.im[(c ^ x) * h.dim + c];
    }
    vr /= h.dim;
    vi /= h.dim;
  };
  for (const auto& kv : parts) {
    uint32_t sites = 0;
    for (const Part& p : kv.second) sites |= site_mask(*p.t, L, p.t->dim - 1);
    if (kv.first == 0 || __builtin_popcount(sites) > kBits) {
      // term by term: the diagonal (every row multiplies it, so a rounding beside a
      // zero entry spreads nothing), and flips that reach many sites, where each term
      // has to be one string (an entry in every column, so no pattern is empty)
      for (const Part& p : kv.second) {
        const HostTerm& h = *p.t;
        std::vector<double> vr(h.dim), vi(h.dim);
        int strings = 0;
        for (int z = 0; z < h.dim; ++z) {
          walsh(h, p.x, z, vr[z], vi[z]);
          strings += vr[z] != 0.0 || vi[z] != 0.0;
        }
        if (kv.first != 0 && strings != 1) return false;
        double big = 0.0;
        for (int c = 0; c < h.dim; ++c)
          big = std::max(big, std::fabs(h.re[(c ^ p.x) * h.dim + c]) +
                                  std::fabs(h.im[(c ^ p.x) * h.dim + c]));
        for (int c = 0; c < h.dim; ++c) {
          double re = 0.0, im = 0.0;
          for (int z = 0; z < h.dim; ++z) {
            const double sg = (__builtin_popcount(c & z) & 1) ? -1.0 : 1.0;
            re += sg * vr[z];
            im += sg * vi[z];
          }
          const double er = h.re[(c ^ p.x) * h.dim + c], ei = h.im[(c ^ p.x) * h.dim + c];
          // (a zero on the diagonal may carry a rounding, and so may what is near it)
          const double s = kv.first == 0 ? big : std::fabs(er) + std::fabs(ei);
          if (kv.first == 0 && er != 0.0 && std::fabs(er) < 1e-3 * big) return false;
          if (!near(re, er, s, big, e64) || !near(im, ei, s, big, e64)) return false;
        }
      }
      continue;
    }
    const auto first = sum.lower_bound({kv.first, 0u}), last = sum.upper_bound({kv.first, ~0u});
    auto entries = [&](uint32_t pat, double& re, double& im) {  // the terms' sum; its size
      double s = 0.0;
      re = im = 0.0;
      for (const Part& p : kv.second) {
        const HostTerm& h = *p.t;
        int c = 0;
        for (int v : h.sites) c = 2 * c + (int)((pat >> (L - v)) & 1u);
        const double er = h.re[(c ^ p.x) * h.dim + c], ei = h.im[(c ^ p.x) * h.dim + c];
        re += er;
        im += ei;
        s += std::fabs(er) + std::fabs(ei);
      }
      return s;
    };
    double re, im, big = 0.0;
    uint32_t pat = 0;  // the patterns of the sites, in ascending order
    do {
      const double s = entries(pat, re, im);
      big = std::max(big, s);
      if (s == 0.0) empty.insert(kv.first);
      pat = (pat - sites) & sites;
    } while (pat != 0);
    do {
      const double s = entries(pat, re, im);
      double dr = 0.0, di = 0.0;
      float fr = 0.f, fi = 0.f;
      for (auto it = first; it != last; ++it) {
        const bool neg = __builtin_popcount(pat & it->first.second) & 1;
        const double vr = it->second.first, vi = it->second.second;
        dr += neg ? -vr : vr;
        di += neg ? -vi : vi;
        fr += neg ? -(float)vr : (float)vr;
        fi += neg ? -(float)vi : (float)vi;
      }
      if (!near(dr, re, s, big, e64) || !near(di, im, s, big, e64) || !near(fr, re, s, big, e32) ||
          !near(fi, im, s, big, e32))
        return false;
      pat = (pat - sites) & sites;
    } while (pat != 0);
  }
  return true;
}

// True when the strings cost a row less than the terms.  Both kernels are bound by
// instructions, so the rule counts them, in units of 0.1 us fitted to measured products.
// Large spaces, for 2^20 rows (FP64, 20 sites, launch and host taken off):
//   strings: 0.4 a plain flip, 0.55 a string, 0.6 a flip mask of several strings;
//   terms: 2.8 a term and 0.9 an off-diagonal entry of its columns (their mean);
//   bond families: 3.8 an off-diagonal entry; diagonals are popcounts in both.
// Strings / terms in us a product there: 20 x fields 26 / 87, of x and z 37 / 89; 19
// projected flips of two sites 52 / 65, eight 35 / 35, 18 of three 64 / 72, eight 40 / 41,
// 17 of four 90 / 67; dense two-site terms 28 / 23 (one) and 124 / 114 (19), three-site 50
// / 28 and 190 / 86 (eight), four-site 128 / 34 and 217 / 49 (two).
// Small spaces, whose rows eight lanes share (16 sites): terms 3 once, 0.2 a term or
// entry; strings 0.05 a plain flip, 0.16 a string, 0.4 a flip mask of several.  16
// fields 21 / 26, complex 31 / 29; 15 projected flips of two sites 30 / 25, 14 of three
// 28 / 26; dense two-site terms 23 / 24 (one) and 41 / 32 (15), four-site 42 / 29 (one).
bool strings_win(const std::vector<HostTerm>& terms, const std::vector<char>& in_family,
                 const BasisDev& b, const PauliFlips& flips, size_t groups, size_t strings) {
  const bool small = lanes_fit(b, b.D, many_lanes<BK_TENSOR>());
  double rows = small ? 30.0 : 0.0;
  for (size_t t = 0; t < terms.size(); ++t) {
    const HostTerm& h = terms[t];
    int off = 0;
    for (int r = 0; r < h.dim; ++r)
      for (int c = 0; c < h.dim; ++c)
        off += r != c && !(h.re[r * h.dim + c] == 0.0 && h.im[r * h.dim + c] == 0.0);
    const double entries = (double)off / h.dim;
    if (small) rows += (in_family[t] ? 0.0 : 2.0) + 2.0 * entries;
    else rows += in_family[t] ? 38.0 * entries : 28.0 + 9.0 * entries;
  }
  return (small ? 0.5 * flips.n + 1.6 * strings + 4.0 * groups
                : 4.0 * flips.n + 5.5 * strings + 6.0 * groups) <= rows;
}

// Pauli strings of the terms' off-diagonal parts, grouped by flip mask, and of the
// diagonals of the terms outside the bond families.  False when there are more than
// kPauliMax (tables and host time), they do not give the matrix elements back, or the
// terms cost less.
constexpr size_t kPauliMax = 512;
bool pauli_strings(const std::vector<HostTerm>& terms, const std::vector<char>& in_family,
                   const BasisDev& b, PauliFlips& flips, std::vector<PauliGroup>& group,
                   std::vector<PauliStr>& str, std::vector<PauliStr>& diag) {
  const int L = b.L;
  PauliSum sum;
  for (size_t t = 0; t < terms.size(); ++t) {
    const HostTerm& h = terms[t];
    const int ns = (int)h.sites.size();
    if (ns > 4) return false;
    auto mask = [&](int c) { return site_mask(h, L, c); };
    for (int x = 0; x < h.dim; ++x) {
      if (x == 0 && in_family[t]) continue;
      for (int z = 0; z < h.dim; ++z) {
        double vr = 0.0, vi = 0.0;
        for (int c = 0; c < h.dim; ++c) {
          const double sg = (__builtin_popcount(c & z) & 1) ? -1.0 : 1.0;
          vr += sg * h.re[(c ^ x) * h.dim + c];
          vi += sg * h.im[(c ^ x) * h.dim + c];
        }
        if (vr == 0.0 && vi == 0.0) continue;
        auto& v = sum[{mask(x), mask(z)}];
        v.first += vr / h.dim;
        v.second += vi / h.dim;
      }
    }
    if (sum.size() > kPauliMax) return false;
  }
  std::set<uint32_t> empty;
  if (!strings_give_entries(terms, in_family, L, sum, empty)) return false;
  std::map<uint32_t, int> per_mask;
  for (auto it = sum.begin(); it != sum.end();)
    if (it->second.first == 0.0 && it->second.second == 0.0) it = sum.erase(it);
    else ++per_mask[(it++)->first.first];
  flips.n = 0;
  for (auto& kv : sum) {
    const uint32_t x = kv.first.first, z = kv.first.second;
    PauliStr p{};
    p.v = make_double2(kv.second.first, kv.second.second);
    p.z = z;
    if (x == 0) {
      diag.push_back(p);
    } else if (z == 0 && per_mask[x] == 1 && p.v.y == 0.0 && flips.n < kPauliFlips) {
      flips.x[flips.n] = x;
      flips.v[flips.n++] = p.v.x;
    } else {
      if (group.empty() || group.back().x != x)
        group.push_back(PauliGroup{x, (int)str.size(), (int)str.size(), (int)empty.count(x)});
      str.push_back(p);
      group.back().s1 = (int)str.size();
    }
  }
  return strings_win(terms, in_family, b, flips, group.size(), str.size() + diag.size());
}

}  // namespace
}  // namespace edk

using namespace edk;

edk_operator::~edk_operator() {
  handles_unregister(handles);
  p_slab.reset();
  for (cudaEvent_t e : cevents) cudaEventDestroy(e);
  if (cstream) cudaStreamDestroy(cstream);
  if (stream) cudaStreamDestroy(stream);
}

namespace edk {

bool rows_apply_ok(const edk_operator* op) {
  if (!op->gather) return false;
  return op->sell_ok || (op->ff_ok && op->use_ff);
}

edk_status apply_rows(edk_operator* op, int dtype, const void* x, void* y, int64_t row0,
                      int64_t row1, int accumulate, cudaStream_t st) {
  const BasisDev& b = op->b->dev;
  EDK_RETURN_IF(check_basis_dev(b));
  if (op->sell_ok) return apply_sell_rows(op, dtype, x, y, row0, row1, accumulate, st);
  if (plan_applies(op)) return apply_plan(op, dtype, x, y, 1, b.D, b.D, accumulate, st, row0, row1);
  const FFParams& ff = *reinterpret_cast<const FFParams*>(op->ff_params.data());
  const int64_t D = b.D;
#define EDK_FF_ROWS(VT)                                                                      \
  switch (op->tps) {                                                                         \
    case 2: return launch_apply_ff<VT, 2>(b, op->dev, ff, x, y, 1, D, D, accumulate, st,     \
                                          row0, row1);                                       \
    case 4: return launch_apply_ff<VT, 4>(b, op->dev, ff, x, y, 1, D, D, accumulate, st,     \
                                          row0, row1);                                       \
    default: return launch_apply_ff<VT, 1>(b, op->dev, ff, x, y, 1, D, D, accumulate, st,    \
                                           row0, row1);                                      \
  }
  switch (dtype) {
    case EDK_F64: EDK_FF_ROWS(double)
    case EDK_C128: EDK_FF_ROWS(double2)
    case EDK_F32: EDK_FF_ROWS(float)
    case EDK_C64: EDK_FF_ROWS(float2)
  }
#undef EDK_FF_ROWS
  set_error("apply: unknown dtype");
  return EDK_INVALID_ARG;
}

}  // namespace edk

extern "C" edk_status edk_operator_create(edk_basis* b, int32_t nterms, const int32_t* nsites,
                                          const int32_t* sites, const int64_t* nnz,
                                          const int64_t* colptr, const int64_t* rowval,
                                          const double* nzval, edk_operator** out) {
  EDK_CHECK_ARG(out != nullptr, "edk_operator_create: out is NULL");
  *out = nullptr;
  EDK_CHECK_ARG(b != nullptr, "edk_operator_create: basis is NULL");
  EDK_CHECK_ARG(nterms >= 0, "edk_operator_create: nterms < 0");
  EDK_CHECK_ARG(nterms == 0 || (nsites && sites && nnz && colptr && rowval && nzval),
                "edk_operator_create: NULL term array");
  const int L = b->L;
  std::vector<HostTerm> terms;
  size_t so = 0, co = 0, no = 0;
  for (int t = 0; t < nterms; ++t) {
    int ns = nsites[t];
    EDK_CHECK_ARG(ns >= 1 && ns <= 8, "edk_operator_create: a term must act on 1..8 sites");
    HostTerm h;
    h.sites.assign(sites + so, sites + so + ns);
    so += ns;
    std::vector<int> seen(L + 1, 0);
    for (int s : h.sites) {
      EDK_CHECK_ARG(s >= 1 && s <= L, "edk_operator_create: site outside 1:L");
      EDK_CHECK_ARG(!seen[s], "edk_operator_create: repeated site in one term");
      seen[s] = 1;
    }
    h.dim = 1 << ns;
    h.re.assign(h.dim * h.dim, 0.0);
    h.im.assign(h.dim * h.dim, 0.0);
    int64_t nz = nnz[t];
    EDK_CHECK_ARG(nz >= 0, "edk_operator_create: nnz < 0");
    for (int c = 0; c < h.dim; ++c) {
      int64_t q0 = colptr[co + c], q1 = colptr[co + c + 1];
      EDK_CHECK_ARG(q0 >= 1 && q1 >= q0 && q1 - 1 <= nz, "edk_operator_create: bad colptr");
      for (int64_t q = q0; q < q1; ++q) {
        int64_t r = rowval[no + q - 1];
        EDK_CHECK_ARG(r >= 1 && r <= h.dim, "edk_operator_create: bad rowval");
        h.re[(r - 1) * h.dim + c] += nzval[2 * (no + q - 1)];
        h.im[(r - 1) * h.dim + c] += nzval[2 * (no + q - 1) + 1];
      }
    }
    co += h.dim + 1;
    no += nz;
    terms.push_back(std::move(h));
  }
  auto* op = new edk_operator;
  std::unique_ptr<edk_operator> guard(op);
  op->b = b;
  // properties
  bool cplx = b->phase_complex;
  for (auto& t : terms)
    for (double v : t.im) cplx |= v != 0.0;
  bool herm = true;
  for (auto& t : terms) herm &= term_hermitian(t);
  if (herm && b->kind != EDK_TENSOR && b->kind != EDK_PROJECTED) {
    std::vector<uint8_t> noinv(L, 0);
    if (b->kind == EDK_TRANSLATIONAL || b->kind == EDK_TRANSPARITY) {
      std::vector<int> tr(L);
      for (int i = 1; i <= L; ++i) tr[i - 1] = (i - 1 + b->A) % L + 1;
      herm &= invariant(terms, tr, noinv);
      if (b->kind == EDK_TRANSPARITY) {
        std::vector<int> rv(L);
        for (int i = 1; i <= L; ++i) rv[i - 1] = L - i + 1;
        herm &= invariant(terms, rv, noinv);
      }
    } else {
      for (size_t g = 0; g < b->gen_perm.size(); ++g)
        herm &= invariant(terms, b->gen_perm[g], b->gen_inv[g]);
    }
  }
  op->gather = herm;
  op->is_complex = cplx;
  if (const char* e = std::getenv("EDK_DISABLE_FAST")) op->use_ff = !(e[0] == '1');
  if (const char* e = std::getenv("EDK_DISABLE_PLAN")) op->use_plan = !(e[0] == '1');
  // families of 2-site terms with one shared matrix
  std::map<std::pair<int, std::vector<double>>, std::vector<int>> groups;
  for (size_t t = 0; t < terms.size(); ++t) {
    if (terms[t].sites.size() != 2) continue;
    int d = ((terms[t].sites[1] - terms[t].sites[0]) % L + L) % L;
    std::vector<double> key(terms[t].re);
    key.insert(key.end(), terms[t].im.begin(), terms[t].im.end());
    groups[{d, key}].push_back((int)t);
  }
  std::vector<char> in_family(terms.size(), 0);
  std::vector<FamDev> fams;
  for (auto& kv : groups) {
    if (kv.second.size() < 3) continue;
    FamDev F{};
    F.d = kv.first.first;
    const HostTerm& t0 = terms[kv.second[0]];
    for (int t : kv.second) {
      F.valid |= 1ull << (L - terms[t].sites[0]);
      in_family[t] = 1;
    }
    for (int c = 0; c < 4; ++c) {
      F.dval[c] = make_double2(t0.re[c * 4 + c], t0.im[c * 4 + c]);
      int n = 0;
      for (int r = 0; r < 4; ++r) {
        if (r == c) continue;
        double vr = t0.re[r * 4 + c], vi = t0.im[r * 4 + c];
        if (vr == 0.0 && vi == 0.0) continue;
        F.xr[c][n] = c ^ r;
        F.val[c][n] = make_double2(vr, vi);
        ++n;
      }
      F.nnz[c] = n;
    }
    fams.push_back(F);
  }
  std::vector<TermDev> tds;
  std::vector<int> cp;
  std::vector<uint64_t> xm;
  std::vector<double2> vals, dvals;
  for (size_t t = 0; t < terms.size(); ++t) {
    if (in_family[t]) continue;
    const HostTerm& h = terms[t];
    TermDev td{};
    int ns = (int)h.sites.size();
    td.nsites = ns;
    for (int k = 0; k < ns; ++k) td.bitpos[k] = L - h.sites[k];
    td.col_off = (int)cp.size();
    td.diag_off = (int)dvals.size();
    for (int c = 0; c < h.dim; ++c) {
      cp.push_back((int)xm.size());
      dvals.push_back(make_double2(h.re[c * h.dim + c], h.im[c * h.dim + c]));
      for (int r = 0; r < h.dim; ++r) {
        if (r == c) continue;
        double vr = h.re[r * h.dim + c], vi = h.im[r * h.dim + c];
        if (vr == 0.0 && vi == 0.0) continue;
        int x = c ^ r;
        uint64_t mask = 0;
        for (int k = 0; k < ns; ++k)
          if ((x >> (ns - 1 - k)) & 1) mask |= 1ull << td.bitpos[k];
        xm.push_back(mask);
        vals.push_back(make_double2(vr, vi));
      }
    }
    cp.push_back((int)xm.size());
    tds.push_back(td);
  }
  op->nfam = (int)fams.size();
  op->ngeneric = (int)tds.size();
  // flip-flop fast path eligibility
  {
    bool ok = L <= 32 && op->gather && b->dev.bk != BK_ABELIAN && !fams.empty() &&
              fams.size() <= (size_t)kMaxFF && xm.empty();
    for (const FamDev& F : fams)
      ok = ok && F.nnz[0] == 0 && F.nnz[3] == 0 && F.nnz[1] == 1 && F.nnz[2] == 1 &&
           F.xr[1][0] == 3 && F.xr[2][0] == 3;
    op->ff_ok = ok;
    if (ok) {
      FFParams ff{};
      ff.nfam = (int)fams.size();
      for (size_t f = 0; f < fams.size(); ++f) {
        ff.d[f] = fams[f].d;
        ff.valid[f] = (uint32_t)fams[f].valid;
        for (int c = 0; c < 4; ++c) ff.dval[f][c] = fams[f].dval[c];
        ff.v1[f] = fams[f].val[1][0];
        ff.v2[f] = fams[f].val[2][0];
        ff.same[f] = ff.v1[f].x == ff.v2[f].x && ff.v1[f].y == ff.v2[f].y;
      }
      op->ff_params.resize(sizeof(FFParams));
      std::memcpy(op->ff_params.data(), &ff, sizeof(FFParams));
    }
  }
  std::vector<PauliGroup> pgroup;
  std::vector<PauliStr> pstr, pdiag;
  op->pauli_ok = op->use_ff && op->gather && !op->ff_ok && b->dev.bk == BK_TENSOR && L <= 31 &&
                 pauli_strings(terms, in_family, b->dev, op->pauli_flips, pgroup, pstr, pdiag);
  auto upload = [&](DevBuf& buf, const void* src, size_t bytes) -> edk_status {
    if (bytes == 0) return EDK_OK;
    EDK_RETURN_IF(buf.alloc(bytes));
    EDK_TRY_CUDA(cudaMemcpy(buf.p, src, bytes, cudaMemcpyHostToDevice));
    return EDK_OK;
  };
  EDK_RETURN_IF(upload(op->fam, fams.data(), fams.size() * sizeof(FamDev)));
  EDK_RETURN_IF(upload(op->term, tds.data(), tds.size() * sizeof(TermDev)));
  EDK_RETURN_IF(upload(op->colptr, cp.data(), cp.size() * sizeof(int)));
  EDK_RETURN_IF(upload(op->xmask, xm.data(), xm.size() * sizeof(uint64_t)));
  EDK_RETURN_IF(upload(op->val, vals.data(), vals.size() * sizeof(double2)));
  EDK_RETURN_IF(upload(op->dval, dvals.data(), dvals.size() * sizeof(double2)));
  if (op->pauli_ok) {
    EDK_RETURN_IF(upload(op->pa_group, pgroup.data(), pgroup.size() * sizeof(PauliGroup)));
    EDK_RETURN_IF(upload(op->pa_str, pstr.data(), pstr.size() * sizeof(PauliStr)));
    EDK_RETURN_IF(upload(op->pa_diag, pdiag.data(), pdiag.size() * sizeof(PauliStr)));
    op->pauli = PauliDev{(int)pgroup.size(), (int)pdiag.size(), op->pa_group.as<PauliGroup>(),
                         op->pa_str.as<PauliStr>(), op->pa_diag.as<PauliStr>()};
  }
  op->dev.nfam = op->nfam;
  op->dev.fam = op->fam.as<FamDev>();
  op->dev.nterm = op->ngeneric;
  op->dev.term = op->term.as<TermDev>();
  op->dev.colptr = op->colptr.as<int>();
  op->dev.xmask = op->xmask.as<uint64_t>();
  op->dev.val = op->val.as<double2>();
  op->dev.dval = op->dval.as<double2>();
  EDK_TRY_CUDA(cudaStreamCreateWithFlags(&op->stream, cudaStreamNonBlocking));
  *out = guard.release();
  return EDK_OK;
}

extern "C" edk_status edk_operator_destroy(edk_operator* op) {
  delete op;
  return EDK_OK;
}

extern "C" edk_status edk_operator_info(const edk_operator* op, int32_t* gather,
                                        int32_t* is_complex, int32_t* n_families,
                                        int32_t* n_generic) {
  EDK_CHECK_ARG(op != nullptr, "edk_operator_info: NULL operator");
  if (gather) *gather = op->gather ? 1 : 0;
  if (is_complex) *is_complex = op->is_complex ? 1 : 0;
  if (n_families) *n_families = op->nfam;
  if (n_generic) *n_generic = op->ngeneric;
  return EDK_OK;
}

// after a synchronised product: a bounded wait of the staged materialised
// kernel that ran out (never expected) is reported instead of a silent result
static edk_status staged_status(edk_operator* op) {
  if (!(op->sell_ok && op->sell_tma && op->sell_tma_ok && op->s_err.p)) return EDK_OK;
  int err = 0;
  EDK_TRY_CUDA(cudaMemcpy(&err, op->s_err.p, sizeof(int), cudaMemcpyDeviceToHost));
  if (err) {
    // the device did not complete a bulk copy: never use the staged kernel on
    // this operator again (later products take the plain materialised kernel)
    op->sell_tma_ok = false;
    op->sell_tma = false;
    set_error("apply: the staged materialised product timed out waiting for its copies");
    return EDK_TIMEOUT;
  }
  return EDK_OK;
}

static edk_status check_dtype(const edk_operator* op, int dtype) {
  EDK_CHECK_ARG(dtype >= EDK_F64 && dtype <= EDK_C64, "apply: unknown dtype");
  if (op->is_complex && (dtype == EDK_F64 || dtype == EDK_F32)) {
    set_error("apply: the operator has complex matrix elements; use a complex dtype");
    return EDK_INVALID_ARG;
  }
  return EDK_OK;
}

extern "C" edk_status edk_apply_async(edk_operator* op, int32_t dtype, const void* x, void* y,
                                      int64_t nvec, int64_t ldx, int64_t ldy, int32_t accumulate,
                                      void* stream) {
  EDK_CHECK_ARG(op && x && y, "edk_apply_async: NULL argument");
  EDK_RETURN_IF(check_dtype(op, dtype));
  EDK_CHECK_ARG(nvec >= 0 && ldx >= op->b->D && ldy >= op->b->D, "edk_apply_async: bad ld");
  return apply_device(op, dtype, x, y, nvec, ldx, ldy, accumulate,
                      static_cast<cudaStream_t>(stream));
}

extern "C" edk_status edk_apply(edk_operator* op, int32_t dtype, const void* x, void* y,
                                int64_t nvec, int64_t ldx, int64_t ldy, int32_t accumulate,
                                int32_t ptr_kind) {
  EDK_CHECK_ARG(op && x && y, "edk_apply: NULL argument");
  EDK_RETURN_IF(check_dtype(op, dtype));
  const int64_t D = op->b->D;
  EDK_CHECK_ARG(nvec >= 0 && ldx >= D && ldy >= D, "edk_apply: ldx/ldy smaller than the dimension");
  std::lock_guard<std::mutex> lk(op->mu);
  cudaStream_t st = op->stream;
  if (ptr_kind == EDK_DEVICE) {
    EDK_RETURN_IF(apply_device(op, dtype, x, y, nvec, ldx, ldy, accumulate, st));
    EDK_TRY_CUDA(cudaStreamSynchronize(st));
    return staged_status(op);
  }
  EDK_CHECK_ARG(ptr_kind == EDK_HOST, "edk_apply: bad ptr_kind");
  if (nvec == 0 || D == 0) return EDK_OK;
  size_t es = dtype_size(dtype);
  DevBuf& dx = op->hx;
  DevBuf& dy = op->hy;
  size_t need = (size_t)D * nvec * es;
  if (dx.bytes < need) EDK_RETURN_IF(dx.alloc(need));
  if (dy.bytes < need) EDK_RETURN_IF(dy.alloc(need));
  EDK_TRY_CUDA(cudaMemcpy2DAsync(dx.p, D * es, x, ldx * es, D * es, nvec, cudaMemcpyHostToDevice, st));
  if (accumulate)
    EDK_TRY_CUDA(cudaMemcpy2DAsync(dy.p, D * es, y, ldy * es, D * es, nvec, cudaMemcpyHostToDevice, st));
  constexpr int64_t kChunkRows = 262144;  // a multiple of every tile height
  if (nvec == 1 && D >= 2 * kChunkRows && rows_apply_ok(op)) {
    // pipelined: row chunks computed in order on the operator's stream, each
    // chunk of y copied back on the copy stream while the next one computes
    // (psi gathers reach any row, so the input copy cannot be split this way)
    const int nch = (int)((D + kChunkRows - 1) / kChunkRows);
    if (!op->cstream) EDK_TRY_CUDA(cudaStreamCreateWithFlags(&op->cstream, cudaStreamNonBlocking));
    while ((int)op->cevents.size() < nch) {
      cudaEvent_t e;
      EDK_TRY_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      op->cevents.push_back(e);
    }
    for (int c = 0; c < nch; ++c) {
      const int64_t r0 = (int64_t)c * kChunkRows, r1 = std::min<int64_t>(D, r0 + kChunkRows);
      EDK_RETURN_IF(apply_rows(op, dtype, dx.p, dy.p, r0, r1, accumulate, st));
      EDK_TRY_CUDA(cudaEventRecord(op->cevents[c], st));
      EDK_TRY_CUDA(cudaStreamWaitEvent(op->cstream, op->cevents[c], 0));
      EDK_TRY_CUDA(cudaMemcpyAsync((char*)y + r0 * es, (char*)dy.p + r0 * es, (r1 - r0) * es,
                                   cudaMemcpyDeviceToHost, op->cstream));
    }
    EDK_TRY_CUDA(cudaStreamSynchronize(op->cstream));
    EDK_TRY_CUDA(cudaStreamSynchronize(st));
    return staged_status(op);
  }
  EDK_RETURN_IF(apply_device(op, dtype, dx.p, dy.p, nvec, D, D, accumulate, st));
  EDK_TRY_CUDA(cudaMemcpy2DAsync(y, ldy * es, dy.p, D * es, D * es, nvec, cudaMemcpyDeviceToHost, st));
  EDK_TRY_CUDA(cudaStreamSynchronize(st));
  return staged_status(op);
}
