// edk_plan.cu — row plans of the flip-flop fast path on rank-searched sectors
// (translation and translation + parity sectors with their rank table, and
// complete fixed-charge sectors), and the kernel that applies H through them.
//
// A plan is built once per operator, on the device, the first time the
// operator is applied with such a search: for every 256-row window the rows
// are ordered by their number of off-diagonal hits, and each slot keeps the
// row's 32-bit state, its colex rank, `row | norm class << 27` and the rank of
// its wrap-around exchange (plus the summed diagonal when the operator has
// diagonal-only generic terms, e.g. random fields).  The product then runs
// one thread per slot with the tables it reads per hit (binomials, norms,
// phases) in shared memory; edk_rankrows.cuh holds the per-row arithmetic.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <set>
#include <type_traits>

#include "edk_rankrows.cuh"

namespace edk {

namespace {

// Order the 256 rows of window blockIdx.x by hit count (ties by row, so the
// plan is the same on every build) and write their slots.  A counting sort:
// lanes with equal counts find their order with one match, warps through a
// shared histogram (comparing every pair of rows took most of the build,
// 89 us for 1,432,860 rows; 29 us now).
template <int BK>
__global__ void __launch_bounds__(256) k_plan_build(BasisDev b, OpDev op, FFParams ff,
                                                    int want_diag,
                                                    uint4* __restrict__ slot_o,
                                                    double* __restrict__ dg_o,
                                                    int* __restrict__ bad) {
  constexpr int kKeys = 160;  // hits 0 .. 128, then rows past the last; five per lane
  __shared__ unsigned short s_hist[kPlanWindow / 32][kKeys], s_base[kKeys];
  __shared__ uint32_t s_binom[32 * 33];
  fill_binom32(s_binom);
  for (int e = threadIdx.x; e < kPlanWindow / 32 * kKeys; e += kPlanWindow) (&s_hist[0][0])[e] = 0;
  __syncthreads();
  const int t = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * kPlanWindow, i = r0 + t;
  const bool valid = i < b.D;
  const uint32_t mask = (uint32_t)b.maskL;
  uint32_t s = 0, rk = 0, rw = ~0u, rkw = ~0u;
  int key = kKeys - 1;  // past the last row: sorted to the end
  double dr = 0.0, di = 0.0;
  if (valid) {
    s = (uint32_t)__ldg(b.I + i);
    key = 0;
    for (int f = 0; f < ff.nfam; ++f)
      key += __popc((s ^ rotl_L(s, ff.d[f], b.L, mask)) & ff.valid[f]);
    uint32_t cls = 0;
    if constexpr (BK == BK_PROJ_RANK) {
      rk = (uint32_t)i;
    } else {
      rk = __ldg(b.rowrank + i);
      const uint32_t v = __ldg(b.rankmap + rk);
      if (v == ~0u || (int64_t)(v >> b.rank_shift) != i) atomicOr(bad, 1);
      cls = v & 31u;
    }
    rw = (uint32_t)i | (cls << 27);
    // the wrap-around bond (bits 0 and L-1) of a nearest-neighbour family:
    // its target rank walks the set bits in between, so it is kept per row
    bool wrap = false;
    for (int f = 0; f < ff.nfam; ++f) wrap |= ff.d[f] == 1 && (ff.valid[f] & 1u);
    if (wrap && ((s ^ (s >> (b.L - 1))) & 1u)) rkw = rank_after_swap(s, rk, 0, b.L - 1, s_binom);
    if (want_diag) {
      for (int f = 0; f < ff.nfam; ++f)
        ff_diag(ff, f, s, rotl_L(s, ff.d[f], b.L, mask), ff.valid[f], dr, di);
      term_diag(op, s, dr, di);
      if (di != 0.0) atomicOr(bad, 2);
    }
  }
  const int warp = t >> 5, lane = t & 31;
  const unsigned peers = __match_any_sync(0xffffffffu, key);
  const int mine = __popc(peers & ((1u << lane) - 1u));
  if (mine == 0) s_hist[warp][key] = (unsigned short)__popc(peers);
  __syncthreads();
  if (warp == 0) {  // rows with smaller keys, for the lane's five keys
    int n[5], sum = 0;
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      n[u] = 0;
      for (int w = 0; w < kPlanWindow / 32; ++w) n[u] += s_hist[w][5 * lane + u];
      sum += n[u];
    }
    int before = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += v;
    }
    before -= sum;
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      s_base[5 * lane + u] = (unsigned short)before;
      before += n[u];
    }
  }
  __syncthreads();
  int pos = s_base[key] + mine;
  for (int w = 0; w < warp; ++w) pos += s_hist[w][key];
  const int64_t slot = r0 + pos;
  slot_o[slot] = make_uint4(rw, s, rk, rkw);
  if (want_diag) dg_o[slot] = dr;
}

// NN = 1: the operator is one nearest-neighbour family of equal exchange
// values (its loop only); NN = 2: any other operator (the general loop only)
template <int BK, class VT, int NN>
__global__ void __launch_bounds__(256, plan_min_blocks<BK, VT>())
    k_apply_plan(BasisDev b, OpDev op, FFParams ff, const VT* __restrict__ x,
                 VT* __restrict__ y, int64_t ldx, int64_t ldy, int accumulate, int64_t slot0,
                 int64_t slot1) {
  __shared__ FFTab<BK> sm;
  ff_tab_fill<BK>(sm, b);
  __syncthreads();
  const VT* xk = x + (int64_t)blockIdx.y * ldx;
  VT* yk = y + (int64_t)blockIdx.y * ldy;
  for (int64_t s = slot0 + (int64_t)blockIdx.x * kPlanWindow + threadIdx.x; s < slot1;
       s += (int64_t)gridDim.x * kPlanWindow)
    plan_row<BK, VT, NN>(b, op, ff, sm, s, xk, yk, accumulate);
}

// Several columns at once (blockIdx.y = group of kPlanCols columns): a target is
// located once for all of them.  Taken for eight and more real columns (5 of 48,620
// rows 27.8 -> 29.9 us a product, complex columns 112 -> 120) whose groups and windows
// make two blocks per SM, one where rows have more than nearest neighbours: fewer, and the single-column kernel's larger number of
// blocks counts for more than its repeated searches.  FP64, one by one / grouped:
// 16 columns of 924 rows 24.9 / 26.9, of 12,870 28.4 / 29.3, of 48,620 35.8 / 38.9,
// of 184,756 74 / 65, of 400,024 rank-searched 196 / 143; 31 of 12,870 rows with two
// families 40.8 / 36.2; single precision, 13 of 48,620 34.0 / 32.8, of 12,870 with two
// families 27.3 / 25.5.
// A last group of two or three columns repeats its last one (11 of 400,024 rows: 111
// us, 124 with the three one by one); a single column goes alone where the windows
// fill the GPU by themselves (9 of 400,024 rows 107 -> 100 us, of 705,432 135 -> 122;
// but of 112,720 48.6 -> 50.8: the second launch).
constexpr int kPlanCols = 4;
constexpr int64_t kPlanColsMin = 8;
constexpr int kPlanColsBlocks = 4;  // resident blocks per SM of the grouped kernel

template <int BK, class VT, int NN, int NC>
__global__ void __launch_bounds__(256, (sizeof(VT) == 4 && NN == 1) ? 5 : 4)
    k_apply_plan_cols(BasisDev b, OpDev op, FFParams ff, const VT* __restrict__ x,
                      VT* __restrict__ y, int64_t ldx, int64_t ldy, int accumulate, int nvec,
                      int64_t slot0, int64_t slot1) {
  __shared__ FFTab<BK> sm;
  ff_tab_fill<BK>(sm, b);
  __syncthreads();
  const VT* xk[NC];
  VT* yk[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int k = (int)blockIdx.y * NC + c;
    xk[c] = x + (int64_t)(k < nvec ? k : nvec - 1) * ldx;
    yk[c] = k < nvec ? y + (int64_t)k * ldy : nullptr;
  }
  for (int64_t s = slot0 + (int64_t)blockIdx.x * kPlanWindow + threadIdx.x; s < slot1;
       s += (int64_t)gridDim.x * kPlanWindow)
    plan_row_cols<BK, VT, NN, NC>(b, op, ff, sm, s, xk, yk, accumulate);
}

int sm_count() {
  static int n[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    n[dev] = 148;
  return n[dev];
}

template <int BK, class VT, int NN>
edk_status launch_plan_nn(const BasisDev& b, const OpDev& op, const FFParams& ff, const VT* X,
                          VT* Y, int64_t nvec, int64_t ldx, int64_t ldy, int accumulate,
                          cudaStream_t st, int64_t slot0, int64_t slot1) {
  static int per_sm = 0;  // resident blocks per SM of this instantiation
  if (!per_sm) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_apply_plan<BK, VT, NN>,
                                                      kPlanWindow, 0) != cudaSuccess || per_sm < 1)
      per_sm = 1;
  }
  const int64_t nwin = (slot1 - slot0) / kPlanWindow;
  if constexpr (!VTraits<VT>::cx) {
    constexpr int NC = kPlanCols;
    const int64_t nsm = sm_count();
    if (nvec >= kPlanColsMin && nwin * ((nvec + NC - 1) / NC) >= (NN == 1 ? 2 : 1) * nsm) {
      const unsigned gc = (unsigned)std::min<int64_t>(nwin, nsm * kPlanColsBlocks);
      const bool alone = nvec % NC == 1 && nwin >= nsm * kPlanColsBlocks;
      const int64_t grouped = alone ? nvec - 1 : nvec;
      for (int64_t k0 = 0; k0 < grouped; k0 += (int64_t)NC * 65535) {
        const int64_t nk = std::min<int64_t>(grouped - k0, (int64_t)NC * 65535);
        k_apply_plan_cols<BK, VT, NN, NC>
            <<<dim3(gc, (unsigned)((nk + NC - 1) / NC)), kPlanWindow, 0, st>>>(
                b, op, ff, X + k0 * ldx, Y + k0 * ldy, ldx, ldy, accumulate, (int)nk, slot0, slot1);
        EDK_TRY_CUDA(cudaGetLastError());
      }
      if (!alone) return EDK_OK;
      X += grouped * ldx;
      Y += grouped * ldy;
      nvec = 1;
    }
  }
  const unsigned gx = (unsigned)std::min<int64_t>(nwin, (int64_t)sm_count() * per_sm);
  for (int64_t k0 = 0; k0 < nvec; k0 += 65535) {
    const int64_t nk = std::min<int64_t>(nvec - k0, 65535);
    k_apply_plan<BK, VT, NN><<<dim3(gx, (unsigned)nk), kPlanWindow, 0, st>>>(
        b, op, ff, X + k0 * ldx, Y + k0 * ldy, ldx, ldy, accumulate, slot0, slot1);
    EDK_TRY_CUDA(cudaGetLastError());
  }
  return EDK_OK;
}

template <int BK, class VT>
edk_status launch_plan_kind(const BasisDev& b, const OpDev& op, const FFParams& ff, const VT* X,
                            VT* Y, int64_t nvec, int64_t ldx, int64_t ldy, int accumulate,
                            cudaStream_t st, int64_t slot0, int64_t slot1) {
  if (plan_nn(ff))
    return launch_plan_nn<BK, VT, 1>(b, op, ff, X, Y, nvec, ldx, ldy, accumulate, st, slot0, slot1);
  return launch_plan_nn<BK, VT, 2>(b, op, ff, X, Y, nvec, ldx, ldy, accumulate, st, slot0, slot1);
}

// lookup kind of the plan kernels for the basis as it is searched now, or -1
int plan_kind(const BasisDev& b) {
  if (b.bk == BK_PROJ_RANK) return BK_PROJ_RANK;
  if (b.search != 2) return -1;
  switch (b.bk) {
    case BK_TRANS0: return BK_TRANS0_RANK;
    case BK_TRANS: return BK_TRANS_RANK;
    case BK_TRANSPAR: return BK_TRANSPAR_RANK;
  }
  return -1;
}

template <int BK>
void launch_plan_build(edk_operator* op, uint4* slot, double* dg, int* bad, cudaStream_t st) {
  const BasisDev& b = op->b->dev;
  const FFParams& ff = *reinterpret_cast<const FFParams*>(op->ff_params.data());
  const unsigned nwin = (unsigned)((b.D + kPlanWindow - 1) / kPlanWindow);
  k_plan_build<BK><<<nwin, kPlanWindow, 0, st>>>(b, op->dev, ff, dg != nullptr, slot, dg, bad);
}

}  // namespace

// The plan applies to this operator as its basis is searched now.
bool plan_applies(const edk_operator* op) {
  const BasisDev& b = op->b->dev;
  return op->use_plan && op->ff_ok && op->use_ff && op->gather && op->tps == 1 && b.L <= 32 &&
         b.D > 0 && b.D <= (int64_t)kPlanRowMask && plan_kind(b) >= 0 &&
         (b.bk == BK_PROJ_RANK || b.packed) && op->plan_state >= 0;
}

// A batch's plans share allocations of up to this size (a larger plan has its own), so
// what one operator that stays holds of the others' memory is bounded.
constexpr size_t kPlanSlab = (size_t)64 << 20;

// Build the plans of the operators that need one and have none yet (plan_state: 0
// not built yet, 1 built, -1 not available for this operator).  Allocates and
// synchronises: call it outside any stream capture.  The plans of a call share
// allocations and one synchronisation: the first solve of a new batch pays
// for them (96 chains of 12 to 20 sites: 21 ms one by one, 1.9 ms together).
edk_status plan_ensure(const std::vector<edk_operator*>& ops, cudaStream_t st) {
  auto pad = [](size_t n) { return (n + 255) / 256 * 256; };
  struct Place { size_t slab, at; };
  std::vector<edk_operator*> need;
  std::set<edk_operator*> seen;
  std::vector<Place> place;
  std::vector<size_t> size;  // of each slab
  for (edk_operator* op : ops) {
    if (op->plan_state != 0 || plan_kind(op->b->dev) < 0 || !seen.insert(op).second) continue;
    const size_t ns = (size_t)((op->b->D + kPlanWindow - 1) / kPlanWindow) * kPlanWindow;
    const size_t n = pad(ns * sizeof(uint4)) + (op->ngeneric > 0 ? pad(ns * 8) : 0);
    if (size.empty() || size.back() + n > kPlanSlab) size.push_back(0);
    need.push_back(op);
    place.push_back({size.size() - 1, size.back()});
    size.back() += n;
  }
  if (need.empty()) return EDK_OK;
  const size_t flags = size[0];  // the build's flags, at the end of the first
  size[0] += need.size() * sizeof(int);
  std::vector<std::shared_ptr<PlanSlab>> slabs;
  for (size_t n : size) {
    slabs.push_back(std::make_shared<PlanSlab>());
    slabs.back()->device = need[0]->b->device;
    EDK_RETURN_IF(slabs.back()->buf.alloc_async(n, st, keep_pool()));
  }
  auto where = [&](size_t i) { return slabs[place[i].slab]->buf.as<char>() + place[i].at; };
  int* bad = reinterpret_cast<int*>(slabs[0]->buf.as<char>() + flags);
  EDK_TRY_CUDA(cudaMemsetAsync(bad, 0, need.size() * sizeof(int), st));
  for (size_t i = 0; i < need.size(); ++i) {
    edk_operator* op = need[i];
    const int64_t ns = (op->b->D + kPlanWindow - 1) / kPlanWindow * kPlanWindow;
    uint4* slot = reinterpret_cast<uint4*>(where(i));
    double* dg = op->ngeneric > 0 ? reinterpret_cast<double*>(where(i) + pad(ns * sizeof(uint4)))
                                  : nullptr;
    switch (plan_kind(op->b->dev)) {
      case BK_PROJ_RANK: launch_plan_build<BK_PROJ_RANK>(op, slot, dg, bad + i, st); break;
      case BK_TRANS0_RANK: launch_plan_build<BK_TRANS0_RANK>(op, slot, dg, bad + i, st); break;
      case BK_TRANS_RANK: launch_plan_build<BK_TRANS_RANK>(op, slot, dg, bad + i, st); break;
      default: launch_plan_build<BK_TRANSPAR_RANK>(op, slot, dg, bad + i, st); break;
    }
  }
  EDK_TRY_CUDA(cudaGetLastError());
  std::vector<int> h(need.size());
  EDK_TRY_CUDA(cudaMemcpyAsync(h.data(), bad, h.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
  EDK_TRY_CUDA(cudaStreamSynchronize(st));
  for (size_t i = 0; i < need.size(); ++i) {
    edk_operator* op = need[i];
    if (h[i] & 1) {
      set_error("row plan: a representative's rank-table entry does not point back at its row");
      return EDK_CUDA_ERROR;
    }
    if (h[i] & 2) {  // complex diagonal: keep the tile kernel
      op->plan_state = -1;
      continue;
    }
    const int64_t ns = (op->b->D + kPlanWindow - 1) / kPlanWindow * kPlanWindow;
    RowPlanDev& pl = op->dev.plan;
    pl.slot = reinterpret_cast<uint4*>(where(i));
    pl.dg = op->ngeneric > 0 ? reinterpret_cast<double*>(where(i) + pad(ns * sizeof(uint4)))
                             : nullptr;
    pl.nslots = ns;
    op->p_slab = slabs[place[i].slab];
    op->plan_state = 1;
  }
  return EDK_OK;
}

// Rows [row0, row1) of y = H x through the plan (row0 a multiple of 256,
// row1 a multiple of 256 or the dimension): the slots of the same windows.
edk_status apply_plan(edk_operator* op, int dtype, const void* x, void* y, int64_t nvec,
                      int64_t ldx, int64_t ldy, int accumulate, cudaStream_t st, int64_t row0,
                      int64_t row1) {
  EDK_RETURN_IF(plan_ensure({op}, op->stream));
  const BasisDev& b = op->b->dev;
  const FFParams& ff = *reinterpret_cast<const FFParams*>(op->ff_params.data());
  if (op->plan_state != 1) {
    set_error("row plan: not available for this operator");
    return EDK_UNSUPPORTED;
  }
  if (row1 < 0) row1 = b.D;
  const int64_t slot0 = (row0 / kPlanWindow) * kPlanWindow;
  const int64_t slot1 = std::min<int64_t>(((row1 + kPlanWindow - 1) / kPlanWindow) * kPlanWindow,
                                          op->dev.plan.nslots);
  if (slot1 <= slot0 || nvec <= 0) return EDK_OK;
  auto go = [&](auto vp) -> edk_status {
    using VT = std::remove_pointer_t<decltype(vp)>;
    const VT* X = static_cast<const VT*>(x);
    VT* Y = static_cast<VT*>(y);
    switch (plan_kind(b)) {
      case BK_PROJ_RANK:
        return launch_plan_kind<BK_PROJ_RANK, VT>(b, op->dev, ff, X, Y, nvec, ldx, ldy, accumulate,
                                                  st, slot0, slot1);
      case BK_TRANS0_RANK:
        return launch_plan_kind<BK_TRANS0_RANK, VT>(b, op->dev, ff, X, Y, nvec, ldx, ldy,
                                                    accumulate, st, slot0, slot1);
      case BK_TRANS_RANK:
        return launch_plan_kind<BK_TRANS_RANK, VT>(b, op->dev, ff, X, Y, nvec, ldx, ldy,
                                                   accumulate, st, slot0, slot1);
      case BK_TRANSPAR_RANK:
        return launch_plan_kind<BK_TRANSPAR_RANK, VT>(b, op->dev, ff, X, Y, nvec, ldx, ldy,
                                                      accumulate, st, slot0, slot1);
    }
    set_error("row plan: unknown lookup kind");
    return EDK_INVALID_ARG;
  };
  switch (dtype) {
    case EDK_F64: return go((double*)nullptr);
    case EDK_C128: return go((double2*)nullptr);
    case EDK_F32: return go((float*)nullptr);
    case EDK_C64: return go((float2*)nullptr);
  }
  set_error("apply: unknown dtype");
  return EDK_INVALID_ARG;
}

}  // namespace edk
