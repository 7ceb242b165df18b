// edk_batch.cu — Lanczos over many independent operators in lockstep
// (momentum sectors of one chain, disorder instances), and the single-operator
// ground state as a batch of one.
//
// Every kernel of a step covers all operators of the batch in one launch: a
// block owns a tile of one operator's rows (tile2op map) or, in the
// reorthogonalisation kernels, an equal share of all rows (RowSplit), reads
// that operator's basis/term descriptors from a device array, and works on
// its slice of the concatenated buffers.  The step index j, the recurrence
// coefficients alpha/beta, 1/beta and the per-operator stop flags live on the
// device, so a step has no host round trip: it is captured once into a CUDA
// graph and replayed.  Every check_every steps the device solves the
// tridiagonal problems and tests convergence (edk_tridiag.cu); the host reads
// only how many operators are left.  One step per operator q:
//   wt_q = H_q v_j                       (row-gather matvec)
//   s = V_q^H v_j, r = V_q^H wt_q          (one read of V for both)
//   v_j = (v_j - V_q s) / a                (the second sweep of the step before)
//   w_q = H v_j - V_q V_q^H H v_j          (the first sweep of this step; the same
//                                          second read of V serves both)
//   beta_j = ||w_q|| ; lucky breakdown beta <= sqrt(eps) max(1, |alpha|) stops q
//   v_{j+1} = w_q / beta_j
// (classical Gram-Schmidt twice, as _lanczos_build! in
// src/algorithms/TimeEvolution.jl:250-306, with its three-term recurrence
// folded into the first sweep, and the second sweep delayed by one step; see
// k_rdots2).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <complex>
#include <cstring>
#include <map>
#include <memory>
#include <vector>

#include "edk_rankrows.cuh"

namespace edk {

namespace {

constexpr int kTile = 256;          // rows per matvec / update tile
// Steps of a run, as edk.h has it.  No kernel needs a limit; a longer run would spend
// its time in T's eigenvalues (a chain of as many dependent multiply-adds a count).
// Krylov bases, which look at no eigenvalues here, may have more vectors.
constexpr int kMaxSteps = 12791;
// resident reorthogonalisation blocks per SM (128 registers a thread)
constexpr int kSplitBlocks = 2;

template <class T> struct IsCx;
template <> struct IsCx<double> { static constexpr bool v = false; };
template <> struct IsCx<double2> { static constexpr bool v = true; };
template <> struct IsCx<float> { static constexpr bool v = false; };
template <> struct IsCx<float2> { static constexpr bool v = true; };

__device__ __forceinline__ double2 l2(const double* p) { return make_double2(*p, 0.0); }
__device__ __forceinline__ double2 l2(const double2* p) { return *p; }
__device__ __forceinline__ double2 l2(const float* p) { return make_double2((double)*p, 0.0); }
__device__ __forceinline__ double2 l2(const float2* p) {
  float2 v = *p;
  return make_double2((double)v.x, (double)v.y);
}
__device__ __forceinline__ void s2(double* p, double2 v) { *p = v.x; }
__device__ __forceinline__ void s2(double2* p, double2 v) { *p = v; }
__device__ __forceinline__ void s2(float* p, double2 v) { *p = (float)v.x; }
__device__ __forceinline__ void s2(float2* p, double2 v) { *p = make_float2((float)v.x, (float)v.y); }

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace

// One operator of a batch, as the kernels see it.
struct __align__(16) BOp {
  BasisDev b;
  OpDev op;
  FFParams ff;
  int64_t D;
  int64_t voff;   // element offset of V_q (D x ncap, column-major)
  int64_t woff;   // element offset into w / wt
  int64_t tile0;  // first matvec tile
  int64_t sblk0;  // first block of the materialised-matrix product (8 slices each)
  int ntile;
};

// ---------------------------------------------------------------------------
// kernels (j = *step; operators with done[q] != 0 are skipped)
// ---------------------------------------------------------------------------
template <int BK, class VT>
__global__ void __launch_bounds__(256) k_bapply_ff(const BOp* __restrict__ ops,
                                                   const int* __restrict__ tile2op,
                                                   const VT* __restrict__ V, VT* __restrict__ wt,
                                                   const int* __restrict__ step,
                                                   const int* __restrict__ done) {
  const int q = tile2op[blockIdx.x];
  if (done[q]) return;
  const BOp& o = ops[q];
  const int j = *step;
  ff_tile<BK, VT>(o.b, o.op, o.ff, (blockIdx.x - o.tile0) * (int64_t)kTile,
                  V + o.voff + (int64_t)j * o.D, wt + o.woff, 0);
}

// the row-plan form of k_bapply_ff (rank-searched sectors whose operators all
// carry a plan): tile t of operator q is window t of q's plan
template <int BK, class VT, int NN>
__global__ void __launch_bounds__(256, plan_min_blocks<BK, VT>()) k_bapply_plan(const BOp* __restrict__ ops,
                                                     const int* __restrict__ tile2op,
                                                     int64_t ntiles,
                                                     const VT* __restrict__ V, VT* __restrict__ wt,
                                                     const int* __restrict__ step,
                                                     const int* __restrict__ done) {
  // a resident grid walks the tiles; the operator record and its tables are
  // loaded into shared memory again only when the operator changes
  __shared__ FFTab<BK> sm;
  __shared__ __align__(16) BOp s_op;  // the operator record, read from shared memory
  const int j = *step;
  int cur = -1;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int q = tile2op[tile];
    if (done[q]) continue;
    if (q != cur) {
      __syncthreads();  // the previous operator's rows no longer read the tables
      const int4* src = reinterpret_cast<const int4*>(ops + q);
      int4* dst = reinterpret_cast<int4*>(&s_op);
      for (int e = threadIdx.x; e < (int)(sizeof(BOp) / sizeof(int4)); e += blockDim.x) dst[e] = src[e];
      __syncthreads();
      ff_tab_fill<BK>(sm, s_op.b);
      __syncthreads();
      cur = q;
    }
    const BOp& o = s_op;
    plan_row<BK, VT, NN>(o.b, o.op, o.ff, sm, (tile - o.tile0) * (int64_t)kTile + threadIdx.x,
                         V + o.voff + (int64_t)j * o.D, wt + o.woff, 0);
  }
}

template <class VT>
__global__ void __launch_bounds__(256) k_bapply_sell(const BOp* __restrict__ ops,
                                                     const int* __restrict__ sblk2op,
                                                     const VT* __restrict__ V, VT* __restrict__ wt,
                                                     const int* __restrict__ step,
                                                     const int* __restrict__ done) {
  const int q = sblk2op[blockIdx.x];
  if (done[q]) return;
  const BOp& o = ops[q];
  const int64_t slice = (blockIdx.x - o.sblk0) * 8 + (threadIdx.x >> 5);
  if (slice >= o.op.sell.nslices) return;
  const int j = *step;
  sell_slice<VT>(o.b, o.op.sell, slice, threadIdx.x & 31, V + o.voff + (int64_t)j * o.D,
                 wt + o.woff, 0);
}

template <int BK, class VT>
__global__ void __launch_bounds__(256) k_bapply_gen(const BOp* __restrict__ ops,
                                                    const int* __restrict__ tile2op,
                                                    const VT* __restrict__ V,
                                                    VT* __restrict__ wt,
                                                    const int* __restrict__ step,
                                                    const int* __restrict__ done) {
  __shared__ uint32_t s_binom[32 * 33];
  if constexpr (BK == BK_PROJ_RANK) {
    fill_binom32(s_binom);
    __syncthreads();
  }
  const int q = tile2op[blockIdx.x];
  if (done[q]) return;
  const BOp& o = ops[q];
  const int64_t i = (blockIdx.x - o.tile0) * (int64_t)kTile + threadIdx.x;
  if (i >= o.D) return;
  const int j = *step;
  gen_row<BK, uint32_t, VT, true>(o.b, o.op, i, V + o.voff + (int64_t)j * o.D, wt + o.woff, 0,
                                  s_binom);
}

// Sum of eight values over a warp, one value index per lane group: three
// halving exchanges (offsets 16, 8, 4: a lane keeps half of its values and
// adds its partner's copy of that half) then two butterfly steps.  Nine
// shuffles for eight sums instead of forty; lane l ends with the total of
// value (l >> 2) & 7.
__device__ __forceinline__ double wsum8(const double (&a)[8], int lane) {
  double b[4], c[2];
  const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double send = h16 ? a[i] : a[i + 4];
    b[i] = (h16 ? a[i + 4] : a[i]) + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double send = h8 ? b[i] : b[i + 2];
    c[i] = (h8 ? b[i + 2] : b[i]) + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  double d = (h4 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, h4 ? c[0] : c[1], 4);
  d += __shfl_xor_sync(0xffffffffu, d, 2);
  d += __shfl_xor_sync(0xffffffffu, d, 1);
  return d;
}

// ---------------------------------------------------------------------------
// Reorthogonalisation kernels.  Their grid is G blocks that are all resident
// at once (G = SMs x blocks per SM), and block b owns rows
// [b T / G, (b + 1) T / G) of the concatenated rows of the operators still
// running (T rows in all, recomputed by k_bsplit at the start of every step):
// every block streams the same number of bytes, so no partly filled last
// wave of blocks holds the launch up and operators that have stopped leave
// no block idle.  A block whose rows run from one operator into the next
// handles each piece in turn; its slot among operator q's partial sums is
// b - bfirst_q (nslot_q slots in all).
// ---------------------------------------------------------------------------
struct SplitOp {
  int64_t off;    // first row among the running operators' rows
  int64_t pofs;   // offset of the dot-product partial sums (ncols x nslot)
  int64_t slot0;  // first norm partial sum
  int bfirst, nslot;
};

struct RowSplit {
  const SplitOp* sp;
  const int64_t* TG;  // rows of the running operators, blocks that share them
  int nops;
};

// exclusive prefix sum over the block (blockDim.x a multiple of 32, at most
// 1024); *total gets the sum
__device__ int64_t block_scan(int64_t v, int64_t* s_warp, int64_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int64_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int64_t t = lane < nw ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < nw) s_warp[lane] = t;  // inclusive over warps
  }
  __syncthreads();
  const int64_t before = (warp > 0 ? s_warp[warp - 1] : 0) + x - v;
  *total = s_warp[nw - 1];
  __syncthreads();
  return before;
}

// the block holding row r: the largest b with b T / G <= r
__device__ __forceinline__ int split_owner(int64_t r, int64_t T, int G) {
  int64_t b = r * G / T;
  while (b + 1 < G && (b + 1) * T / G <= r) ++b;
  while (b > 0 && b * T / G > r) --b;
  return (int)b;
}

// The running operators' row offsets, blocks and partial-sum slots, by one
// whole block.  The grid's first G' = min(G, ceil(T / 128)) blocks share the
// rows, so each has at least one and every slot of an operator is written.
// The stop flags are read past L1: in k_bfinish other blocks have just set
// them.
__device__ void split_rows_dev(const BOp* __restrict__ ops, int nops, int Gmax, int ncap,
                               const int* done, SplitOp* __restrict__ sp,
                               int64_t* __restrict__ TG) {
  __shared__ int64_t s_warp[32];
  const int per = (nops + (int)blockDim.x - 1) / (int)blockDim.x;
  const int q0 = min(nops, (int)threadIdx.x * per), q1 = min(nops, q0 + per);
  int64_t loc = 0;
  for (int q = q0; q < q1; ++q) loc += __ldcg(done + q) ? 0 : ops[q].D;
  int64_t T = 0;
  int64_t off = block_scan(loc, s_warp, &T);
  const int G = (int)max((int64_t)1, min((int64_t)Gmax, (T + 127) / 128));
  int64_t nsl = 0;
  for (int q = q0; q < q1; ++q) {
    const int64_t d = __ldcg(done + q) ? 0 : ops[q].D;
    SplitOp o;
    o.off = off;
    o.pofs = 0;
    o.slot0 = 0;
    if (d > 0) {
      o.bfirst = split_owner(off, T, G);
      o.nslot = split_owner(off + d - 1, T, G) - o.bfirst + 1;
    } else {
      o.bfirst = 0;
      o.nslot = 0;
    }
    sp[q] = o;
    nsl += o.nslot;
    off += d;
  }
  int64_t nslot_all = 0;
  int64_t s0 = block_scan(nsl, s_warp, &nslot_all);
  for (int q = q0; q < q1; ++q) {
    sp[q].slot0 = s0;
    sp[q].pofs = s0 * ncap;
    s0 += sp[q].nslot;
  }
  if (threadIdx.x == 0) {
    TG[0] = T;
    TG[1] = G;
  }
}

// the split before the first step (one block of 1024 threads); later steps
// get theirs from the last block of k_bfinish
__global__ void __launch_bounds__(1024) k_bsplit(const BOp* __restrict__ ops, int nops, int Gmax,
                                                 int ncap, const int* __restrict__ done,
                                                 SplitOp* __restrict__ sp, int64_t* __restrict__ TG) {
  split_rows_dev(ops, nops, Gmax, ncap, done, sp, TG);
}

template <class F>
__device__ __forceinline__ void for_block_rows(const BOp* __restrict__ ops, RowSplit rs, F&& f) {
  const int64_t T = rs.TG[0], G = rs.TG[1];
  if ((int64_t)blockIdx.x >= G) return;
  const int64_t gb = (int64_t)blockIdx.x * T / G;
  const int64_t ge = (int64_t)(blockIdx.x + 1) * T / G;
  if (gb >= ge) return;
  int lo = 0, hi = rs.nops - 1;  // the last operator starting at or before gb
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (rs.sp[mid].off <= gb) lo = mid;
    else hi = mid - 1;
  }
  for (int q = lo; q < rs.nops; ++q) {
    const SplitOp& s = rs.sp[q];
    if (s.off >= ge) break;
    if (s.nslot == 0) continue;  // stopped
    const BOp& o = ops[q];
    const int64_t a = max(gb, s.off), b = min(ge, s.off + o.D);
    if (a < b) f(q, o, a - s.off, b - s.off, (int)blockIdx.x - s.bfirst, s);
  }
}

// loads of the Krylov vectors: each is used once per kernel, so it leaves L1 to
// the vectors every column is combined with
__device__ __forceinline__ double lv(const double* p) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 lv(const double2* p) {
  double2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float lv(const float* p) {
  float v;
  asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 lv(const float2* p) {
  float2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 wide(double v) { return make_double2(v, 0.0); }
__device__ __forceinline__ double2 wide(double2 v) { return v; }
__device__ __forceinline__ double2 wide(float v) { return make_double2((double)v, 0.0); }
__device__ __forceinline__ double2 wide(float2 v) { return make_double2((double)v.x, (double)v.y); }

// ---------------------------------------------------------------------------
// Gram-Schmidt twice with two reads of V per step.  Each sweep has to know all
// its dot products before it updates, so two sweeps of one vector read V four
// times (three with the middle update and dot products fused).  Here the second
// sweep of v_j waits for the first sweep of the next vector (delayed
// re-orthogonalisation, as in Bielich, Langou, Thomas, Swirydowicz, Yamazaki and
// Boman, "Low-synch Gram-Schmidt with delayed reorthogonalization for Krylov
// solvers", 2022).  With u = v_j after one sweep, normalised, V the final columns
// before it and wt = H u, one read of V gives s = V^H u and r = V^H wt (and
// |u|^2, u^H wt from column j).  Then, with a^2 = |u|^2 - |s|^2,
//   q = (u - V s) / a                                     (v_j, final)
//   H q = (wt - V T s - beta_{j-1} s_{j-1} q) / a         (H V = V T + beta q e^T)
//   g = q^H wt / a = (u^H wt - s^H r) / a^2
//   alpha_j = Re(g - beta_{j-1} s_{j-1} / a)
//   H q - V V^H H q - q q^H H q = (wt - g u - V (r - g s)) / a
// so the second read of V updates both vectors.  V^H H q is exact to the
// rounding of the recurrence times |s|, which one sweep leaves at eps |H| / beta.
// In a space that V already spans (a sector with fewer levels than steps) u is the
// rounding of the first sweep, s takes in all of it and a is close to zero: beta a,
// the length the second sweep leaves, then ends the run (k_breduce2) by the rule
// that a vector orthogonalised twice in its own step would meet there.
// Mean over the 131 steps of 96 random-field chains of 12 to 20 sites (FP64):
// 194 + 247 + 173 us for the three passes before, 171 + 177 us for the two here,
// which is the HBM rate (two blocks of 128 registers per SM; three of 80 spill:
// 199 + 170; four of 64: slower in every case measured).
// ---------------------------------------------------------------------------

// part[pofs_q + c nslot_q + slot] = sum over the block's rows of conj(V_q[r, c])
// V_q[r, j], and the same with wt_q at part + pstride, c <= j.  Bound by HBM: a
// warp takes four columns over its rows and reduces once at the end, all loads of
// RU rows of them in flight; the two vectors every warp needs stay in L1.  With
// few columns the warps split the rows as well (up to eight ways) and meet in
// shared memory.
template <class VV>
__global__ void __launch_bounds__(256, kSplitBlocks) k_rdots2(const BOp* __restrict__ ops, RowSplit rs,
                                                const VV* __restrict__ V,
                                                const VV* __restrict__ wt,
                                                double2* __restrict__ part, int64_t pstride,
                                                const int* __restrict__ step,
                                                const int* __restrict__ done) {
  constexpr bool CX = IsCx<VV>::v;
  constexpr int NC = CX ? 2 : 1;
  constexpr int RU = sizeof(VV) == 16 ? 2 : 4;
  __shared__ double2 s_part[256][2];
  const int ncols = *step + 1, ng = (ncols + 3) / 4;
  const int nsub = ng <= 8 ? 8 : (ng <= 16 ? 4 : (ng <= 32 ? 2 : 1));
  const int pad = 256 / nsub;  // columns of a row share in s_part
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for_block_rows(ops, rs, [&](int q, const BOp& o, int64_t r0, int64_t r1, int slot, const SplitOp& sq) {
    if (done[q]) return;
    const int64_t D = o.D, rows = r1 - r0;
    const VV* Vq = V + o.voff;
    const VV* x = Vq + (int64_t)(ncols - 1) * D;
    const VV* y = wt + o.woff;
    for (int un = warp; un < ng * nsub; un += 8) {
      const int cg = un % ng, sub = un / ng;
      const int64_t a = r0 + rows * sub / nsub, b = r0 + rows * (sub + 1) / nsub;
      const VV* Vc[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) Vc[u] = Vq + (int64_t)min(4 * cg + u, ncols - 1) * D;
      double fs[4 * NC], fr[4 * NC];
#pragma unroll
      for (int u = 0; u < 4 * NC; ++u) fs[u] = fr[u] = 0.0;
      auto pass = [&](int64_t rb, bool full) {
        VV v[4][RU], xv[RU], yv[RU];
#pragma unroll
        for (int k = 0; k < RU; ++k) {
          const int64_t r = rb + 32 * k;
          const bool on = full || r < b;
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u][k] = on ? lv(Vc[u] + r) : VV{};
          xv[k] = on ? x[r] : VV{};
          yv[k] = on ? y[r] : VV{};
        }
#pragma unroll
        for (int k = 0; k < RU; ++k) {
          const double2 xw = wide(xv[k]), yw = wide(yv[k]);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const double2 c = wide(v[u][k]);
            if constexpr (CX) {
              fs[2 * u] += c.x * xw.x + c.y * xw.y;
              fs[2 * u + 1] += c.x * xw.y - c.y * xw.x;
              fr[2 * u] += c.x * yw.x + c.y * yw.y;
              fr[2 * u + 1] += c.x * yw.y - c.y * yw.x;
            } else {
              fs[u] += c.x * xw.x;
              fr[u] += c.x * yw.x;
            }
          }
        }
      };
      int64_t rb = a + lane;
      for (; rb - lane + 32 * RU <= b; rb += 32 * RU) pass(rb, true);
      if (rb - lane < b) pass(rb, false);
      // lane 4 v ends with value v: the sums of a column (and vector) in turn
      auto put = [&](int col, int vec, int comp, double t) {
        if (col >= ncols) return;
        if (nsub > 1) {
          reinterpret_cast<double*>(&s_part[sub * pad + col][vec])[comp] = t;
          if (!CX) reinterpret_cast<double*>(&s_part[sub * pad + col][vec])[1] = 0.0;
        } else {
          double* d = reinterpret_cast<double*>(part + (vec ? pstride : 0) + sq.pofs +
                                                (int64_t)col * sq.nslot + slot);
          d[comp] = t;
          if (!CX) d[1] = 0.0;
        }
      };
      const int vi = lane >> 2;
      if constexpr (CX) {
        const double ts = wsum8(fs, lane), tr = wsum8(fr, lane);
        if ((lane & 3) == 0) {
          put(4 * cg + (vi >> 1), 0, vi & 1, ts);
          put(4 * cg + (vi >> 1), 1, vi & 1, tr);
        }
      } else {
        double f[8];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          f[u] = fs[u];
          f[u + 4] = fr[u];
        }
        const double t = wsum8(f, lane);
        if ((lane & 3) == 0) put(4 * cg + (vi & 3), vi >> 2, 0, t);
      }
    }
    if (nsub > 1) {
      __syncthreads();
      for (int e = threadIdx.x; e < 2 * ncols; e += blockDim.x) {
        const int c = e >> 1, vec = e & 1;
        double2 t = make_double2(0.0, 0.0);
        for (int sub = 0; sub < nsub; ++sub) {
          t.x += s_part[sub * pad + c][vec].x;
          t.y += s_part[sub * pad + c][vec].y;
        }
        part[(vec ? pstride : 0) + sq.pofs + (int64_t)c * sq.nslot + slot] = t;
      }
      __syncthreads();  // s_part is free for the next piece
    }
  });
}

__device__ __forceinline__ double bsum256(double v, double* sh) {  // all threads get the sum
  v = wsum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int k = 0; k < 8; ++k) t += sh[k];
  return t;
}

constexpr double kBreakdown = 1.4901161193847656e-08;  // sqrt(eps(Float64))
// Part of |u|^2 outside the span of V below which column u is taken as inside it:
// dividing by a would raise u's rounding (6e-8 in FP32 storage) by more than 100.
// In storage of either width a vector whose beta is above the breakdown rule's
// limit leaves 1 - O(eps |H| / beta)^2.
constexpr double kInSpan = 1e-4;

// Sums operator q's slots (one warp per column; both vectors), and in the last
// block of the operator turns them into the update's coefficients:
// cs = s, ce = r - g s, scal = {1 / a, g}, and alpha_j; or stops the operator with
// j steps and beta_{j-1} = 0 when the second sweep leaves nothing of column j.
// `closing`: only that test, for the column past the last step.
__global__ void __launch_bounds__(256) k_breduce2(const SplitOp* __restrict__ sp, int ncap, int m,
                                                  const double2* __restrict__ part, int64_t pstride,
                                                  double2* __restrict__ cs, double2* __restrict__ ce,
                                                  double4* __restrict__ scal,
                                                  double* __restrict__ alpha,
                                                  double* __restrict__ beta,
                                                  unsigned* __restrict__ cnt,
                                                  const int* __restrict__ step, int* done,
                                                  int closing) {
  __shared__ bool s_last;
  __shared__ double sh[8];
  const int q = blockIdx.y;
  if (done[q]) return;
  const int j = *step, lane = threadIdx.x & 31;
  const SplitOp& o = sp[q];
  double2* csq = cs + (int64_t)q * ncap;
  double2* ceq = ce + (int64_t)q * ncap;
  for (int c = blockIdx.x * 8 + (threadIdx.x >> 5); c <= j; c += gridDim.x * 8) {
    const double2* ps = part + o.pofs + (int64_t)c * o.nslot;
    const double2* pr = ps + pstride;
    // independent loads in flight a lane (a large operator has hundreds of
    // slots and few columns, so few warps carry the whole reduction)
    double2 a[2], b[2];
    a[0] = a[1] = b[0] = b[1] = make_double2(0.0, 0.0);
    int k = lane;
    for (; k + 32 < o.nslot; k += 64) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const double2 v = ps[k + 32 * u], w = pr[k + 32 * u];
        a[u].x += v.x;
        a[u].y += v.y;
        b[u].x += w.x;
        b[u].y += w.y;
      }
    }
    if (k < o.nslot) {
      const double2 v = ps[k], w = pr[k];
      a[0].x += v.x;
      a[0].y += v.y;
      b[0].x += w.x;
      b[0].y += w.y;
    }
    const double sx = wsum(a[0].x + a[1].x), sy = wsum(a[0].y + a[1].y);
    const double rx = wsum(b[0].x + b[1].x), ry = wsum(b[0].y + b[1].y);
    if (lane == 0) {
      csq[c] = make_double2(sx, sy);
      ceq[c] = make_double2(rx, ry);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // this block's sums before its count
    s_last = atomicAdd(cnt + q, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // of the step before (read here, beside the loads of the sums)
  const double aprev = j > 0 ? alpha[(int64_t)q * m + j - 1] : 0.0;
  const double bprev = j > 0 ? beta[(int64_t)q * m + j - 1] : 0.0;
  double ss = 0.0, hx = 0.0, hy = 0.0;  // |s|^2 and s^H r over the final columns
  for (int c = threadIdx.x; c < j; c += blockDim.x) {
    const double2 s = __ldcg(csq + c), r = __ldcg(ceq + c);
    ss += s.x * s.x + s.y * s.y;
    hx += s.x * r.x + s.y * r.y;
    hy += s.x * r.y - s.y * r.x;
  }
  ss = bsum256(ss, sh);
  hx = bsum256(hx, sh);
  hy = bsum256(hy, sh);
  const double2 uu = __ldcg(csq + j), uw = __ldcg(ceq + j);
  const double a2 = uu.x - ss, root = sqrt(a2 < 0.0 ? 0.0 : a2);  // (NaN stays)
  if (j > 0) {  // (NaN runs on)
    if (a2 <= kInSpan * uu.x || bprev * root <= kBreakdown * fmax(1.0, fabs(aprev))) {
      if (threadIdx.x == 0) {
        beta[(int64_t)q * m + j - 1] = 0.0;
        done[q] = 2;  // (every block of the operator has read the flag: all have counted)
        cnt[q] = 0;
      }
      return;
    }
  }
  if (closing) {
    if (threadIdx.x == 0) cnt[q] = 0;
    return;
  }
  const double inva = 1.0 / root, gx = (uw.x - hx) / a2, gy = (uw.y - hy) / a2;
  for (int c = threadIdx.x; c < j; c += blockDim.x) {
    const double2 s = __ldcg(csq + c), r = __ldcg(ceq + c);
    ceq[c] = make_double2(r.x - (gx * s.x - gy * s.y), r.y - (gx * s.y + gy * s.x));
  }
  if (threadIdx.x == 0) {
    const double last = j > 0 ? bprev * __ldcg(csq + j - 1).x * inva : 0.0;
    alpha[(int64_t)q * m + j] = gx - last;
    scal[q] = make_double4(inva, gx, gy, 0.0);
    cnt[q] = 0;
  }
}

// V_q[:, j] = (V_q[:, j] - V_q cs) / a (final) and w_q = (wt_q - g V_q[:, j] - V_q
// ce) / a over the block's rows, columns below j, newest first: k_rdots2 has read
// the newest columns last and reads the oldest first in the next step, so each
// kernel starts with what the other has left in L2.  A thread holds four rows of
// both vectors and loads 128 bytes a pass; the coefficients go through shared
// memory 128 columns at a time.  normpart[slot0_q + slot] = sum |w|^2.
template <class VV, class WD>
__global__ void __launch_bounds__(256, kSplitBlocks) k_rupdate2(const BOp* __restrict__ ops, RowSplit rs,
                                                  int ncap, VV* __restrict__ V,
                                                  const double2* __restrict__ cs,
                                                  const double2* __restrict__ ce,
                                                  const double4* __restrict__ scal,
                                                  const VV* __restrict__ wt, WD* __restrict__ w,
                                                  double* __restrict__ normpart,
                                                  const int* __restrict__ step,
                                                  const int* __restrict__ done) {
  constexpr bool CX = IsCx<VV>::v;
  constexpr int R = 4, U = 128 / (R * (int)sizeof(VV)), CH = 128;
  static_assert(CH % U == 0, "chunks hold whole passes");
  __shared__ double2 s_k[CH * (CX ? 2 : 1)];  // real: {cs, ce}; complex: cs, ce
  __shared__ double s_n[8];
  const int j = *step, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for_block_rows(ops, rs, [&](int q, const BOp& o, int64_t r0, int64_t r1, int slot, const SplitOp& sq) {
    if (done[q]) return;
    const int64_t D = o.D;
    VV* Vq = V + o.voff;
    VV* uj = Vq + (int64_t)j * D;
    const double4 k4 = scal[q];
    double nrm = 0.0;
    for (int64_t rb0 = r0; rb0 < r1; rb0 += 256 * R) {
      const int64_t rb = rb0 + threadIdx.x;
      const bool full = rb0 + 256 * R <= r1;
      double2 aq[R], au[R];
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int64_t r = rb + 256 * k;
        const bool on = full || r < r1;
        const double2 u = on ? l2(uj + r) : make_double2(0.0, 0.0);
        const double2 h = on ? l2(wt + o.woff + r) : make_double2(0.0, 0.0);
        aq[k] = u;
        au[k].x = h.x - k4.y * u.x;
        au[k].y = 0.0;
        if constexpr (CX) {
          au[k].x += k4.z * u.y;
          au[k].y = h.y - (k4.y * u.y + k4.z * u.x);
        }
      }
      for (int c1 = j; c1 > 0; c1 = (c1 - 1) / CH * CH) {  // columns [c0, c1) of one chunk
        const int c0 = (c1 - 1) / CH * CH;
        const int npad = (c1 - c0 + U - 1) / U * U;
        __syncthreads();  // the previous chunk's coefficients are read
        for (int e = threadIdx.x; e < npad; e += blockDim.x) {
          const int c = c0 + e;
          const double2 s = c < c1 ? cs[(int64_t)q * ncap + c] : make_double2(0.0, 0.0);
          const double2 t = c < c1 ? ce[(int64_t)q * ncap + c] : make_double2(0.0, 0.0);
          if constexpr (CX) {
            s_k[2 * e] = s;
            s_k[2 * e + 1] = t;
          } else {
            s_k[e] = make_double2(s.x, t.x);
          }
        }
        __syncthreads();
        for (int e = npad - U; e >= 0; e -= U) {
          VV v[U][R];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const VV* Vc = Vq + (int64_t)min(c0 + e + u, c1 - 1) * D + rb;
#pragma unroll
            for (int k = 0; k < R; ++k) v[u][k] = full || rb + 256 * k < r1 ? lv(Vc + 256 * k) : VV{};
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if constexpr (CX) {
              const double2 s = s_k[2 * (e + u)], t = s_k[2 * (e + u) + 1];
#pragma unroll
              for (int k = 0; k < R; ++k) {
                const double2 x = wide(v[u][k]);
                aq[k].x -= x.x * s.x - x.y * s.y;
                aq[k].y -= x.x * s.y + x.y * s.x;
                au[k].x -= x.x * t.x - x.y * t.y;
                au[k].y -= x.x * t.y + x.y * t.x;
              }
            } else {
              const double2 st = s_k[e + u];
#pragma unroll
              for (int k = 0; k < R; ++k) {
                const double x = wide(v[u][k]).x;
                aq[k].x -= x * st.x;
                au[k].x -= x * st.y;
              }
            }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int64_t r = rb + 256 * k;
        if (full || r < r1) {
          s2(uj + r, make_double2(aq[k].x * k4.x, aq[k].y * k4.x));
          const double2 t = make_double2(au[k].x * k4.x, au[k].y * k4.x);
          s2(w + o.woff + r, t);
          nrm += t.x * t.x + (CX ? t.y * t.y : 0.0);
        }
      }
    }
    nrm = wsum(nrm);
    __syncthreads();
    if (lane == 0) s_n[warp] = nrm;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int k = 0; k < 8; ++k) t += s_n[k];
      normpart[sq.slot0 + slot] = t;
    }
  });
}

// w_q = the start vector, normpart = sum |w|^2 over the block's rows
template <class WD>
__global__ void __launch_bounds__(256) k_rstart(const BOp* __restrict__ ops, RowSplit rs,
                                                const WD* __restrict__ start, WD* __restrict__ w,
                                                double* __restrict__ normpart,
                                                const int* __restrict__ done) {
  __shared__ double s_n[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for_block_rows(ops, rs, [&](int q, const BOp& o, int64_t r0, int64_t r1, int slot, const SplitOp& sq) {
    if (done[q]) return;
    double nrm = 0.0;
    for (int64_t r = r0 + threadIdx.x; r < r1; r += 256) {
      const double2 v = l2(start + o.woff + r);
      s2(w + o.woff + r, v);
      nrm += v.x * v.x + v.y * v.y;
    }
    nrm = wsum(nrm);
    __syncthreads();
    if (lane == 0) s_n[warp] = nrm;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int k = 0; k < 8; ++k) t += s_n[k];
      normpart[sq.slot0 + slot] = t;
    }
  });
}

// per operator: beta_j, breakdown, 1/beta (one block per operator; alpha_j is
// there already).
// The last block to finish then closes the step: it splits the rows of the
// operators still running for the next step's reorthogonalisation kernels
// and advances the step counter (every block has read it by then).
__global__ void __launch_bounds__(256) k_bfinish(const BOp* __restrict__ ops, int nops, int Gmax,
                                                 SplitOp* __restrict__ sp,
                                                 int64_t* __restrict__ TG,
                                                 unsigned* __restrict__ nfinished, int ncap, int m,
                                                 const double* __restrict__ normpart,
                                                 double* __restrict__ alpha,
                                                 double* __restrict__ beta,
                                                 double* __restrict__ invb,
                                                 int* __restrict__ nsteps,
                                                 int* __restrict__ step,
                                                 int* __restrict__ done, int setup) {
  const int q = blockIdx.x;
  const int j = *step;
  __shared__ double sh[8];
  __shared__ bool s_last;
  if (!done[q]) {
    const SplitOp o = sp[q];
    double s = 0.0;
    for (int k = threadIdx.x; k < o.nslot; k += blockDim.x) s += normpart[o.slot0 + k];
    s = wsum(s);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double n2 = 0.0;
      for (int k = 0; k < 8; ++k) n2 += sh[k];
      const double nrm = sqrt(n2);
      if (setup) {  // starting vector: zero or non-finite norm is an error for this operator
        if (!isfinite(nrm)) { done[q] = 4; invb[q] = 0.0; }
        else if (!(nrm > 0.0)) { done[q] = 3; invb[q] = 0.0; }
        else invb[q] = 1.0 / nrm;
        alpha[(int64_t)q * m] = nrm;  // for the Krylov driver; step 0 overwrites it
      } else {
        const double a = alpha[(int64_t)q * m + j];
        beta[(int64_t)q * m + j] = nrm;
        nsteps[q] = j + 1;
        if (nrm <= kBreakdown * fmax(1.0, fabs(a))) {
          beta[(int64_t)q * m + j] = 0.0;
          done[q] = 2;
          invb[q] = 0.0;
        } else {
          invb[q] = 1.0 / nrm;
        }
      }
    }
  }
  if (threadIdx.x == 0) {
    __threadfence();  // this block's stop flag before its count
    s_last = atomicAdd(nfinished, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  split_rows_dev(ops, nops, Gmax, ncap, done, sp, TG);
  if (threadIdx.x == 0) {
    *nfinished = 0;
    *step = j + 1;
  }
}

// V_q[:, j+1] = w_q / beta (skipped past the last column); k_bfinish has
// advanced the step counter to j + 1
template <class WV, class VV>
__global__ void __launch_bounds__(256) k_bscale(const BOp* __restrict__ ops,
                                                const int* __restrict__ tile2op, int ncap,
                                                const WV* __restrict__ w, VV* __restrict__ V,
                                                const double* __restrict__ invb,
                                                const int* __restrict__ step,
                                                const int* __restrict__ done) {
  const int q = tile2op[blockIdx.x];
  if (done[q]) return;
  const BOp& o = ops[q];
  const int col = *step;
  if (col >= ncap) return;
  const int64_t r = (blockIdx.x - o.tile0) * (int64_t)kTile + threadIdx.x;
  if (r >= o.D) return;
  const double sc = invb[q];
  const double2 v = l2(w + o.woff + r);
  s2(V + o.voff + (int64_t)col * o.D + r, make_double2(v.x * sc, v.y * sc));
}

// out_q = V_q[:, 0:nc_q] c_q (coefficients per operator, FP64 output)
template <class VV, class OV>
__global__ void __launch_bounds__(256) k_bcombine(const BOp* __restrict__ ops,
                                                  const int* __restrict__ tile2op, int ncap,
                                                  const VV* __restrict__ V,
                                                  const double2* __restrict__ c,
                                                  const int* __restrict__ ncols,
                                                  OV* __restrict__ out) {
  const int q = tile2op[blockIdx.x];
  const BOp& o = ops[q];
  const int64_t r = (blockIdx.x - o.tile0) * (int64_t)kTile + threadIdx.x;
  if (r >= o.D) return;
  const int nc = ncols[q];
  double ar = 0.0, ai = 0.0;
  for (int k = 0; k < nc; ++k) {
    const double2 v = l2(V + o.voff + (int64_t)k * o.D + r);
    const double2 ck = c[(int64_t)q * ncap + k];
    ar += v.x * ck.x - v.y * ck.y;
    ai += v.x * ck.y + v.y * ck.x;
  }
  s2(out + o.woff + r, make_double2(ar, ai));
}

namespace {

size_t esz(int dt) { return (dt == EDK_F64 || dt == EDK_C64) ? 8 : (dt == EDK_C128 ? 16 : 4); }

template <class F> edk_status with_vt(int dt, F&& f) {
  switch (dt) {
    case EDK_F64: return f((double*)nullptr);
    case EDK_C128: return f((double2*)nullptr);
    case EDK_F32: return f((float*)nullptr);
    case EDK_C64: return f((float2*)nullptr);
  }
  set_error("batch: unknown dtype");
  return EDK_INVALID_ARG;
}

double wall() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// A batch of operators sharing a lookup kind, kernel family and storage type.
struct BatchEngine {
  int nops = 0, vdt = EDK_F64, wdt = EDK_F64, ncap = 0, m = 0;
  int bk = 0;
  bool ff = false;
  bool plan = false;  // every operator carries a row plan (rank-searched sectors)
  bool plan_nn_all = false;  // ... and is one nearest-neighbour family of equal values
  bool sell = false;
  const edk_operator* pauli = nullptr;  // a batch of one on the Pauli-string kernel
  // a batch of one whose product has no batched kernel (symmetry groups, more
  // than 32 sites): launched step by step through apply_device
  edk_operator* direct = nullptr;
  int hj = 0;  // the next step, where steps are launched one by one
  int64_t nsblk = 0;
  cudaStream_t st = nullptr;
  std::vector<BOp> hops;
  std::vector<int64_t> Ds;
  int64_t ntiles = 0, totalD = 0;
  int G = 1;             // blocks of the reorthogonalisation grid
  int nsm = 1;           // SMs of the device
  DevBuf maps, work;  // what the parts below lie in
  DevBuf dops, tile2op, sblk2op, splitops, splitT, nfin, V, w, wt, part, cs, ce, scal, cnt,
      normpart, alpha, beta, invb, done, step, nsteps, cbuf, cnc;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t gexec = nullptr;
  bool graph_ok = false;
  cudaStream_t side = nullptr;     // the first operator's copy stream
  cudaEvent_t checked = nullptr;   // the last convergence check has run

  ~BatchEngine() {
    if (checked) cudaEventDestroy(checked);
    if (gexec) cudaGraphExecDestroy(gexec);
    if (graph) cudaGraphDestroy(graph);
  }

  // The operators as they are now: their device records, tile maps and the
  // kernel of the product.  Called again (with the stream idle) when one of them
  // has been materialised, cleared or configured since.
  edk_status load(const std::vector<edk_operator*>& ops, int lookup_kind, bool use_ff) {
    if (gexec) cudaGraphExecDestroy(gexec);
    if (graph) cudaGraphDestroy(graph);
    gexec = nullptr;
    graph = nullptr;
    graph_ok = false;
    hops.clear();
    Ds.clear();
    ntiles = nsblk = 0;
    pauli = nullptr;
    // row plans (built here, outside any capture) when the sectors are ranked
    plan = use_ff && (lookup_kind == BK_TRANS0_RANK || lookup_kind == BK_TRANS_RANK ||
                      lookup_kind == BK_TRANSPAR_RANK || lookup_kind == BK_PROJ_RANK);
    plan_nn_all = plan;
    for (auto* op : ops) plan = plan && plan_applies(op);
    plan_nn_all = plan;
    if (plan) EDK_RETURN_IF(plan_ensure(ops, st));
    for (auto* op : ops) {
      if (!plan) break;
      plan = op->plan_state == 1;
      plan_nn_all = plan_nn_all && plan_nn(*reinterpret_cast<const FFParams*>(op->ff_params.data()));
    }
    bk = lookup_kind;
    ff = use_ff;
    std::vector<int> t2o, s2o;
    int64_t voff = 0, woff = 0;
    sell = true;
    for (auto* op : ops) sell = sell && op->sell_ok;
    for (int q = 0; q < nops; ++q) {
      edk_operator* op = ops[q];
      BOp o{};
      o.b = op->b->dev;
      o.b.bk = bk;
      o.op = op->dev;
      if (use_ff) std::memcpy(&o.ff, op->ff_params.data(), sizeof(FFParams));
      o.D = op->b->D;
      o.ntile = (int)((o.D + kTile - 1) / kTile);
      o.voff = voff;
      o.woff = woff;
      o.tile0 = ntiles;
      o.sblk0 = nsblk;
      if (sell) {
        const int64_t nb = (op->dev.sell.nslices + 7) / 8;
        for (int64_t k = 0; k < nb; ++k) s2o.push_back(q);
        nsblk += nb;
      }
      for (int k = 0; k < o.ntile; ++k) t2o.push_back(q);
      ntiles += o.ntile;
      voff += o.D * ncap;
      woff += o.D;
      hops.push_back(o);
      Ds.push_back(o.D);
    }
    totalD = woff;
    if (nops == 1 && !sell && ops[0]->pauli_ok && ops[0]->use_ff) pauli = ops[0];
    DevParts parts;
    parts.add(dops, hops.size() * sizeof(BOp));
    parts.add(tile2op, t2o.size() * 4);
    if (sell) parts.add(sblk2op, std::max<size_t>(s2o.size(), 1) * 4);
    EDK_RETURN_IF(parts.alloc(maps, st));
    EDK_TRY_CUDA(cudaMemcpyAsync(dops.p, hops.data(), hops.size() * sizeof(BOp),
                                 cudaMemcpyHostToDevice, st));
    EDK_TRY_CUDA(cudaMemcpyAsync(tile2op.p, t2o.data(), t2o.size() * 4, cudaMemcpyHostToDevice, st));
    if (sell && !s2o.empty())
      EDK_TRY_CUDA(cudaMemcpyAsync(sblk2op.p, s2o.data(), s2o.size() * 4, cudaMemcpyHostToDevice, st));
    return EDK_OK;
  }

  edk_status init(const std::vector<edk_operator*>& ops, int vdtype, int m_, int lookup_kind,
                  bool use_ff, cudaStream_t s) {
    nops = (int)ops.size();
    if (nops > 65535) {
      set_error("batch Lanczos: at most 65535 operators per batch");
      return EDK_UNSUPPORTED;
    }
    vdt = vdtype;
    wdt = (vdt == EDK_C128 || vdt == EDK_C64) ? EDK_C128 : EDK_F64;
    m = m_;
    ncap = m + 1;
    st = s;
    EDK_RETURN_IF(load(ops, lookup_kind, use_ff));
    if (!ops[0]->cstream)
      EDK_TRY_CUDA(cudaStreamCreateWithFlags(&ops[0]->cstream, cudaStreamNonBlocking));
    side = ops[0]->cstream;
    EDK_TRY_CUDA(cudaEventCreateWithFlags(&checked, cudaEventDisableTiming));
    EDK_RETURN_IF(split_rows());
    DevParts parts;
    parts.add(V, (size_t)totalD * ncap * esz(vdt));
    parts.add(w, (size_t)totalD * esz(wdt));
    parts.add(wt, (size_t)totalD * esz(vdt));
    // a block meets at most one operator more than it starts in: G + nops slots
    parts.add(part, 2 * (size_t)(G + nops) * ncap * sizeof(double2));
    parts.add(splitops, (size_t)nops * sizeof(SplitOp));
    parts.add(splitT, 2 * sizeof(int64_t));
    parts.add(nfin, sizeof(unsigned));
    parts.add(cs, (size_t)nops * ncap * sizeof(double2));
    parts.add(ce, (size_t)nops * ncap * sizeof(double2));
    parts.add(scal, (size_t)nops * sizeof(double4));
    parts.add(cnt, (size_t)nops * sizeof(unsigned));
    parts.add(normpart, (size_t)(G + nops) * sizeof(double));
    parts.add(alpha, (size_t)nops * m * sizeof(double));
    parts.add(beta, (size_t)nops * m * sizeof(double));
    parts.add(invb, (size_t)nops * sizeof(double));
    parts.add(done, (size_t)nops * sizeof(int));
    parts.add(nsteps, (size_t)nops * sizeof(int));
    parts.add(step, sizeof(int));
    parts.add(cbuf, (size_t)nops * ncap * sizeof(double2));
    parts.add(cnc, (size_t)nops * sizeof(int));
    EDK_RETURN_IF(parts.alloc(work, st));
    EDK_TRY_CUDA(cudaMemsetAsync(nfin.p, 0, sizeof(unsigned), st));
    EDK_TRY_CUDA(cudaMemsetAsync(cnt.p, 0, (size_t)nops * sizeof(unsigned), st));
    EDK_TRY_CUDA(cudaMemsetAsync(alpha.p, 0, (size_t)nops * m * sizeof(double), st));
    EDK_TRY_CUDA(cudaMemsetAsync(beta.p, 0, (size_t)nops * m * sizeof(double), st));
    return EDK_OK;
  }

  // Size the reorthogonalisation grid to what is resident at once.
  edk_status split_rows() {
    int dev = 0;
    EDK_TRY_CUDA(cudaGetDevice(&dev));
    EDK_TRY_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    int per_sm = 0;
    edk_status s = with_vt(vdt, [&](auto vp) -> edk_status {
      using VV = std::remove_pointer_t<decltype(vp)>;
      return with_vt(wdt, [&](auto wp) -> edk_status {
        using WD = std::remove_pointer_t<decltype(wp)>;
        int n[2] = {0, 0};
        const auto kd = k_rdots2<VV>;
        const auto ku = k_rupdate2<VV, WD>;
        EDK_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n[0], kd, 256, 0));
        EDK_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n[1], ku, 256, 0));
        per_sm = std::min(n[0], n[1]);
        return EDK_OK;
      });
    });
    EDK_RETURN_IF(s);
    // at least 256 rows a block, at most the resident blocks
    const int64_t want = std::max<int64_t>(1, (totalD + 255) / 256);
    G = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)nsm * std::max(per_sm, 1), want));
    return EDK_OK;
  }

  const BOp* d_ops() const { return dops.as<BOp>(); }

  edk_status launch_apply() {
    if (direct)
      return apply_device(direct, vdt, (const char*)V.p + (size_t)hj * totalD * esz(vdt), wt.p, 1,
                          totalD, totalD, 0, st);
    const int* t2o = tile2op.as<int>();
    const int* stp = step.as<int>();
    const int* dn = done.as<int>();
    return with_vt(vdt, [&](auto vp) -> edk_status {
      using VT = std::remove_pointer_t<decltype(vp)>;
      const VT* Vv = V.as<VT>();
      VT* wv = wt.as<VT>();
      if (sell) {
        if (nsblk > 0)
          k_bapply_sell<VT><<<(unsigned)nsblk, 256, 0, st>>>(d_ops(), sblk2op.as<int>(), Vv, wv,
                                                             stp, dn);
        return EDK_OK;
      }
      if (pauli) return apply_pauli(pauli, vdt, Vv, wv, 1, totalD, totalD, 0, st, stp, dn);
      if (plan) {
        switch (bk) {
          case BK_PROJ_RANK:
            if (plan_nn_all)
              k_bapply_plan<BK_PROJ_RANK, VT, 1><<<plan_grid(plan_min_blocks<BK_PROJ_RANK, VT>()), 256, 0, st>>>(
                  d_ops(), t2o, ntiles, Vv, wv, stp, dn);
            else
              k_bapply_plan<BK_PROJ_RANK, VT, 2><<<plan_grid(plan_min_blocks<BK_PROJ_RANK, VT>()), 256, 0, st>>>(
                  d_ops(), t2o, ntiles, Vv, wv, stp, dn);
            return EDK_OK;
          case BK_TRANS0_RANK:
            if (plan_nn_all)
              k_bapply_plan<BK_TRANS0_RANK, VT, 1><<<plan_grid(plan_min_blocks<BK_TRANS0_RANK, VT>()), 256, 0, st>>>(
                  d_ops(), t2o, ntiles, Vv, wv, stp, dn);
            else
              k_bapply_plan<BK_TRANS0_RANK, VT, 2><<<plan_grid(plan_min_blocks<BK_TRANS0_RANK, VT>()), 256, 0, st>>>(
                  d_ops(), t2o, ntiles, Vv, wv, stp, dn);
            return EDK_OK;
          case BK_TRANS_RANK:
            if (plan_nn_all)
              k_bapply_plan<BK_TRANS_RANK, VT, 1><<<plan_grid(plan_min_blocks<BK_TRANS_RANK, VT>()), 256, 0, st>>>(
                  d_ops(), t2o, ntiles, Vv, wv, stp, dn);
            else
              k_bapply_plan<BK_TRANS_RANK, VT, 2><<<plan_grid(plan_min_blocks<BK_TRANS_RANK, VT>()), 256, 0, st>>>(
                  d_ops(), t2o, ntiles, Vv, wv, stp, dn);
            return EDK_OK;
          case BK_TRANSPAR_RANK:
            if (plan_nn_all)
              k_bapply_plan<BK_TRANSPAR_RANK, VT, 1><<<plan_grid(plan_min_blocks<BK_TRANSPAR_RANK, VT>()), 256, 0, st>>>(
                  d_ops(), t2o, ntiles, Vv, wv, stp, dn);
            else
              k_bapply_plan<BK_TRANSPAR_RANK, VT, 2><<<plan_grid(plan_min_blocks<BK_TRANSPAR_RANK, VT>()), 256, 0, st>>>(
                  d_ops(), t2o, ntiles, Vv, wv, stp, dn);
            return EDK_OK;
        }
      }
#define EDK_BAPPLY(BK)                                                                       \
  case BK:                                                                                   \
    if (ff) k_bapply_ff<BK, VT><<<(unsigned)ntiles, 256, 0, st>>>(d_ops(), t2o, Vv, wv, stp, dn); \
    else k_bapply_gen<BK, VT><<<(unsigned)ntiles, 256, 0, st>>>(d_ops(), t2o, Vv, wv, stp, dn);  \
    break;
      switch (bk) {
        EDK_BAPPLY(BK_TENSOR)
        EDK_BAPPLY(BK_PROJ_RANK)
        EDK_BAPPLY(BK_PROJ_HASH)
        EDK_BAPPLY(BK_TRANS0)
        case BK_TRANS0_RANK:  // bond-family fast path only (other paths keep the hash)
          k_bapply_ff<BK_TRANS0_RANK, VT><<<(unsigned)ntiles, 256, 0, st>>>(d_ops(), t2o, Vv, wv,
                                                                           stp, dn);
          break;
        case BK_TRANS_RANK:
          k_bapply_ff<BK_TRANS_RANK, VT><<<(unsigned)ntiles, 256, 0, st>>>(d_ops(), t2o, Vv, wv,
                                                                          stp, dn);
          break;
        case BK_TRANSPAR_RANK:
          k_bapply_ff<BK_TRANSPAR_RANK, VT><<<(unsigned)ntiles, 256, 0, st>>>(d_ops(), t2o, Vv,
                                                                             wv, stp, dn);
          break;
        EDK_BAPPLY(BK_TRANS)
        EDK_BAPPLY(BK_TRANSPAR)
        default:
          set_error("batch Lanczos: lookup kind not supported in batches");
          return EDK_UNSUPPORTED;
      }
#undef EDK_BAPPLY
      return EDK_OK;
    });
  }

  // resident grid of the row-plan matvec: per_sm blocks on every SM, at
  // most one block per tile
  unsigned plan_grid(int per_sm) const {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ntiles, (int64_t)nsm * per_sm));
  }

  RowSplit rsplit() const {
    return RowSplit{splitops.as<SplitOp>(), splitT.as<int64_t>(), nops};
  }

  void launch_split() {
    k_bsplit<<<1, 1024, 0, st>>>(d_ops(), nops, G, ncap, done.as<int>(), splitops.as<SplitOp>(),
                                 splitT.as<int64_t>());
  }

  // alpha / beta / stop flags, then (last block) the next step's split and
  // the step counter
  void launch_finish(int setup) {
    k_bfinish<<<nops, 256, 0, st>>>(d_ops(), nops, G, splitops.as<SplitOp>(),
                                    splitT.as<int64_t>(), nfin.as<unsigned>(), ncap, m,
                                    normpart.as<double>(), alpha.as<double>(), beta.as<double>(), invb.as<double>(),
                                    nsteps.as<int>(), step.as<int>(), done.as<int>(), setup);
  }

  // the dot products of column *step and their sums; see k_breduce2 for `closing`
  void launch_dots(int closing) {
    const int64_t pst = (int64_t)(G + nops) * ncap;
    // blocks per operator of the sums: two per SM over all operators
    const int rx = std::max(1, std::min((ncap + 7) / 8, (2 * nsm + nops - 1) / nops));
    with_vt(vdt, [&](auto vp) -> edk_status {
      using VV = std::remove_pointer_t<decltype(vp)>;
      k_rdots2<VV><<<(unsigned)G, 256, 0, st>>>(d_ops(), rsplit(), V.as<VV>(), wt.as<VV>(),
                                                part.as<double2>(), pst, step.as<int>(),
                                                done.as<int>());
      k_breduce2<<<dim3(rx, nops), 256, 0, st>>>(
          splitops.as<SplitOp>(), ncap, m, part.as<double2>(), pst, cs.as<double2>(),
          ce.as<double2>(), scal.as<double4>(), alpha.as<double>(), beta.as<double>(),
          cnt.as<unsigned>(), step.as<int>(), done.as<int>(), closing);
      return EDK_OK;
    });
  }

  // After a run's last step: true when some running operator's last vector is
  // so short beside its T that its second sweep, which comes with the next step,
  // could take all of it.  (Above 1e-3 one sweep leaves |s| below 1e-3 even in FP32
  // storage.)
  bool may_close(const double* a, const double* b, const int* dn, const int* ns) const {
    for (int q = 0; q < nops; ++q) {
      if (dn[q] != 0 || ns[q] < 1) continue;
      const double *aq = a + (size_t)q * m, *bq = b + (size_t)q * m;
      double big = 0.0;
      for (int k = 0; k < ns[q]; ++k) big = std::max({big, std::fabs(aq[k]), std::fabs(bq[k])});
      if (bq[ns[q] - 1] <= 1e-3 * big) return true;
    }
    return false;
  }

  // Test the vector past the last step: beta of that step becomes 0 and the
  // operator stops (status 2) when the space is closed.
  edk_status close() {
    launch_dots(1);
    EDK_TRY_CUDA(cudaGetLastError());
    return EDK_OK;
  }

  // one Lanczos step for every live operator (graph-capturable)
  edk_status enqueue_step() {
    EDK_RETURN_IF(launch_apply());
    launch_dots(0);
    edk_status s = with_vt(vdt, [&](auto vp) -> edk_status {
      using VV = std::remove_pointer_t<decltype(vp)>;
      return with_vt(wdt, [&](auto wp) -> edk_status {
        using WD = std::remove_pointer_t<decltype(wp)>;
        k_rupdate2<VV, WD><<<(unsigned)G, 256, 0, st>>>(
            d_ops(), rsplit(), ncap, V.as<VV>(), cs.as<double2>(), ce.as<double2>(),
            scal.as<double4>(), wt.as<VV>(), w.as<WD>(), normpart.as<double>(), step.as<int>(),
            done.as<int>());
        launch_finish(0);
        k_bscale<WD, VV><<<(unsigned)ntiles, 256, 0, st>>>(d_ops(), tile2op.as<int>(), ncap,
                                                           w.as<WD>(), V.as<VV>(),
                                                           invb.as<double>(), step.as<int>(),
                                                           done.as<int>());
        return EDK_OK;
      });
    });
    EDK_RETURN_IF(s);
    EDK_TRY_CUDA(cudaGetLastError());
    return EDK_OK;
  }

  // V[:, 0] = start / ||start||; start is FP64 (wdt) concatenated on the device
  edk_status setup(const void* start_dev) {
    int minus1 = -1;
    hj = 0;
    EDK_TRY_CUDA(cudaMemsetAsync(done.p, 0, nops * sizeof(int), st));
    EDK_TRY_CUDA(cudaMemsetAsync(nsteps.p, 0, nops * sizeof(int), st));
    EDK_TRY_CUDA(cudaMemcpyAsync(step.p, &minus1, sizeof(int), cudaMemcpyHostToDevice, st));
    launch_split();
    edk_status s = with_vt(vdt, [&](auto vp) -> edk_status {
      using VV = std::remove_pointer_t<decltype(vp)>;
      return with_vt(wdt, [&](auto wp) -> edk_status {
        using WD = std::remove_pointer_t<decltype(wp)>;
        k_rstart<WD><<<(unsigned)G, 256, 0, st>>>(d_ops(), rsplit(), (const WD*)start_dev,
                                                  w.as<WD>(), normpart.as<double>(),
                                                  done.as<int>());
        launch_finish(1);
        k_bscale<WD, VV><<<(unsigned)ntiles, 256, 0, st>>>(d_ops(), tile2op.as<int>(), ncap,
                                                           w.as<WD>(), V.as<VV>(),
                                                           invb.as<double>(), step.as<int>(),
                                                           done.as<int>());
        return EDK_OK;
      });
    });
    EDK_RETURN_IF(s);
    EDK_TRY_CUDA(cudaGetLastError());
    return EDK_OK;
  }

  edk_status capture() {
    if (graph_ok || direct) return EDK_OK;
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return EDK_OK;  // replay not available: launch directly
    edk_status s = enqueue_step();
    cudaError_t e2 = cudaStreamEndCapture(st, &graph);
    if (s != EDK_OK) return s;
    if (e2 != cudaSuccess || !graph) { cudaGetLastError(); return EDK_OK; }
    if (cudaGraphInstantiate(&gexec, graph, 0) != cudaSuccess) {
      cudaGetLastError();
      return EDK_OK;
    }
    graph_ok = true;
    return EDK_OK;
  }

  edk_status run_step() {
    if (graph_ok) {
      EDK_TRY_CUDA(cudaGraphLaunch(gexec, st));
      return EDK_OK;
    }
    EDK_RETURN_IF(enqueue_step());
    ++hj;
    return EDK_OK;
  }
};

// Run the batch until every operator is done or max steps.  Convergence checks
// (every `check_every` steps) run on the device between two steps and set the
// stop flags there; the host reads only how many operators are left, on the
// copy stream while the next step already runs, so a check leaves the GPU no
// gap (the step that runs past the last check finds every operator stopped).
edk_status run_batch(BatchEngine& E, int max_steps, int nev, double tol, int check_every,
                     std::vector<OpResult>& res, int* nchecks = nullptr) {
  const int nops = E.nops;
  res.assign(nops, OpResult{});
  EDK_RETURN_IF(E.capture());
  DevBuf whole, ev, seen, left;
  DevParts parts;
  parts.add(ev, (size_t)nops * nev * sizeof(double));
  parts.add(seen, (size_t)nops * sizeof(int));
  parts.add(left, sizeof(int));
  EDK_RETURN_IF(parts.alloc(whole, E.st));
  EDK_TRY_CUDA(cudaMemsetAsync(seen.p, 0, (size_t)nops * sizeof(int), E.st));
  const int every = check_every > 0 ? check_every : 10;
  bool pending = false;
  for (int j = 0; j < max_steps; ++j) {
    EDK_RETURN_IF(E.run_step());
    if (pending) {
      int h = 0;
      EDK_TRY_CUDA(cudaStreamWaitEvent(E.side, E.checked, 0));
      EDK_TRY_CUDA(cudaMemcpyAsync(&h, left.p, sizeof(int), cudaMemcpyDeviceToHost, E.side));
      EDK_TRY_CUDA(cudaStreamSynchronize(E.side));
      pending = false;
      if (h == 0) break;
    }
    const bool last = (j + 1 == max_steps);
    if (!last && !((j + 1) % every == 0 && tol > 0)) continue;
    if (nchecks) ++*nchecks;
    if (tol > 0) {
      EDK_RETURN_IF(tridiag_check_device(nops, E.alpha.as<double>(), E.beta.as<double>(), E.m,
                                         E.nsteps.as<int>(), nev, ev.as<double>(), tol,
                                         seen.as<int>(), E.done.as<int>(), left.as<int>(), E.st));
      EDK_TRY_CUDA(cudaEventRecord(E.checked, E.st));
      pending = true;
    }
  }
  EDK_RETURN_IF(tridiag_lowest_device(nops, E.alpha.as<double>(), E.beta.as<double>(), E.m,
                                      E.nsteps.as<int>(), nullptr, 0, nev, ev.as<double>(), E.st));
  std::vector<double> ha((size_t)nops * E.m), hb((size_t)nops * E.m), he((size_t)nops * nev);
  std::vector<int> hdone(nops), hsteps(nops);
  EDK_TRY_CUDA(cudaMemcpyAsync(hdone.data(), E.done.p, nops * sizeof(int), cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaMemcpyAsync(hsteps.data(), E.nsteps.p, nops * sizeof(int), cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaMemcpyAsync(ha.data(), E.alpha.p, ha.size() * 8, cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaMemcpyAsync(hb.data(), E.beta.p, hb.size() * 8, cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaMemcpyAsync(he.data(), ev.p, he.size() * 8, cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaStreamSynchronize(E.st));
  if (E.may_close(ha.data(), hb.data(), hdone.data(), hsteps.data())) {
    EDK_RETURN_IF(E.close());
    EDK_TRY_CUDA(cudaMemcpyAsync(hdone.data(), E.done.p, nops * sizeof(int), cudaMemcpyDeviceToHost, E.st));
    EDK_TRY_CUDA(cudaMemcpyAsync(hb.data(), E.beta.p, hb.size() * 8, cudaMemcpyDeviceToHost, E.st));
    EDK_TRY_CUDA(cudaStreamSynchronize(E.st));
  }
  for (int q = 0; q < nops; ++q) {
    OpResult& r = res[q];
    r.status = hdone[q];
    r.steps = hsteps[q];
    r.a.assign(ha.begin() + (size_t)q * E.m, ha.begin() + (size_t)q * E.m + r.steps);
    r.b.assign(hb.begin() + (size_t)q * E.m, hb.begin() + (size_t)q * E.m + r.steps);
    const double* w = he.data() + (size_t)q * nev;
    r.ev.assign(w, w + std::min(nev, r.steps));
  }
  return EDK_OK;
}

// FP64 start vectors for the refinement of each operator into out (wdt
// layout): the sum of its `nev` lowest Ritz vectors, so the refined Krylov
// space holds every wanted eigenvector.  With `user` the vectors go to the
// caller and keep the sign of the QL eigensolver's (tridiag_eigen).
edk_status ritz_vectors(BatchEngine& E, const std::vector<OpResult>& res, void* out, int nev,
                        bool user) {
  std::vector<double2> c((size_t)E.nops * E.ncap, make_double2(0.0, 0.0));
  std::vector<int> nc(E.nops, 0);
  for (int q = 0; q < E.nops; ++q) {
    int mq = res[q].steps;
    if (mq <= 0) continue;
    const int nk = std::min({nev, mq, (int)res[q].ev.size()});
    std::vector<double> Q((size_t)mq * nk);
    for (int e = 0; e < nk; ++e)
      if (!std::isfinite(res[q].ev[e])) {
        set_error("tridiagonal eigensolver did not converge");
        return EDK_NOT_CONVERGED;
      }
    tridiag_vectors(mq, res[q].a.data(), res[q].b.data(), nk, res[q].ev.data(), Q.data());
    double sign = 1.0;
    if (user) {
      std::vector<double> w(mq), z(mq);
      if (tridiag_first_row(mq, res[q].a.data(), res[q].b.data(), w.data(), z.data()) != 0) {
        set_error("tridiagonal eigensolver did not converge");
        return EDK_NOT_CONVERGED;
      }
      sign = z[0] < 0 ? -1.0 : 1.0;
    }
    for (int k = 0; k < mq; ++k) {
      double v = 0.0;
      for (int e = 0; e < nk; ++e) v += Q[k + (size_t)e * mq];
      c[(size_t)q * E.ncap + k] = make_double2(sign * v, 0.0);
    }
    nc[q] = mq;
  }
  const size_t cb = c.size() * sizeof(double2), nb = nc.size() * sizeof(int);
  EDK_TRY_CUDA(cudaMemcpyAsync(E.cbuf.p, c.data(), cb, cudaMemcpyHostToDevice, E.st));
  EDK_TRY_CUDA(cudaMemcpyAsync(E.cnc.p, nc.data(), nb, cudaMemcpyHostToDevice, E.st));
  return with_vt(E.vdt, [&](auto vp) -> edk_status {
    using VV = std::remove_pointer_t<decltype(vp)>;
    return with_vt(E.wdt, [&](auto wp) -> edk_status {
      using WD = std::remove_pointer_t<decltype(wp)>;
      k_bcombine<VV, WD><<<(unsigned)E.ntiles, 256, 0, E.st>>>(
          E.d_ops(), E.tile2op.as<int>(), E.ncap, E.V.as<VV>(), E.cbuf.as<double2>(),
          E.cnc.as<int>(), (WD*)out);
      EDK_TRY_CUDA(cudaGetLastError());
      return EDK_OK;
    });
  });
}

// convert/copy concatenated start vectors into a device FP64 buffer of dtype wdt
template <class S, class D>
__global__ void k_cast(const S* __restrict__ src, int64_t n, D* __restrict__ dst) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    s2(dst + i, l2(src + i));
}

}  // namespace

// Group-level driver: FP64 or mixed (FP32 Krylov vectors + FP64 refinement).
edk_status batch_lanczos(const std::vector<edk_operator*>& ops, const edk_lanczos_opts& o,
                         const void* v0_dev, int v0_dt, cudaStream_t st,
                         std::vector<OpResult>& res, edk_lanczos_diag* diag, void* ritz_out) {
  double t0 = wall();
  const int nops = (int)ops.size();
  bool cx = o.complex_vectors != 0 || v0_dt == EDK_C128 || v0_dt == EDK_C64;
  for (auto* op : ops) cx |= op->is_complex;
  bool mixed = o.precision == EDK_PREC_MIXED;
  int vdt = mixed ? (cx ? EDK_C64 : EDK_F32) : (cx ? EDK_C128 : EDK_F64);
  int wdt = cx ? EDK_C128 : EDK_F64;
  // common lookup kind: translation sectors with and without phases share BK_TRANS
  int bk = ops[0]->b->dev.bk;
  bool all_mat = true;  // materialised operators run on the sliced-ELL kernel, whatever the basis
  for (auto* op : ops) all_mat = all_mat && op->sell_ok;
  bool ff = true;
  int64_t Dmin = INT64_MAX;
  for (auto* op : ops) {
    int k = op->b->dev.bk;
    if (k != bk) {
      if ((k == BK_TRANS0 || k == BK_TRANS) && (bk == BK_TRANS0 || bk == BK_TRANS)) bk = BK_TRANS;
      else if (!all_mat) {
        set_error("batch Lanczos: operators of different basis kinds");
        return EDK_UNSUPPORTED;
      }
    }
    ff = ff && op->ff_ok && op->use_ff;
    if (!op->gather) {
      set_error("batch Lanczos: an operator is not Hermitian in its basis");
      return EDK_NOT_HERMITIAN;
    }
    if (op->b->L > 32 && !op->sell_ok) {
      set_error("batch Lanczos: L > 32 runs only on materialised operators");
      return EDK_UNSUPPORTED;
    }
    Dmin = std::min<int64_t>(Dmin, op->b->D);
  }
  // translation sectors searched through their rank tables (with a phase:
  // every table must carry the shift M)
  bool ranked = (bk == BK_TRANS0 || bk == BK_TRANS || bk == BK_TRANSPAR) && ff;
  for (auto* op : ops)
    ranked = ranked && op->b->dev.search == 2 && (bk != BK_TRANS || op->b->dev.rank_shift == 10);
  if (ranked)
    bk = bk == BK_TRANS0 ? BK_TRANS0_RANK : (bk == BK_TRANS ? BK_TRANS_RANK : BK_TRANSPAR_RANK);
  if (bk == BK_ABELIAN && !all_mat) {
    set_error("batch Lanczos: symmetry-group (abelian) bases run one at a time unless materialised");
    return EDK_UNSUPPORTED;
  }
  if (o.max_steps > kMaxSteps) {
    set_error("batch Lanczos: at most " + std::to_string(kMaxSteps) + " steps");
    return EDK_UNSUPPORTED;
  }
  (void)Dmin;  // operators smaller than max_steps stop by the breakdown rule
  BatchEngine E;
  double ts0 = wall();
  int nchecks = 0;
  EDK_RETURN_IF(E.init(ops, vdt, o.max_steps, bk, ff, st));
  // start vectors in FP64 working dtype
  DevBuf start;
  EDK_RETURN_IF(start.alloc_async((size_t)E.totalD * esz(wdt), st));
  edk_status s = with_vt(v0_dt, [&](auto sp) -> edk_status {
    using SV = std::remove_pointer_t<decltype(sp)>;
    return with_vt(wdt, [&](auto dp) -> edk_status {
      using DV = std::remove_pointer_t<decltype(dp)>;
      k_cast<SV, DV><<<1184, 256, 0, st>>>((const SV*)v0_dev, E.totalD, (DV*)start.p);
      return EDK_OK;
    });
  });
  EDK_RETURN_IF(s);
  EDK_RETURN_IF(E.setup(start.p));
  EDK_RETURN_IF(E.capture());
  EDK_TRY_CUDA(cudaStreamSynchronize(st));
  double ts1 = wall();
  // mixed stage 1 (FP32 vectors): its Ritz values move by rounding at ~1e-7,
  // so it stops well above that — a ground state needs only a good start for
  // the FP64 refinement (1e-5), several levels a better one (1e-7) — and, for
  // a few operators, it checks every 5 steps so that it stops early
  double tol1 = mixed ? std::max(o.tol, o.nev > 1 ? 1e-7 : 1e-5) : o.tol;
  // (larger batches keep the caller's interval)
  const int check1 = (mixed && nops <= 8)
                         ? std::max(1, std::min(o.check_every > 0 ? o.check_every : 5, 5))
                         : o.check_every;
  EDK_RETURN_IF(run_batch(E, o.max_steps, o.nev, tol1, check1, res, &nchecks));
  double ts2 = wall();
  int rounds = 0;
  for (int q = 0; q < nops; ++q) {
    if (res[q].status == 4) {
      set_error("Initial state has non-finite entries (NaN or Inf)");
      return EDK_INVALID_ARG;
    }
    if (res[q].status == 3) {
      set_error("Initial state has zero norm");
      return EDK_ZERO_NORM;
    }
  }
  int steps_low = 0, mvs = 0, bd = 0;
  for (auto& r : res) { steps_low = std::max(steps_low, r.steps); mvs += r.steps; bd |= r.status == 2; }
  // global element offset of each operator in the concatenated layout
  std::vector<int64_t> goff(nops);
  for (int q = 0; q < nops; ++q) goff[q] = E.hops[q].woff;
  if (!mixed && ritz_out) EDK_RETURN_IF(ritz_vectors(E, res, ritz_out, 1, true));
  if (mixed) {
    // FP64 refinement restarted from the sum of the nev lowest Ritz vectors,
    // in one round that may run to max_steps (each operator stops when it
    // converges: a few steps for a ground state, more to separate close
    // levels).  Operators that reach the step limit unconverged are
    // restarted again, alone.
    const int mr = std::max(o.max_steps, o.refine_steps);
    std::vector<int> active(nops);
    for (int q = 0; q < nops; ++q) active[q] = q;
    DevBuf cur;  // start vectors of `active`, compact in that order
    EDK_RETURN_IF(ritz_vectors(E, res, start.p, o.nev, ritz_out != nullptr));
    void* cur_p = start.p;
    for (int round = 0; round < 4 && !active.empty(); ++round) {
      std::vector<edk_operator*> sub;
      for (int q : active) sub.push_back(ops[q]);
      BatchEngine F;
      EDK_RETURN_IF(F.init(sub, wdt, mr, bk, ff, st));
      EDK_RETURN_IF(F.setup(cur_p));
      std::vector<OpResult> r2;
      ++rounds;
      EDK_RETURN_IF(run_batch(F, mr, o.nev, o.tol, std::min(5, mr), r2, &nchecks));
      std::vector<int> next;
      std::vector<int> keep;  // positions in `active` of the operators to restart
      for (size_t i = 0; i < active.size(); ++i) {
        const int q = active[i];
        bool finite = r2[i].status < 3;  // (3, 4: the refinement's start vector is none)
        for (double x : r2[i].ev) finite = finite && std::isfinite(x);
        if (!finite) {
          set_error("batch Lanczos: the FP64 refinement of a mixed-precision run is not finite");
          return EDK_NOT_CONVERGED;
        }
        bool still = r2[i].ev.size() == res[q].ev.size();
        for (size_t k = 0; k < r2[i].ev.size() && still; ++k) {
          const double a = r2[i].ev[k], b = res[q].ev[k];
          still = std::fabs(a - b) <= std::max(o.tol, 1e-14) * std::max(1.0, std::fabs(a));
        }
        mvs += r2[i].steps;
        res[q] = r2[i];
        if (r2[i].status == 0 && !still && o.tol > 0) {
          next.push_back(q);
          keep.push_back((int)i);
        }
      }
      if (ritz_out) {
        // lowest Ritz vectors of the operators this round finalises
        DevBuf gs;
        EDK_RETURN_IF(gs.alloc_async((size_t)F.totalD * esz(wdt), st));
        EDK_RETURN_IF(ritz_vectors(F, r2, gs.p, 1, true));
        size_t k = 0;
        const bool last_round = round == 3;  // restarts end here: every vector is final
        for (size_t i = 0; i < active.size(); ++i) {
          if (!last_round && k < keep.size() && keep[k] == (int)i) { ++k; continue; }
          const int q = active[i];
          EDK_TRY_CUDA(cudaMemcpyAsync((char*)ritz_out + goff[q] * esz(wdt),
                                       (char*)gs.p + F.hops[i].woff * esz(wdt),
                                       (size_t)F.Ds[i] * esz(wdt), cudaMemcpyDeviceToDevice, st));
        }
        EDK_TRY_CUDA(cudaStreamSynchronize(st));
      }
      if (next.empty()) break;
      // Ritz vectors of this round (F's layout), then the restarted subset
      DevBuf full;
      EDK_RETURN_IF(full.alloc_async((size_t)F.totalD * esz(wdt), st));
      EDK_RETURN_IF(ritz_vectors(F, r2, full.p, o.nev, ritz_out != nullptr));
      int64_t tot = 0;
      for (int i : keep) tot += F.Ds[i];
      DevBuf nb;
      EDK_RETURN_IF(nb.alloc_async((size_t)std::max<int64_t>(tot, 1) * esz(wdt), st));
      int64_t dst = 0;
      for (int i : keep) {
        EDK_TRY_CUDA(cudaMemcpyAsync((char*)nb.p + dst * esz(wdt),
                                     (char*)full.p + F.hops[i].woff * esz(wdt),
                                     (size_t)F.Ds[i] * esz(wdt), cudaMemcpyDeviceToDevice, st));
        dst += F.Ds[i];
      }
      EDK_TRY_CUDA(cudaStreamSynchronize(st));
      std::swap(cur.p, nb.p);
      std::swap(cur.bytes, nb.bytes);
      std::swap(cur.pooled, nb.pooled);
      std::swap(cur.pool_stream, nb.pool_stream);
      cur_p = cur.p;
      active = next;
    }
  }
  EDK_TRY_CUDA(cudaStreamSynchronize(st));
  if (diag) {
    diag->steps = 0;
    for (auto& r : res) diag->steps = std::max(diag->steps, r.steps);
    diag->steps_low = mixed ? steps_low : diag->steps;
    diag->matvecs = mvs;
    diag->breakdown = bd;
    diag->seconds = wall() - t0;
    diag->seconds_matvec = NAN;
    diag->seconds_reorth = NAN;
    double resid = 0.0;
    for (auto& r : res) {
      int mm = r.steps;
      if (mm <= 0) continue;
      std::vector<double> y(mm);
      if (r.ev.empty() || !std::isfinite(r.ev[0])) continue;
      tridiag_vectors(mm, r.a.data(), r.b.data(), 1, r.ev.data(), y.data());
      resid = std::max(resid, std::fabs(r.b[mm - 1] * y[mm - 1]));
    }
    diag->residual = resid;
    diag->seconds_setup = ts1 - ts0;
    diag->seconds_stage1 = ts2 - ts1;
    diag->seconds_refine = mixed ? wall() - ts2 : 0.0;
    diag->refine_rounds = rounds;
    diag->checks = nchecks;
  }
  return EDK_OK;
}

// ---------------------------------------------------------------------------
// The Krylov driver's Lanczos basis: a batch of one, advanced in blocks of
// steps without a host round trip per step.
// ---------------------------------------------------------------------------
struct KrylovBasis::Impl {
  BatchEngine E;
  edk_operator* op = nullptr;
  // the operator as the engine's record and graph have it
  struct Form {
    uint64_t tables;
    bool ff;
    int tps, search;
    bool operator==(const Form& o) const {
      return tables == o.tables && ff == o.ff && tps == o.tps && search == o.search;
    }
  } form{};
  bool loaded = false;

  Form now() const { return Form{op->sell_tables, op->use_ff, op->tps, op->b->dev.search}; }
  // the lookup kind and kernel family of the product, as apply_device takes them
  int kind(bool& ff) {
    const BasisDev& b = op->b->dev;
    int bk = b.bk;
    ff = op->ff_ok && op->use_ff;
    if (ff && b.search == 2) {
      if (bk == BK_TRANS0) bk = BK_TRANS0_RANK;
      else if (bk == BK_TRANS && b.rank_shift == 10) bk = BK_TRANS_RANK;
      else if (bk == BK_TRANSPAR) bk = BK_TRANSPAR_RANK;
    }
    E.direct = !op->sell_ok && (bk == BK_ABELIAN || b.L > 32) ? op : nullptr;
    ff = ff && !E.direct;
    return bk;
  }
  // A cache outlives calls that materialise, clear or configure its operator: the
  // matrix that the record and the graph point to may be gone by then.
  edk_status refresh() {
    if (loaded && form == now()) return EDK_OK;
    loaded = false;  // also after a failure below: the next call tries again
    EDK_TRY_CUDA(cudaStreamSynchronize(E.st));
    bool ff = false;
    const int bk = kind(ff);
    EDK_RETURN_IF(E.load(std::vector<edk_operator*>(1, op), bk, ff));
    form = now();
    loaded = true;
    return E.capture();
  }
};
KrylovBasis::KrylovBasis() = default;
KrylovBasis::~KrylovBasis() = default;

edk_status KrylovBasis::init(edk_operator* op, int vdt, int m_max, cudaStream_t st) {
  impl = std::make_unique<Impl>();
  impl->op = op;
  bool ff = false;
  const int bk = impl->kind(ff);
  EDK_RETURN_IF(impl->E.init(std::vector<edk_operator*>(1, op), vdt, m_max, bk, ff, st));
  impl->form = impl->now();
  impl->loaded = true;
  return EDK_OK;
}

const void* KrylovBasis::vectors() const { return impl->E.V.p; }

edk_status KrylovBasis::start(const void* src, double* nrm, int* status) {
  BatchEngine& E = impl->E;
  EDK_RETURN_IF(impl->refresh());
  EDK_RETURN_IF(E.setup(src));
  EDK_RETURN_IF(E.capture());
  EDK_TRY_CUDA(cudaMemcpyAsync(nrm, E.alpha.p, sizeof(double), cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaMemcpyAsync(status, E.done.p, sizeof(int), cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaStreamSynchronize(E.st));
  return EDK_OK;
}

edk_status KrylovBasis::extend(int from, int to, double* alpha, double* beta, int* m) {
  BatchEngine& E = impl->E;
  EDK_RETURN_IF(impl->refresh());
  E.hj = from;
  for (int j = from; j < to; ++j) EDK_RETURN_IF(E.run_step());
  EDK_TRY_CUDA(cudaMemcpyAsync(alpha, E.alpha.p, (size_t)to * sizeof(double), cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaMemcpyAsync(beta, E.beta.p, (size_t)to * sizeof(double), cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaMemcpyAsync(m, E.nsteps.p, sizeof(int), cudaMemcpyDeviceToHost, E.st));
  EDK_TRY_CUDA(cudaStreamSynchronize(E.st));
  const int running = 0;  // all `to` steps, and no breakdown in the last
  if (*m == to && beta[to - 1] != 0.0 && E.may_close(alpha, beta, &running, m)) {
    // (the controller stops at beta = 0)
    EDK_RETURN_IF(E.close());
    EDK_TRY_CUDA(cudaMemcpyAsync(beta + *m - 1, E.beta.as<double>() + *m - 1, sizeof(double),
                                 cudaMemcpyDeviceToHost, E.st));
    EDK_TRY_CUDA(cudaStreamSynchronize(E.st));
  }
  return EDK_OK;
}

}  // namespace edk

using namespace edk;

extern "C" edk_status edk_batch_lanczos_e0(int32_t nops, edk_operator* const* ops,
                                           const edk_lanczos_opts* opts, const void* v0s,
                                           int32_t v0_dtype, double* evals,
                                           edk_lanczos_diag* diag) {
  EDK_CHECK_ARG(nops >= 1 && ops && opts && v0s && evals, "edk_batch_lanczos_e0: NULL argument");
  EDK_CHECK_ARG(v0_dtype == EDK_F64 || v0_dtype == EDK_C128,
                "edk_batch_lanczos_e0: v0s must be F64 or C128 (host)");
  EDK_CHECK_ARG(opts->max_steps >= 1 && opts->nev >= 1, "edk_batch_lanczos_e0: bad options");
  std::vector<edk_operator*> v(ops, ops + nops);
  int64_t tot = 0;
  for (auto* op : v) {
    EDK_CHECK_ARG(op != nullptr, "edk_batch_lanczos_e0: NULL operator");
    tot += op->b->D;
  }
  const OperatorLocks locks(v);
  cudaStream_t st = v[0]->stream;
  size_t es = v0_dtype == EDK_F64 ? 8 : 16;
  DevBuf v0d;
  EDK_RETURN_IF(v0d.alloc_async((size_t)tot * es, st));
  EDK_TRY_CUDA(cudaMemcpyAsync(v0d.p, v0s, (size_t)tot * es, cudaMemcpyHostToDevice, st));
  std::vector<OpResult> res;
  EDK_RETURN_IF(batch_lanczos(v, *opts, v0d.p, v0_dtype, st, res, diag));
  for (int q = 0; q < nops; ++q)
    for (int k = 0; k < opts->nev; ++k)
      evals[(size_t)q * opts->nev + k] = k < (int)res[q].ev.size() ? res[q].ev[k] : NAN;
  return EDK_OK;
}
