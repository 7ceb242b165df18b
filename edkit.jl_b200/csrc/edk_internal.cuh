// edk_internal.cuh — device-side data layout shared by the libedk sources.
//
// HBM layout of one basis (sector):
//   I     uint64[D]   sorted 0-based representative states (EDKit's I - 1)
//   R     f64[D]      orbit norms (symmetric kinds only)
//   htab  slots       open-addressing table state -> (row << 5 | norm class)
//   phase c128[len]   translation phase table C (or generator phase tables)
// Vectors are column-major blocks x[row + k*ld] of f64 / c128 / f32 / c64.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstdio>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/edk.h"

namespace edk {

void set_error(const std::string& msg);
const std::string& get_error();

#define EDK_TRY_CUDA(call)                                                          \
  do {                                                                              \
    cudaError_t e_ = (call);                                                        \
    if (e_ != cudaSuccess) {                                                        \
      edk::set_error(std::string(#call) + " failed: " + cudaGetErrorString(e_));    \
      return (e_ == cudaErrorMemoryAllocation) ? EDK_OOM : EDK_CUDA_ERROR;          \
    }                                                                               \
  } while (0)

#define EDK_CHECK_ARG(cond, msg)                 \
  do {                                           \
    if (!(cond)) {                               \
      edk::set_error(msg);                       \
      return EDK_INVALID_ARG;                    \
    }                                            \
  } while (0)

#define EDK_RETURN_IF(st) \
  do {                    \
    edk_status s_ = (st); \
    if (s_ != EDK_OK) return s_; \
  } while (0)

// Owning device buffer.  alloc() uses cudaMalloc; alloc_async() takes the
// memory from the device's stream-ordered pool on stream `s` (workspace of the
// Lanczos/Krylov drivers, reused across calls without new allocations).
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaStream_t pool_stream = nullptr;
  bool pooled = false;
  bool part = false;  // a part of another buffer (DevParts), which owns the memory
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { release(); }
  void release() {
    if (p && !part) {
      if (pooled) cudaFreeAsync(p, pool_stream);
      else cudaFree(p);
    }
    p = nullptr;
    bytes = 0;
    pooled = part = false;
  }
  edk_status alloc_async(size_t n, cudaStream_t s, cudaMemPool_t from = nullptr);
  edk_status alloc(size_t n) {
    release();
    if (n == 0) return EDK_OK;
    cudaError_t e = cudaMalloc(&p, n);
    if (e != cudaSuccess) {
      cudaGetLastError();  // an allocation failure is not sticky: clear it for later checks
      p = nullptr;
      set_error(std::string("cudaMalloc(") + std::to_string(n) + " bytes) failed: " +
                cudaGetErrorString(e));
      return EDK_OOM;
    }
    bytes = n;
    return EDK_OK;
  }
  template <class T> T* as() const { return reinterpret_cast<T*>(p); }
};

// keep freed pool memory cached in the process, up to half of the device's
// memory; what the pool holds beyond that goes back at the next synchronisation
// (set once per device)
inline void keep_pool_memory() {
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || done[dev]) return;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
    size_t fr = 0, total = 0;
    uint64_t thr = cudaMemGetInfo(&fr, &total) == cudaSuccess ? total / 2 : 0;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
  }
  done[dev] = true;
}

inline edk_status DevBuf::alloc_async(size_t n, cudaStream_t s, cudaMemPool_t from) {
  release();
  if (n == 0) return EDK_OK;
  keep_pool_memory();
  cudaError_t e = from ? cudaMallocFromPoolAsync(&p, n, from, s) : cudaMallocAsync(&p, n, s);
  if (e != cudaSuccess) {
    cudaGetLastError();  // an allocation failure is not sticky: clear it for later checks
    p = nullptr;
    set_error(std::string("cudaMallocAsync(") + std::to_string(n) + " bytes) failed: " +
              cudaGetErrorString(e));
    return EDK_OOM;
  }
  bytes = n;
  pool_stream = s;
  pooled = true;
  return EDK_OK;
}

// Several buffers of one allocation.  A pool that many streams have used can take 25 us
// an allocation (each free block's stream is looked at) instead of one, and a solver has
// some thirty small buffers: 0.65 ms of a 3 ms ground state.
struct DevParts {
  std::vector<std::pair<DevBuf*, size_t>> parts;
  void add(DevBuf& b, size_t n) { parts.push_back({&b, n}); }
  edk_status alloc(DevBuf& whole, cudaStream_t s) {
    size_t total = 0;
    for (auto& q : parts) total += (q.second + 255) / 256 * 256;
    edk_status rc = whole.alloc_async(total, s);
    if (rc != EDK_OK) return rc;
    size_t at = 0;
    for (auto& q : parts) {
      q.first->release();
      q.first->p = q.second ? static_cast<char*>(whole.p) + at : nullptr;
      q.first->bytes = q.second;
      q.first->part = true;
      at += (q.second + 255) / 256 * 256;
    }
    return EDK_OK;
  }
};

// The pool of what operators keep (row plans): apart from the default pool, whose
// free space the solvers' large workspaces need in one piece.  It holds at most
// 512 MB beyond what is in use.  Null (then the default pool serves) on failure.
inline cudaMemPool_t keep_pool() {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (!pools[dev]) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    if (cudaMemPoolCreate(&pools[dev], &props) != cudaSuccess) {
      cudaGetLastError();
      pools[dev] = nullptr;
      return nullptr;
    }
    uint64_t thr = 512ull << 20;
    cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &thr);
  }
  return pools[dev];
}

// ---------------------------------------------------------------------------
// lookup / canonicalisation kinds (compile-time dispatch)
// ---------------------------------------------------------------------------
enum LookupKind : int {
  BK_TENSOR = 0,     // row = state
  BK_PROJ_RANK = 1,  // row = colex rank among fixed-popcount states
  BK_PROJ_HASH = 2,  // row = hash(state)
  BK_TRANS0 = 3,     // translation, trivial phase (k = 0): min over rotations
  BK_TRANS = 4,      // translation, phase C[M] from the first-minimum shift M
  BK_TRANSPAR = 5,   // translation + reflection
  BK_ABELIAN = 6,    // generic odometer over commuting generators
  // BK_TRANS0 basis searched through its rank table (EDK_SEARCH_RANK); only
  // the bond-family fast path instantiates it, every other path keeps the hash
  BK_TRANS0_RANK = 7,
  // BK_TRANS basis searched through its rank table (entries carry the shift M)
  BK_TRANS_RANK = 8,
  // BK_TRANSPAR basis searched through its rank table (entries carry the sign)
  BK_TRANSPAR_RANK = 9
};

constexpr int kMaxGen = 8;
constexpr int kMaxLayers = 64;
constexpr int kNormClasses = 32;
constexpr uint32_t kHashEmpty32 = 0xFFFFFFFFu;

enum GenKind : int { GEN_PERM = 0, GEN_ROTL = 1, GEN_REV = 2, GEN_ID = 3 };

struct GenDev {
  int kind;      // GenKind
  int order;     // cyclic order
  int shift;     // rotation amount for GEN_ROTL
  int nlayers;   // delta-swap layers for GEN_PERM
  uint64_t inv_mask;
  int phase_off; // offset into the phase table
  int pad;
  uint64_t lmask[kMaxLayers];
  int lshift[kMaxLayers];
};

// Everything a kernel needs to know about a basis; passed by value.
struct BasisDev {
  int bk;          // LookupKind
  int L, A, len;   // sites, unit cell, number of translations
  int64_t D;
  uint64_t maskL;  // (1 << L) - 1
  const uint64_t* I;     // states (nullptr for TensorBasis)
  const double* R;       // norms (nullptr for onsite kinds)
  // hash table (BK_PROJ_HASH / translation kinds / abelian)
  const void* htab;
  uint64_t hmask;        // slots - 1
  int hbits;             // log2(slots)
  int packed;            // 1: value = row << 5 | class; 0: value = row, R gathered
  // sorted-array search (edk_basis_set_search): two-level binary search over
  // the ascending representatives instead of the hash table
  int search;              // 0: hash table, 1: sorted array
  const uint32_t* keys32;  // representatives as 32-bit words (L <= 32), else null
  const uint32_t* fence;   // keys32[32 j]: first level of the search
  int64_t nfence;
  const uint8_t* rcls8;    // norm class of each row (packed values), else null
  // rank table (edk_basis_set_search(EDK_SEARCH_RANK), search == 2): for every
  // state with the sector's popcount, indexed by its colex rank, the entry
  // row << rank_shift | M << 5 | norm class of its representative (M, the
  // first-minimum shift, only when rank_shift == 10; for translation + parity
  // sectors rank_shift == 6 and bit 5 is the sign of the coefficient), or ~0u
  // when the orbit is not in the basis; binom32[p * 33 + k] = C(p, k), p < 32
  int rank_shift;            // 5 (row < 2^27), 6 (row < 2^26, sign), 10 (row < 2^22, M)
  const uint32_t* rankmap;
  const uint32_t* binom32;
  const uint32_t* rowrank;   // colex rank of each representative I[i]
  int nclass;
  double Rcls[kNormClasses];
  // BK_PROJ_RANK
  int K;                 // popcount of every state
  // phases
  const double2* phase;  // translation: len entries; abelian: concatenated tables
  int P;                 // parity sign (TranslationParityBasis)
  int phase_real;        // 1 when every phase is real
  int runs_canon;        // 1: canonicalise from zero-run tops (unit cell 1, phase-free)
  // 1: compare rotations at the zero-run tops where the shift counts too (unit cell
  // 1, at least 512 rows, two blocks, per SM).  Fewer, but serial, candidates: where
  // rows fill the GPU the kernel is bound by issue and gains, below by latency and
  // loses.  Products with nearest neighbours, every rotation -> zero-run tops, us
  // (double / double complex): 2,704 rows 33.9 -> 34.8 / 33.7 -> 35.7; 32,066 45.0 ->
  // 47.8 / 46.7 -> 48.1; 58,786 - / 48.9 -> 50.7; 81,752 43.7 -> 43.5 / 45.5 -> 45.5;
  // 111,038 53.3 -> 49.3 / 52.7 -> 50.1; 204,248 68.4 -> 65.2 / 71.3 -> 66.7; 476,913
  // 132 -> 114 / 136 -> 118; single precision and next-nearest neighbours alike.
  int runs_arg;
  int sms;               // SMs of the device (host side: rules that fill the GPU)
  // abelian generators
  int ngen;
  const GenDev* gens;
};

// Local terms compiled for the device.
// Family: 2-site terms (i, i+d mod L) sharing one 4x4 matrix, evaluated on
// whole bit planes: X = s, Y = rotl(s, d), local column c = 2*X_p + Y_p.
struct FamDev {
  int d;
  int nnz[4];         // off-diagonal entries per local column
  uint64_t valid;     // bit p set when the family has a term with site i at bit p
  double2 dval[4];    // diagonal values M[c][c]
  int xr[4][3];       // c ^ r for each off-diagonal entry (bit1: site i, bit0: site j)
  double2 val[4][3];  // M[r][c]
};
// Generic term on up to 8 sites (bit positions, most significant site first).
struct TermDev {
  int nsites;
  int bitpos[8];
  int col_off;        // offset into colptr (2^nsites + 1 entries)
  int diag_off;       // offset into dval (2^nsites entries)
};
// Flip-flop bond families for the fast path (all 2-site off-diagonal terms
// swap the two digits; every other term is diagonal).
constexpr int kMaxFF = 4;
struct FFParams {
  int nfam;
  int d[kMaxFF];
  uint32_t valid[kMaxFF];
  double2 dval[kMaxFF][4];
  double2 v1[kMaxFF];  // M[2][1]: local column "01" -> row "10"
  double2 v2[kMaxFF];  // M[1][2]: local column "10" -> row "01"
  int same[kMaxFF];    // 1 when v1 == v2 (one accumulator for both directions)
};

// Materialised operator (the device counterpart of sparse!(opt)): sliced
// ELLPACK with 32-row slices.  Rows are sorted by their number of nonzeros
// inside windows of 256 rows; slice s holds rows rowid[32 s .. 32 s + 31] and
// its entries k = 0..w_s-1 at off_s + 32 k + lane (lane = row in the slice):
// col = target row, code = index into vt (vt[0] = 0 pads short rows); when
// the code's bits and the row's bits fit together, both share one 32-bit word.
// y[r] = (1/R_r) sum conj(vt[code]) x[col] + conj(diag[r]) x[r].
struct SellDev {
  int64_t nslices;
  int packed;              // > 0: entry = row << packed | code, both in `col`
  int rbits;               // slot word = row | norm class << rbits; ~0u past the last row
  const unsigned* rowid;   // 32 per slice, in slot order
  const int64_t* off;      // entry offset of each slice
  const int* width;        // entries per lane of each slice
  const int* col;          // target rows
  const uint16_t* code;    // coefficient codes
  const double2* val;      // value mode (any operator): the entry's coefficient c, y += conj(c) x;
                           // col holds the row, no codes (null in code mode)
  const double* diag;      // real diagonal per slot (Hermitian operators with real terms)
  const double2* diagc;    // complex diagonal per slot, or null
  const double* rinv;      // 1 / R of each norm class (1 for bases without norms)
  const double2* vt64;     // coefficient table, FP64
  const float2* vt32;      // the same table rounded to FP32
};

// Device memory of the row plans of a batch of operators.  The last of them to go gives
// it back, on the device it lives on, whichever is current then, and after every
// product that still runs there (edk_apply_async, on any stream): one synchronisation
// for the batch.
struct PlanSlab {
  DevBuf buf;
  int device = 0;
  ~PlanSlab() {
    if (!buf.p) return;
    int prev = device;
    cudaGetDevice(&prev);
    if (prev != device) cudaSetDevice(device);
    cudaDeviceSynchronize();
    buf.pool_stream = nullptr;  // the stream it came from may be gone by now
    buf.release();
    if (prev != device) cudaSetDevice(prev);
  }
};

constexpr int kPlanWindow = 256;  // rows per window of a row plan (and per thread block)
// Device view of a row plan: slot k of window w describes row
// rw[k] & kPlanRowMask of that window (rows sorted by their number of hits).
struct RowPlanDev {
  // one 16-byte slot per row, read with one load:
  //   x = row | norm class << 27 (~0u pads the last window)
  //   y = row state (L <= 32)
  //   z = colex rank of the row state (the row itself for complete sectors)
  //   w = rank of the state with bits 0 and L-1 exchanged (the wrap-around
  //       bond of a nearest-neighbour family), or ~0u
  const uint4* slot;
  const double* dg;       // diagonal of the row (operators with diagonal-only generic terms), or null
  int64_t nslots;         // windows * 256
};
constexpr uint32_t kPlanRowMask = (1u << 27) - 1u;

// Pauli-string form of an operator on the full space (edk_pauli.cu).
struct PauliStr { double2 v; uint32_t z, pad; };  // v (-1)^{|s & z|}
// strings s0 .. s1-1 flip the bits x; empty: some rows have no element with that flip
struct PauliGroup { uint32_t x; int s0, s1, empty; };
constexpr int kPauliFlips = 64;
struct PauliFlips {  // strings without z part, one per flip mask, by ascending mask
  int n;
  uint32_t x[kPauliFlips];
  double v[kPauliFlips];
};
struct PauliDev {
  int ngroup, ndiag;
  const PauliGroup* group;  // by flip mask, ascending
  const PauliStr* str;
  const PauliStr* diag;     // diagonal strings of the terms outside the bond families
};

struct OpDev {
  SellDev sell;
  RowPlanDev plan;          // row plan of the rank-searched fast path (plan.slot null: none)
  int nfam;
  const FamDev* fam;
  int nterm;
  const TermDev* term;
  const int* colptr;        // per term: start of the off-diagonal list of each column
  const uint64_t* xmask;    // XOR mask turning the row state into the column state
  const double2* val;       // matrix element M[r][c]
  const double2* dval;      // diagonal M[c][c]
};

}  // namespace edk

// Opaque handles of the C ABI.
struct edk_basis {
  edk_basis_desc desc{};
  int kind = 0;
  int L = 0, A = 1, len = 1, K = -1, P = 1, Kmom = 0;  // Kmom = mod(-k, len)
  int64_t D = 0;
  edk::DevBuf I, R, htab, phase, gens;
  edk::DevBuf keys32, fence, rcls8;  // sorted-array search tables (built on demand)
  edk::DevBuf rankmap, binom32, rowrank;  // rank table of EDK_SEARCH_RANK (built on demand)
  edk::BasisDev dev{};
  std::vector<edk::GenDev> gens_host;
  std::vector<int> gen_order, gen_q;
  std::vector<std::vector<int>> gen_perm;
  std::vector<std::vector<uint8_t>> gen_inv;
  bool phase_complex = false;
  bool pairnorm = false;  // TranslationFlipBasis norms on the abelian path
  int device = 0;  // CUDA device the tables live on
  bool handles = false;  // has borrowed library handles (edk_handles.cu)
  cudaStream_t stream = nullptr;
  std::mutex mu;
  ~edk_basis();
};

struct edk_operator {
  edk_basis* b = nullptr;
  edk::DevBuf fam, term, colptr, xmask, val, dval;
  edk::DevBuf hx, hy;  // staging buffers of edk_apply's host-pointer path (grow only)
  // materialised matrix (edk_operator_materialize)
  edk::DevBuf s_rowid, s_off, s_width, s_col, s_code, s_diag, s_vt64, s_vt32, s_rinv, s_err, s_val;
  int64_t sell_wincap = 0;  // entries of the largest 256-row window
  bool sell_tma_ok = false;  // the staged (bulk-copy) product applies (stages fit in shared memory)
  bool sell_tma = false;     // ... and is used (set by the autotuner)
  uint64_t sell_tables = 0;  // raised when the tables below dev.sell come or go
  bool sell_ok = false;
  int64_t sell_entries = 0;
  edk::OpDev dev{};
  bool gather = true;
  bool is_complex = false;
  bool ff_ok = false;     // flip-flop bond-family fast path applies
  bool use_ff = true;     // callers may switch the fast path (either one) off
  int tps = 1;            // threads per state of the fast path (1, 2 or 4; autotuned)
  // row plan of the fast path on rank-searched sectors (edk_plan.cu): built on
  // first use; plan_state 0 not built, 1 built, -1 not available
  std::shared_ptr<edk::PlanSlab> p_slab;  // shared by the operators of the batch that built it
  int plan_state = 0;
  // Pauli-string form (full space, no flip-flop fast path, few enough strings): the
  // fast kernel of such an operator, taken while use_ff
  edk::DevBuf pa_group, pa_str, pa_diag;
  edk::PauliDev pauli{};
  edk::PauliFlips pauli_flips{};
  bool pauli_ok = false;
  bool use_plan = true;   // tps == 1 on a rank-searched sector runs the plan kernel
  int use_block = -1;     // several right-hand sides through one SpMM: 1 yes, 0 no, -1 auto
                          // (yes unless materialised or on a row plan, whose one-column
                          // products already stream faster)
  std::vector<unsigned char> ff_params;
  int max_hits = 0;
  int nfam = 0, ngeneric = 0;
  // host copy of the merged terms (used by the invariance check)
  std::vector<std::vector<int>> sites;
  std::vector<std::vector<double>> dense_re, dense_im;  // local matrices, row-major
  cudaStream_t stream = nullptr;
  edk::DevBuf bx, by, bop;               // row-major blocks and operator record of the SpMM path
  std::vector<unsigned char> bop_host;   // the record as last uploaded
  cudaStream_t cstream = nullptr;        // copy stream of the pipelined host path
  std::vector<cudaEvent_t> cevents;      // one per row chunk of that path
  bool handles = false;                  // has borrowed library handles (edk_handles.cu)
  std::mutex mu;
  ~edk_operator();
};

// Locks every operator of a batch, each once, in the order of their addresses
// (two batches that share operators cannot wait for each other).
struct OperatorLocks {
  std::vector<std::unique_lock<std::mutex>> held;
  explicit OperatorLocks(std::vector<edk_operator*> ops) {
    std::sort(ops.begin(), ops.end());
    ops.erase(std::unique(ops.begin(), ops.end()), ops.end());
    for (edk_operator* op : ops) held.emplace_back(op->mu);
  }
};

namespace edk {
// implemented in edk_basis.cu
edk_status check_basis_dev(const BasisDev& b);
edk_status index_device(const BasisDev& dv, int64_t n, const uint64_t* s_d, int64_t* p_d,
                        double2* c_d, cudaStream_t st);
// rows [row0, row1) of y = H x (row0, row1 multiples of 256 or row1 = D)
// for one vector, on the row-gather fast or materialised paths; false when the
// operator runs on another path
bool rows_apply_ok(const edk_operator* op);
edk_status apply_rows(edk_operator* op, int dtype, const void* x, void* y, int64_t row0,
                      int64_t row1, int accumulate, cudaStream_t st);
// implemented in edk_plan.cu
bool plan_applies(const edk_operator* op);
edk_status plan_ensure(const std::vector<edk_operator*>& ops, cudaStream_t st);
edk_status apply_plan(edk_operator* op, int dtype, const void* x, void* y, int64_t nvec,
                      int64_t ldx, int64_t ldy, int accumulate, cudaStream_t st, int64_t row0,
                      int64_t row1);
// implemented in edk_pauli.cu
edk_status apply_pauli(const edk_operator* op, int dtype, const void* x, void* y, int64_t nvec,
                       int64_t ldx, int64_t ldy, int accumulate, cudaStream_t st,
                       const int* step = nullptr, const int* done = nullptr);
// implemented in edk_sell.cu
edk_status apply_sell_rows(edk_operator* op, int dtype, const void* x, void* y, int64_t row0,
                           int64_t row1, int accumulate, cudaStream_t st);
edk_status apply_sell(edk_operator* op, int dtype, const void* x, void* y, int64_t nvec,
                      int64_t ldx, int64_t ldy, int accumulate, cudaStream_t st);
// implemented in edk_apply.cu
edk_status apply_device(edk_operator* op, int dtype, const void* x, void* y, int64_t nvec,
                        int64_t ldx, int64_t ldy, int accumulate, cudaStream_t st);
// implemented in edk_batch.cu
struct OpResult {
  std::vector<double> a, b, ev;  // recurrence coefficients and lowest Ritz values
  int steps = 0;
  int status = 0;  // 0 ran to the step limit, 1 converged, 2 breakdown, 3 zero norm,
                   // 4 non-finite start
};
// ritz_out (optional, device): every operator's lowest Ritz vector in the
// FP64 working dtype (F64 or C128), concatenated in operator order
edk_status batch_lanczos(const std::vector<edk_operator*>& ops, const edk_lanczos_opts& o,
                         const void* v0_dev, int v0_dt, cudaStream_t st,
                         std::vector<OpResult>& res, edk_lanczos_diag* diag,
                         void* ritz_out = nullptr);
// One operator's Lanczos basis on the batched engine, for the Krylov driver.
// start(): V[:, 0] = src / |src| (src: D values of the FP64 working dtype on
// the device), *status 3 for a zero and 4 for a non-finite norm; extend(): steps
// from .. to-1, then alpha / beta [0, to) and the steps taken (fewer than `to`
// after a breakdown); vectors(): V, D x (m_max + 1) column-major in dtype vdt.
class KrylovBasis {
 public:
  KrylovBasis();
  ~KrylovBasis();
  edk_status init(edk_operator* op, int vdt, int m_max, cudaStream_t st);
  edk_status start(const void* src, double* nrm, int* status);
  edk_status extend(int from, int to, double* alpha, double* beta, int* m);
  const void* vectors() const;

 private:
  struct Impl;
  std::unique_ptr<Impl> impl;
};
// implemented in edk_eig.cu
edk_status hermitian_eigvals(bool cx, int n, const void* G, double* W, cudaStream_t st);
// implemented in edk_handles.cu: a cuBLAS handle (and on request a cuSOLVER one)
// borrowed for one call on one stream
struct LibHandles {
  void *blas = nullptr, *solver = nullptr;
};
struct HandleLease {
  LibHandles h;
  int device = 0;
  cudaStream_t stream = nullptr;
  HandleLease() = default;
  HandleLease(const HandleLease&) = delete;
  HandleLease& operator=(const HandleLease&) = delete;
  ~HandleLease();
  // `registered`: the borrowing object's flag (edk_basis / edk_operator handles)
  edk_status take(bool& registered, cudaStream_t st);
  edk_status add_solver();
};
void handles_unregister(bool registered);
// implemented in edk_util.cpp
int tridiag_eigvals(int m, const double* a, const double* b, double* w);
// The lowest `nev` distinct eigenvalues of block-tridiagonal Hermitian matrices
// (edk_band.cu): operator q has m[q] blocks; SA and SB (device) hold step j's
// p x p products of operator q at (j nops + q) p^2.  SA's steps are brought into their
// final form in place (k_band_pack); `state`, one per run, keeps how far.  NaN where
// fewer are found.
struct BandState {
  std::vector<int> packed;  // steps of each operator in their final form
  DevBuf diag;              // largest diagonal entries so far
};
edk_status band_lowest_device(int p, int nev, const std::vector<int>& m, void* SA, const void* SB,
                              BandState& state, cudaStream_t st,
                              std::vector<std::vector<double>>& out);
int tridiag_eigen(int m, const double* a, const double* b, double* w, double* Q);
int tridiag_first_row(int m, const double* a, const double* b, double* w, double* z);
// implemented in edk_tridiag.cu: the lowest nk eigenvalues of nops tridiagonal
// matrices on the device (ev: nops x nk), and the convergence check of a
// batch on them; inverse iteration on the host
edk_status tridiag_check_device(int nops, const double* alpha, const double* beta, int64_t ld,
                                const int* nsteps, int nk, double* ev, double tol, int* seen,
                                int* done, int* left, cudaStream_t st);
edk_status tridiag_lowest_device(int nops, const double* alpha, const double* beta, int64_t ld,
                                 const int* nsteps, const int* nfix, int nall, int nk, double* ev,
                                 cudaStream_t st);
void tridiag_vectors(int m, const double* a, const double* b, int nk, const double* w, double* Q);
double elapsed_ms(cudaEvent_t a, cudaEvent_t b);
}  // namespace edk
