/*
 * edk.h — C ABI of libedk, the B200 (sm_100a) implementation of EDKit.jl's
 * matrix-free operator application and the Lanczos / Krylov loops built on it.
 *
 * A Julia host binds these with `ccall`; Python binds them with ctypes.  No CUDA or torch types cross this boundary:
 * only plain pointers, sizes and the POD structs below.
 *
 * Conventions (identical to EDKit.jl):
 *   - digit strings are big-endian: site 1 is the most significant digit
 *     (src/Basis/AbstractBasis.jl:285-298); spin-1/2 digit 0 is Sz=+1/2;
 *   - basis tables cross the boundary as Julia holds them: `I` 1-based int64,
 *     `R` float64 norms;
 *   - vectors are Julia column-major blocks: element (row r, column k) sits at
 *     x[r + k*ldx]; complex numbers are interleaved {re, im};
 *   - every function returns an edk_status; edk_last_error() gives the
 *     message of the last failure on the calling thread.
 *
 * Host pointers are borrowed for the duration of a call.  Handles own their
 * device memory and are released by the matching *_destroy function.
 */
#ifndef EDK_H
#define EDK_H

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

typedef enum {
  EDK_OK = 0,
  EDK_INVALID_ARG = 1,
  EDK_NOT_HERMITIAN = 2,
  EDK_OOM = 3,
  EDK_CUDA_ERROR = 4,
  EDK_TIMEOUT = 5,
  EDK_NOT_CONVERGED = 6,
  EDK_UNSUPPORTED = 7,
  EDK_ZERO_NORM = 8,
  EDK_BACKWARD_TIME = 9
} edk_status;

/* element type of vectors crossing the boundary */
typedef enum { EDK_F64 = 0, EDK_C128 = 1, EDK_F32 = 2, EDK_C64 = 3 } edk_dtype;

/* where the vector pointers of a call live */
typedef enum { EDK_HOST = 0, EDK_DEVICE = 1 } edk_ptr_kind;

typedef enum {
  EDK_TENSOR = 0,        /* TensorBasis            src/Basis/AbstractBasis.jl:217-247 */
  EDK_PROJECTED = 1,     /* ProjectedBasis         src/Basis/ProjectedBasis.jl:14-260 */
  EDK_TRANSLATIONAL = 2, /* TranslationalBasis     src/Basis/TranslationalBasis.jl:22-349 */
  EDK_TRANSPARITY = 3,   /* TranslationParityBasis src/Basis/TranslationalParityBasis.jl:15-241 */
  EDK_ABELIAN = 4,       /* AbelianBasis / basis() src/Basis/AbelianBasis.jl:498-847 */
  EDK_TRANSFLIP = 5      /* TranslationFlipBasis   src/Basis/TranslationalFlipBasis.jl:9-213:
                            generators as for EDK_ABELIAN, exactly two — translation by a
                            (order L/a, q = -k mod L/a: the generator rotates against the
                            reference's circshift!) then spin flip (order 2, q = 0 for
                            p = +1, 1 for p = -1) — with the reference's norms
                            2len/sqrt(period) [/sqrt 2 without a flip match] */
} edk_basis_kind;

typedef struct edk_basis edk_basis;
typedef struct edk_operator edk_operator;

/*
 * Basis description.  Mirrors the keyword arguments of the Julia constructors.
 * When `I` is NULL the library builds the tables on the device (base 2, with
 * or without a charge N; a predicate `f` arrives as the `allow` bitmap the
 * host evaluated).  Alternatively the host passes the tables it already holds
 * (b.I, b.R) and the library uploads them unchanged.
 */
typedef struct {
  int32_t kind;   /* edk_basis_kind */
  int32_t L;      /* number of sites */
  int32_t base;   /* local dimension; the GPU path supports 2 */
  int32_t a;      /* unit cell (translational kinds), 1 otherwise */
  int32_t k;      /* momentum label exactly as passed to the Julia constructor */
  int32_t p;      /* parity +-1 (TranslationParityBasis) */
  int32_t N;      /* charge in EDKit's convention (sum(dgt) == L*(base-1)-N), -1 = nothing;
                     for EDK_ABELIAN it is basis()'s N (set bits on the Gosper path) */
  /* EDK_ABELIAN generators, in the order basis() pushes them */
  int32_t ngen;
  const int32_t* gen_order; /* cyclic order of each generator */
  const int32_t* gen_q;     /* quantum number of each generator */
  const int32_t* gen_perm;  /* ngen x L site permutations, 1-based: site i -> perm[i] */
  const uint8_t* gen_inv;   /* ngen x L spin-inversion flags */
  /* optional predicate result f(dgt) as a bitmap over 0-based states
     (bit s of word s/64); states whose bit is clear are rejected before the
     symmetry check, exactly where the judges test F(dgt) first
     (TranslationalBasis.jl:96, TranslationalParityBasis.jl:70) */
  const uint64_t* allow;
  /* optional tables, as the Julia basis holds them */
  int64_t D;         /* number of rows in I/R */
  const int64_t* I;  /* 1-based, ascending */
  const double* R;   /* norms (ignored for onsite kinds) */
} edk_basis_desc;

/* Build a basis (tables on the device).  Replaces the constructors
 * TensorBasis (AbstractBasis.jl:234), ProjectedBasis (ProjectedBasis.jl:244),
 * TranslationalBasis (TranslationalBasis.jl:235), TranslationParityBasis
 * (TranslationalParityBasis.jl:141) and basis() (AbelianBasis.jl:771). */
edk_status edk_basis_create(const edk_basis_desc* desc, edk_basis** out);
edk_status edk_basis_destroy(edk_basis* b);
/* size(b, 1) — AbstractBasis.jl:142-146 */
edk_status edk_basis_dim(const edk_basis* b, int64_t* D);
/* copy the tables back (I 1-based, R norms; R is all ones for onsite kinds).
 * Used for the bit-exact table check against b.I / b.R. */
edk_status edk_basis_export(const edk_basis* b, int64_t* I, double* R);
/* Batched index(b, dgt) — AbstractBasis.jl:246, ProjectedBasis.jl:52-57,
 * TranslationalBasis.jl:310-341, TranslationalParityBasis.jl:192-234,
 * AbelianBasis.jl:669-693.  `states` are 0-based integer states (index(dgt)-1);
 * pos receives the 1-based position (0 when the state is not in the basis,
 * where EDKit returns (0, 1)), coeff the interleaved complex coefficient. */
edk_status edk_basis_index(const edk_basis* b, int64_t n, const uint64_t* states,
                           int64_t* pos, double* coeff, int32_t ptr_kind);

/* index() for host-resident states without any device allocation: the same
 * results as edk_basis_index(..., EDK_HOST), staged through a fixed 2 MiB
 * scratch area inside the library (at most 65536 states per call; larger n is
 * rejected with EDK_INVALID_ARG).  For callers that cannot allocate device
 * memory where they need a lookup, such as host callbacks that forbid
 * allocation or processes whose device memory another component has already
 * reserved.  The scratch address is resolved on the first call for each
 * device, so make that first call before any stream capture; calls are
 * serialised and synchronous, and work that another caller launched on the
 * same scratch at the same time would race.  This entry point has no
 * counterpart in the reference. */
edk_status edk_basis_index_noalloc(const edk_basis* b, int64_t n, const uint64_t* states,
                                   int64_t* pos, double* coeff);

/* Index search of a basis with a table of representatives (ProjectedBasis
 * outside complete sectors, TranslationalBasis, TranslationParityBasis,
 * AbelianBasis): EDK_SEARCH_HASH (default, open-addressing table) or
 * EDK_SEARCH_SORTED, a two-level binary search over the ascending
 * representatives — the search EDKit's index() performs (binary_search,
 * src/Basis/ProjectedBasis.jl:71-81, called from TranslationalBasis.jl:318-325
 * and AbelianBasis.jl:678-686).  Both give identical rows; the choice is a
 * speed trade made by edk_operator_autotune.  The strategy belongs to the
 * basis and so applies to every operator on it.  EDK_UNSUPPORTED for bases
 * that index rows directly; EDK_INVALID_ARG when the representatives are not
 * strictly ascending. */
#define EDK_SEARCH_HASH 0
#define EDK_SEARCH_SORTED 1
/* EDK_SEARCH_RANK: translation and translation-parity sectors
 * (TranslationalBasis, TranslationParityBasis) of fixed N with L <= 32; with a
 * momentum phase the sector must have fewer than 2^22 rows, with parity fewer
 * than 2^26.  A table over every state of the charge sector, indexed by the
 * state's colex rank, holds the row of its orbit representative and the
 * first-minimum shift M that sets its phase (for translation-parity sectors,
 * the sign of the coefficient); 4 * C(L, N) bytes: 160 MB at L = 28, 2.4 GB
 * at L = 32.  The bond-family row kernel then finds a target row by updating
 * the row state's rank for the exchanged pair of sites and reading one table
 * entry, with no canonicalisation.  Rows and phases are identical to the other strategies'.
 * Paths other than the bond-family row kernel keep using the hash table. */
#define EDK_SEARCH_RANK 2
edk_status edk_basis_set_search(edk_basis* b, int32_t strategy);
edk_status edk_basis_get_search(const edk_basis* b, int32_t* strategy);

/* Build an operator from merged local terms — operator() Operator.jl:56-78
 * after its site-list merge, trans_inv_operator() Operator.jl:102-108.
 * Term t acts on nsites[t] sites (1-based, concatenated in `sites`) with a
 * local (base^nsites)^2 matrix in Julia CSC form: colptr (1-based,
 * base^nsites+1 entries per term), rowval (1-based), nzval (interleaved
 * complex), nnz[t] nonzeros each, all concatenated.  The library checks each
 * term for Hermiticity and the operator for invariance under the basis
 * symmetries; when both hold it applies the row-gather form, otherwise the
 * column-scatter form with atomics. */
edk_status edk_operator_create(edk_basis* b, int32_t nterms, const int32_t* nsites,
                               const int32_t* sites, const int64_t* nnz, const int64_t* colptr,
                               const int64_t* rowval, const double* nzval, edk_operator** out);
edk_status edk_operator_destroy(edk_operator* op);
/* properties: is_hermitian_gather (1 = row-gather form), is_complex (1 = complex
 * matrix elements), n_families (2-site term families on the bit-plane path),
 * n_generic (remaining terms) */
edk_status edk_operator_info(const edk_operator* op, int32_t* gather, int32_t* is_complex,
                             int32_t* n_families, int32_t* n_generic);

/* sparse!(opt) / clear_sparse_cache! (Operator.jl:221-285) for the device:
 * enable=1 expands every row once into a cached sliced-ELLPACK matrix that
 * every later edk_apply / edk_lanczos_e0 / edk_krylov_evolve / batch call on
 * this operator uses; enable=0 frees it.  *entries (may be NULL) receives the
 * number of stored entries.  Bond-family operators (XXZ-type bonds plus
 * diagonal terms, L <= 32) store a target row and a coefficient code per
 * nonzero (4 bytes when they fit one word); every other operator in the
 * row-gather form (Hermitian and symmetric under its basis: generic terms,
 * symmetry-group and dedicated bases, L up to 63) stores the row and the
 * explicit complex coefficient (20 bytes).  Materialised operators of any
 * basis kind run batched. */
edk_status edk_operator_materialize(edk_operator* op, int32_t enable, int64_t* entries);

/* Block Lanczos over a batch of operators (e.g. the momentum sectors of one
 * chain), each with a block of `block` right-hand-side vectors: the block
 * form of EDKit's Lanczos recurrence (_lanczos_build!,
 * src/algorithms/TimeEvolution.jl:250-306) with one classical block
 * Gram-Schmidt pass against the two previous blocks and Cholesky-QR
 * (twice) for the next block.  The lowest `nev` distinct eigenvalues of each
 * operator's block-tridiagonal matrix are returned in evals[q * nev + k]
 * (NaN where fewer exist).  x0: per operator a D_q x block column-major
 * complex128 start block (host), concatenated; NULL draws seeded N(0,1) real
 * and imaginary parts on the device from opts->seed.  Every operator must be
 * Hermitian in the row-gather form and block * max_steps below its dimension.
 * tol > 0 stops when every operator's nev values move less than
 * tol * max(1, |E0|) between checks (every check_every steps); tol = 0 runs
 * max_steps.  Device memory, in bytes, with D the largest dimension: 3 x 16 nops D
 * block for the vectors, 32 nops max_steps block^2 for T, held for the whole run, and
 * 16 nops n min(n, 1201) with n = block * steps for an eigenvalue step.  What does not
 * fit ends in EDK_OOM.  No reference counterpart (EDKit runs one vector). */
typedef struct {
  int32_t block;        /* vectors per operator: multiple of 8, 8..64 */
  int32_t max_steps;    /* block steps */
  int32_t nev;
  double tol;
  int32_t check_every;
  uint64_t seed;
} edk_block_lanczos_opts;
typedef struct {
  int32_t steps;        /* block steps taken */
  int64_t matvecs;      /* single-vector products: steps * block * nops */
  int32_t breakdowns;   /* operators whose Krylov space closed early */
  int32_t converged;    /* 1 when tol stopped the run */
  double seconds, seconds_spmm, seconds_orth, seconds_eig;
} edk_block_lanczos_diag;
void edk_block_lanczos_default_opts(edk_block_lanczos_opts* opts);

/* The eigenvalue step of edk_block_lanczos (which runs it on the device) on
 * a block-tridiagonal matrix the caller holds, computed on the host with no
 * device work: A = m diagonal blocks (p x p,
 * column-major complex, interleaved re/im, Hermitian), B = m-1 sub-diagonal
 * blocks T(j+1, j).  out = the lowest nev distinct eigenvalues, copies that a
 * block Lanczos run without full re-orthogonalisation creates removed by the
 * block Cullum-Willoughby test (NaN where fewer exist). */
edk_status edk_block_tridiag_lowest(int32_t p, int32_t m, const double* A, const double* B,
                                    int32_t nev, double* out);
edk_status edk_block_lanczos(int32_t nops, edk_operator* const* ops,
                             const edk_block_lanczos_opts* opts, const double* x0, double* evals,
                             edk_block_lanczos_diag* diag);

/* Kernel choice of the matrix-free application.  EDK_KERNEL_FAST: the
 * bond-family kernel (operators whose off-diagonal part is flip-flop bonds),
 * with `tps` threads (1, 2, 4) sharing each state, or the Pauli-string kernel
 * (operators other than flip-flop bonds on TensorBasis with L <= 31, where few
 * strings hold them; tps ignored); EDK_KERNEL_GENERIC: the row kernel that handles
 * every operator.  The fast kernel is taken where it applies until the other is
 * chosen (EDK_DISABLE_FAST=1 in the environment at an operator's creation chooses
 * the row kernel from the start).
 * block = 1 applies four or more right-hand sides as one SpMM on the bond-family and materialised paths
 * (each nonzero located once for all columns, as colmn! does,
 * Operator.jl:417-465); block = 0 runs them one column at a time; block = -1
 * (the default) uses the SpMM matrix-free, and the columns on a materialised
 * matrix or a rank-searched sector (row-plan kernel).  On a materialised operator, EDK_KERNEL_MATERIALIZED /
 * EDK_KERNEL_MATERIALIZED_STAGED select its plain or shared-memory-staged
 * product (tps ignored).  Every
 * choice computes the same product as EDKit's mul! (Operator.jl:309-328).
 * No reference counterpart as a call: EDKit has one CPU kernel. */
#define EDK_KERNEL_FAST 0
#define EDK_KERNEL_GENERIC 1
#define EDK_KERNEL_MATERIALIZED 2
#define EDK_KERNEL_MATERIALIZED_STAGED 3  /* entries staged in shared memory by bulk copies */
edk_status edk_operator_configure(edk_operator* op, int32_t kernel, int32_t tps, int32_t block);

/* Autotuner: times every admissible (kernel, threads per state, index
 * search) combination — and, with EDK_TUNE_MATERIALIZE or when the operator
 * is already materialised, the materialised matrix — applying the operator to
 * `nvec` vectors of `dtype` (with nvec >= 4 also the SpMM form), then installs the fastest matrix-free choice
 * (index search on the basis, kernel and tps on the operator) and, when it
 * wins, the materialised matrix on top (kept only then).  Allocates two nvec x D work vectors for the duration.  Not
 * to be called while other calls use the operator or its basis. */
#define EDK_TUNE_MATERIALIZE 1
#define EDK_TUNE_MAX 24
typedef struct {
  int32_t kernel, search, tps, block;  /* the choice installed */
  double ms;                           /* its median time per application */
  int32_t ncand;                       /* candidates timed */
  int32_t cand_kernel[EDK_TUNE_MAX], cand_search[EDK_TUNE_MAX], cand_tps[EDK_TUNE_MAX],
      cand_block[EDK_TUNE_MAX];
  double cand_ms[EDK_TUNE_MAX];
} edk_tune_result;
edk_status edk_operator_autotune(edk_operator* op, int32_t dtype, int64_t nvec, int32_t flags,
                                 edk_tune_result* res);

/* y (+)= H x for an nvec-column block — mul!(y, H, x) Operator.jl:309-328
 * (accumulate=1) and H * x Operator.jl:372-394 (accumulate=0).  Synchronous:
 * returns when y is written (host or device). */
edk_status edk_apply(edk_operator* op, int32_t dtype, const void* x, void* y, int64_t nvec,
                     int64_t ldx, int64_t ldy, int32_t accumulate, int32_t ptr_kind);
/* Same with device pointers on a caller stream (cudaStream_t passed as void*);
 * does not synchronise, so it can be captured into a CUDA graph. */
edk_status edk_apply_async(edk_operator* op, int32_t dtype, const void* x, void* y,
                           int64_t nvec, int64_t ldx, int64_t ldy, int32_t accumulate,
                           void* stream);

/* Lanczos ground state.  Extends the CGS2 builder _lanczos_build!
 * (TimeEvolution.jl:250-306) with a tridiagonal eigensolve; replaces the
 * dense eigvals(Hermitian(H)) path of Operator.jl:287-292 for large D. */
typedef enum {
  EDK_PREC_FP64 = 0,  /* vectors and products in FP64 */
  EDK_PREC_MIXED = 1  /* FP32 vectors + FP32 products, FP64 alpha/beta/reorth
                         accumulation and tridiagonal solve, then FP64 refinement */
} edk_precision;

typedef struct {
  int32_t max_steps;     /* Lanczos steps (m); at most 12,791 on the batched engine */
  int32_t nev;           /* number of lowest eigenvalues wanted */
  double tol;            /* relative stop tolerance on the Ritz values; 0 = run max_steps */
  int32_t check_every;   /* steps between convergence checks */
  int32_t precision;     /* edk_precision */
  int32_t refine_steps;  /* FP64 refinement steps for EDK_PREC_MIXED */
  int32_t reorth;        /* 1 = full CGS2 reorthogonalisation (reference), 0 = none */
  int32_t complex_vectors; /* 1 = complex Krylov vectors even when H is real */
} edk_lanczos_opts;

typedef struct {
  int32_t steps;         /* Lanczos steps taken (last stage) */
  int32_t steps_low;     /* FP32 steps before refinement (mixed) */
  int32_t matvecs;
  int32_t breakdown;     /* 1 if the lucky-breakdown rule fired */
  double seconds;        /* wall time inside the call, device work included */
  double seconds_matvec; /* time in matvec kernels (CUDA events) */
  double seconds_reorth; /* time in orthogonalisation kernels (CUDA events) */
  double residual;       /* |beta_m * y_m| of the lowest Ritz pair */
  double seconds_setup;  /* workspace, start vector and step-graph set-up */
  double seconds_stage1; /* first Lanczos stage (FP64, or FP32 storage when mixed) */
  double seconds_refine; /* FP64 refinement stages (mixed precision) */
  int32_t refine_rounds; /* FP64 refinement restarts taken */
  int32_t checks;        /* convergence checks */
} edk_lanczos_diag;

/* v0: starting vector (dtype v0_dtype, host or device); evals: nev values.
 * alpha/beta (optional, may be NULL): the last stage's recurrence
 * coefficients, max_steps entries each (the first ones, where the FP64 refinement of a
 * mixed run took more steps). */
edk_status edk_lanczos_e0(edk_operator* op, const edk_lanczos_opts* opts, const void* v0,
                          int32_t v0_dtype, int32_t ptr_kind, double* evals, double* alpha,
                          double* beta, edk_lanczos_diag* diag);

/* The same Lanczos run returning the ground state as well: psi (host or
 * device, per ptr_kind, D elements) receives the normalised lowest Ritz
 * vector in the FP64 working dtype — EDK_F64 when the operator and v0 are
 * real, EDK_C128 otherwise (psi_dtype must say which).  With precision mixed
 * the vector comes from the FP64 refinement.  No single reference call: it
 * is the eigenvector half of eigen(SymTridiagonal) on _lanczos_build!'s basis
 * (TimeEvolution.jl:250-323). */
edk_status edk_lanczos_ground_state(edk_operator* op, const edk_lanczos_opts* opts,
                                   const void* v0, int32_t v0_dtype, int32_t ptr_kind,
                                   double* evals, void* psi, int32_t psi_dtype,
                                   edk_lanczos_diag* diag);

/* Adaptive Krylov exp(-iHt) psi — timeevolve (TimeEvolution.jl:563-577)
 * with the cache/controller of TimeEvolution.jl:166-520.  psi0 and out are
 * complex (EDK_C128 interleaved; out is N x nts column-major).  ts may be
 * unsorted; columns come back in the caller's order. */
typedef struct {
  double tol;            /* default 1e-10 */
  int32_t m_init;        /* default 30 */
  int32_t m_max;         /* default 60 */
  int32_t extend_step;   /* default 10 */
  int32_t nsample;       /* default 13 */
  int32_t bisect_iters;  /* default 12 */
  int32_t reuse_basis;   /* default 1 */
  int32_t extend_basis;  /* default 1 */
  int32_t normalize_output; /* default 0 */
  int32_t precision;     /* edk_precision: FP64 or mixed (FP32 Krylov vectors) */
} edk_krylov_opts;

typedef struct {
  int32_t basis_builds, basis_extensions, restarts, matvecs, total_times_served, max_dim_used;
  int32_t n_intervals;
  double accepted_intervals[64]; /* first 64 accepted interval lengths */
  double seconds;
} edk_krylov_diag;

/* Fill *opts with the reference defaults (TimeEvolution.jl:166-176). */
void edk_krylov_default_opts(edk_krylov_opts* opts);
edk_status edk_krylov_evolve(edk_operator* op, const edk_krylov_opts* opts, const void* psi0,
                             const double* ts, int64_t nts, void* out, int32_t ptr_kind,
                             edk_krylov_diag* diag);

/* Resumable Krylov evolution: the handle form of KrylovEvolutionCache
 * (TimeEvolution.jl:166-218) with timeevolve!(cache, t) and
 * timeevolve!(out, cache, ts) (TimeEvolution.jl:586-636).  create() checks the
 * options as the constructor does, stages psi0 (EDK_C128, host or device per
 * ptr_kind) as the anchor and builds the first Lanczos basis on the device.
 * evolve() advances the cache forward: ts must be non-decreasing and not
 * before the last time served (EDK_BACKWARD_TIME otherwise, with the
 * reference's message); out receives N x nts complex columns (EDK_C128,
 * host or device per ptr_kind).  The basis, the anchor and the diagnostics
 * carry over from call to call.  info() reports the anchor time, the last
 * served time, the current basis dimension and the accumulated diagnostics.
 * The operator must outlive the handle; calls on one handle are serialised
 * with the operator's other calls. */
typedef struct edk_krylov_cache edk_krylov_cache;
edk_status edk_krylov_cache_create(edk_operator* op, const edk_krylov_opts* opts,
                                   const void* psi0, int32_t ptr_kind, edk_krylov_cache** out);
edk_status edk_krylov_cache_evolve(edk_krylov_cache* cache, const double* ts, int64_t nts,
                                   void* out, int32_t ptr_kind);
edk_status edk_krylov_cache_info(const edk_krylov_cache* cache, double* t_anchor,
                                 double* t_latest, int32_t* m, edk_krylov_diag* diag);
edk_status edk_krylov_cache_destroy(edk_krylov_cache* cache);

/* Batched Lanczos over independent operators (momentum sectors of one chain,
 * or disorder instances): all matvecs of one step run as ONE kernel launch
 * over a tile queue, the whole step is captured in a CUDA graph.  v0s holds
 * the concatenated starting vectors (F64 or C128 per v0_dtype, host).
 * evals receives nops x opts->nev values. */
edk_status edk_batch_lanczos_e0(int32_t nops, edk_operator* const* ops,
                                const edk_lanczos_opts* opts, const void* v0s, int32_t v0_dtype,
                                double* evals, edk_lanczos_diag* diag);

/* Failure-detection self-test of the library's bounded device waits (the
 * staged materialised product's copy waits use the same helper): one block
 * waits, with a limit of `polls` polls, on a shared-memory barrier that
 * nothing completes, records the time-out and returns.  Returns EDK_TIMEOUT
 * with a message, and leaves the context usable, when the limit works.  No
 * reference counterpart (EDKit has no device waits). */
edk_status edk_selftest_bounded_wait(uint32_t polls);

/* Symmetric tridiagonal eigensolver used by the Lanczos/Krylov drivers
 * (eigen(SymTridiagonal(a, b)), TimeEvolution.jl:311-323): diagonal a[m],
 * off-diagonal b[m-1]; w receives ascending eigenvalues, Q (may be NULL) the
 * eigenvectors column-major m x m.  Returns 0 on success. */
int edk_tridiag_eigen(int m, const double* a, const double* b, double* w, double* Q);

/*
 * Eigenvector post-processing (base 2, L <= 32).
 *
 * schmidt(v, Ainds, b) — src/Schmidt.jl:186-336 (TensorBasis / ProjectedBasis,
 * TranslationalBasis, TranslationParityBasis and TranslationFlipBasis through
 * parity_schmidt, FlipBasis, ParityBasis, ParityFlipBasis) and
 * src/Basis/AbelianBasis.jl:704-719 (AbelianBasis): the 2^nA x 2^(L-nA)
 * Schmidt matrix of the sector vector v (length D, F64 or C128), column-major
 * M[ia + ib * 2^nA].  Ainds: nA 1-based sites of subsystem A; row index =
 * A digits big-endian in Ainds order, column index = the remaining sites
 * ascending (schmidtmatrix, Schmidt.jl:39-57).  M is C128, or F64 when v is
 * F64 and the basis phases are real.  ptr_kind applies to v and M.
 */
edk_status edk_schmidt(const edk_basis* b, int32_t vdtype, const void* v, int32_t nA,
                       const int32_t* Ainds, void* M, int32_t mdtype, int32_t ptr_kind);
/* ent_spec(v, Aind, b) — Schmidt.jl:84: singular values of the Schmidt matrix,
 * descending, into s (host, min(2^nA, 2^(L-nA)) values, count in *ns; s may
 * be NULL to query the count).  Computed as square roots of the eigenvalues
 * of the Gram matrix of the smaller side (cuBLAS SYRK/HERK, then the library's
 * tridiagonalisation in shared memory up to 1,024 rows and cuSOLVER
 * SYEVD/HEEVD above); squared values below n * eps * max are returned as 0.
 * min side <= 32768.  ptr_kind applies to v. */
edk_status edk_ent_spec(const edk_basis* b, int32_t vdtype, const void* v, int32_t nA,
                        const int32_t* Ainds, double* s, int64_t* ns, int32_t ptr_kind);
/* ent_S(v, Aind, b; α, cutoff) — Schmidt.jl:101-153: entropy of the squared
 * Schmidt values (α = 1: von Neumann with the cutoff break; α = 0: the count
 * of values above the cutoff, as the reference returns it; otherwise Rényi
 * log(Σ s^α) / (1 - α)). */
edk_status edk_ent_S(const edk_basis* b, int32_t vdtype, const void* v, int32_t nA,
                     const int32_t* Ainds, double alpha, double cutoff, double* S,
                     int32_t ptr_kind);
/* (B::DoubleBasis)(v) with B = DoubleBasis(B1, B2) — src/LinearMap.jl:140-166:
 * out (C128, length D1) = Σ over full-space states of
 * conj(c1 / order(B1)) * (c2 / order(B2)) * v[pos2], where (c, pos) = index().
 * Both bases on one device with the same L and base
 * (check_doublebasis_compatible, LinearMap.jl:38-42).  ptr_kind applies to v
 * and out. */
edk_status edk_double_basis_apply(const edk_basis* B1, const edk_basis* B2, int32_t vdtype,
                                  const void* v, double* out, int32_t ptr_kind);
/* symmetrizer(DoubleBasis(B1, B2)) — LinearMap.jl:183-185 with
 * basis_embedding :57-70: the D1 x D2 C128 matrix
 * basis_embedding(B1)' * basis_embedding(B2), column-major. */
edk_status edk_symmetrizer(const edk_basis* B1, const edk_basis* B2, double* M,
                           int32_t ptr_kind);

/* last error message of the calling thread ("" if none) */
const char* edk_last_error(void);
/* library version string */
const char* edk_version(void);

#ifdef __cplusplus
}
#endif
#endif /* EDK_H */
