// Device-side data layout of the box-QP engine (shared by the kernels and the host engine).
//
// One resident solve ("instance") owns a device slab holding its CSR and vectors; a
// batch is an array of instance records plus a table of row tiles.  Every kernel is a
// grid-stride loop over the tile table, reads the tile's instance record, and skips
// instances that are not in the phase the kernel serves, so one captured graph serves
// any mix of instances that are admitted, iterating, polishing or retired.
#pragma once
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

namespace bqp {

constexpr int kBlock = 256;          // threads per CTA of every tile kernel
constexpr int kMaxInterval = 32;     // maximum check interval (iterations per chunk)
constexpr int kTileNnz = 4096;       // target nonzeros per tile
constexpr int kTileRows = 512;       // maximum rows per tile
constexpr int kCgUnitMin = 2;        // tiles per work unit of the polish CG product: about
constexpr int kCgUnitMax = 8;        //   this many at least, and up to this many for large instances (work_units)
constexpr int kCgSmall = 16;         // tiles up to which a mixed instance's units are single tiles (work_units)
constexpr int kCgRowsum = 4 * kTileRows;  // rows per CG work unit at most (its row sums, 16 KB)
constexpr int kCgTurns = 4;          // CG iterations per body of the graph's CG loop (a body's start costs 4 us, an idle turn 2)
constexpr int kCgGroups = 2;         // row groups per warp whose loads the CG product keeps in flight
constexpr int kCgUnroll = 2;         // entries per row group and lane (and epilogue rows per thread) per pass of the CG product
constexpr int kMomentumTable = 8192; // FISTA momenta kept in a table (View::momentum)
constexpr int kRearmRows = 1024;     // rows per block when re-arming resident solves (8192: 32 us on 1M rows, latency-bound)
constexpr int64_t kHostPrimal = 131072;  // primals up to this size come back at completion, larger at fetch

enum Phase : int32_t {
    PH_FISTA = 0,        // FISTA iterations (FP64 or FP32 per precision)
    PH_POLISH_INIT = 1,  // FP64 free-set polish: snap the active set, start CG
    PH_POLISH_CG = 2,    // FP64 conjugate gradient on Q_FF
    PH_POLISH_FINISH = 3,  // CG done, xp clipped: the next check verifies the polished point
    PH_DONE = 4
};

enum Status : int32_t {
    ST_OPTIMAL = 0,
    ST_ITERATION_LIMIT = 1,
    ST_TIME_LIMIT = 2,
    ST_NUMERICAL_ERROR = 3,
    ST_RUNNING = 101
};

enum Precision : int32_t { PREC_FP64 = 0, PREC_MIXED = 1, PREC_FP64_EXACT = 2 };

// SpMV structure of a tile's step kernel (chosen per instance by the autotuning table).
enum Variant : int32_t {
    VAR_TILE = 0,    // block-staged: products of the whole tile, then one thread per row
    VAR_WARP = 64,   // warp-staged: 32 rows per warp, products then one lane per row
    VAR_SLICE = 65,  // sliced rows (below): one lane per row over interleaved entries
    VAR_SLICE_SMALL = 66,  // the same for small instances: whole rows loaded ahead of the previous step's end
    // 1, 2, 4, 8, 16, 32: sub-warp rows, that many lanes per row
};

// Step-kernel groups: one kernel per (precision, variant) for the FP64 and mixed engines, each
// over its own list of tiles, so a kernel carries one SpMV structure and the registers of that
// structure alone (the FP64_EXACT engine has one structure and no groups).
constexpr int kVariants = 10;
constexpr int kExactSlices = 2 * kVariants;  // the FP64_EXACT engine's sliced instances, then the small ones
constexpr int kStepGroups = 2 * kVariants + 2;
__host__ __device__ constexpr bool is_sliced(int variant) { return variant == VAR_SLICE || variant == VAR_SLICE_SMALL; }
__host__ __device__ constexpr int variant_index(int variant) {
    return variant == VAR_SLICE_SMALL ? 9 : variant == VAR_SLICE ? 8 : variant == VAR_WARP ? 7 : variant == 32 ? 6 : variant == 16 ? 5 : variant == 8 ? 4 : variant == 4 ? 3
         : variant == 2 ? 2 : variant == 1 ? 1 : 0;
}
__host__ __device__ constexpr int step_group(int precision, int variant) {
    return precision == PREC_FP64_EXACT ? (is_sliced(variant) ? kExactSlices + (variant == VAR_SLICE_SMALL) : -1) : (precision == PREC_MIXED ? kVariants : 0) + variant_index(variant);
}

// Sliced rows (VAR_SLICE).  The rows of each window of kSliceWindow rows are ordered by descending
// length (ties in row order), and the whole instance is kept in that order: position p of a window
// holds one of its rows, every vector is stored by position and the columns are positions.  A
// slice is 32 consecutive positions, one per lane of a warp.  A slice's entries are stored column by
// column without padding: first the first entry of each of its rows, then the second entry of
// each row that has one, and so on.  Because the rows of a slice are in descending length, the rows
// still active at any column are its first lanes, so every load of values, columns and vectors is
// one dense run, each row's sum runs in its own lane in column order (no shuffles, the per-row
// epilogue on full warps), and the lanes of a warp finish nearly together.  The entries of a window
// keep their CSR extent; the order is undone when the primal is handed out.
constexpr int kSliceWindow = 256;
constexpr int kSlicePiece = 128;     // rows of a step work item (a block's four warps take a slice each)
constexpr int64_t kSliceSmall = 65536;  // rows up to which an instance is VAR_SLICE_SMALL
constexpr int kSliceMaxRow = 127;    // longest row of a sliced instance (a window's entries stay within 16-bit offsets; its tiles
                                     // are whole windows, one at least, whatever they hold)
constexpr int kSliceMaxAverage = 48; // longer average rows keep the sub-warp structures (choose_variant)

// Mixed instances longer than this on average keep the sub-warp structures: their FP32 steps are bound by the
// gathers on either layout, while admission and the residual pass cost more on slices.
constexpr int kSliceMaxAverageMixed = 20;
// Order of a row's FP32 sum in the sliced mixed step for a named structure (kernel_variant), the one that
// structure's own kernel has, so that the layout does not change the iterates: 0 rounded products summed
// in column order (block- and warp-staged), 1 fused in column order, 2 two interleaved fused sums (one or
// two lanes per row); -1: none (more lanes keep their CSR kernels).
inline int slice_sums(int variant) {
    return variant == VAR_TILE || variant == VAR_WARP ? 0 : variant == 1 || variant == 2 ? variant : -1;
}
inline bool sliceable(int64_t n, int64_t nnz, int64_t longest_row) {
    return n > 0 && nnz > 0 && longest_row <= kSliceMaxRow && nnz < kSliceMaxAverage * n;
}

struct Tile {
    int32_t inst;
    int32_t row_begin;
    int32_t row_end;
    int32_t variant;  // Variant, or lanes per row (1..32)
};

// Per-tile partial results of one check (or of one CG reduction).  Sums are plain FP64 reduced in
// a fixed tree; maxima of non-negative doubles travel as their IEEE bit patterns, whose unsigned
// integer order is the numeric order, so they reduce on the integer pipes.
struct __align__(16) Partial {
    double obj;           // objective terms
    double bnd;           // tangent dual-bound terms
    double sep;           // separable dual-bound terms
    double a;             // CG: dot product
    uint64_t stat;        // max stationarity (bits)
    uint64_t prim;        // max scaled bound violation (bits, >= +0)
    uint64_t b;           // CG: max scaled residual (bits)
    uint64_t hash;        // active-set signature
    int64_t n_active;     // variables at a bound
    int32_t flags;        // bit0: non-finite x, bit1: infinite bound target
    int32_t pad;
};

// The convexity gate of an instance, computed on the device at admission from the uploaded full
// CSR (convexity_gate_kernel): the fast path of check_convex_hessian (src/qp_admm.cpp:30-39) and the
// Gershgorin bound of src/accelerated_qp.cpp:25-26.  Flags are 0/1, OR-reduced over the rows.
struct __align__(16) GateResult {
    unsigned long long lip_bits;  // max_i sum_k |Q_ik|, row sums in column order, as double bits
    int32_t indefinite;           // a row with Q_ii < 0, or Q_ii = 0 beside an off-diagonal entry
    int32_t nondominant;          // a row with Q_ii < sum_{j != i} |Q_ij| (diagonal dominance fails)
    unsigned long long floor_bits;  // during the pass: the largest lower bound of a row sum seen yet
    int32_t flags;                  // kGate* bits below
    int32_t pad;
};
constexpr int32_t kGateInvalid = 1;      // an entry whose column is out of range or whose value is not finite
constexpr int32_t kGateNonzero = 2;      // some value is not zero
constexpr int32_t kGateOffDiagonal = 4;  // some nonzero value lies off the diagonal
constexpr int32_t kGateNonPositive = 8;  // some row has Q_ii <= 0 (or no diagonal entry)

struct __align__(16) InstDev {
    // problem
    const int32_t* rowptr;
    const int32_t* col;
    const double* val64;   // FP64 values (PREC_FP64, PREC_FP64_EXACT)
    const float* vhi;      // FP32 high part (PREC_MIXED)
    const float* vlo;      // FP32 low part, val ~= hi + lo (PREC_MIXED)
    const uint8_t* slice_len;    // VAR_SLICE: per position, the row's length
    const uint8_t* slice_row;    // VAR_SLICE: per position, the row within its window
    const int32_t* slice_base;   // VAR_SLICE: per slice, its first entry in col / val64 (vhi, vlo)
    const double* c;
    const double* l;
    const double* u;
    const float* c32;
    const float* l32;      // smallest float >= l
    const float* u32;      // largest float <= u
    const double* diag;    // FP64 diagonal of Q
    const double* dinv;    // 1 / diagonal (mixed: Jacobi preconditioner of the polish)
    // iterates
    union {
        double* x64;       // FP64 engines: the iterate
        double* xf;        // mixed engine: the polish's x on the free-list positions (below)
    };
    double* w64[2];
    float* x32;
    float* w32[2];
    double* xp;            // polished point (FP64)
    float2* xp2;           // xp as an FP32 pair (hi, lo) for FP32-only gathers
    // The polish's CG vectors live on free-list positions: free row j of a tile is position
    // row_begin + j (each tile's free rows packed at the front of its row range), so the CG
    // kernels stream them without the row indices, and Q_FF's packed columns are positions.
    float2* p2;            // CG: u as an FP32 pair (gathered by the product)
    double* r;
    double* p;
    double* q;             // CG: w = Q_FF u
    double* s;             // polish: s = Q p (Chronopoulos-Gear CG)
    double* z;             // CG: u = M^-1 r
    int4* xq;              // polish: per row the snapped point's FP32 pair (x, y as bits) and the row's
                           // free-list position (z; -1 held at a bound): one 16-byte gather per entry
                           // of the residual pass's products
    int32_t* pos_of;       // polish: the free-list positions alone (-1 held at a bound), for its count
    int32_t* free_rows;    // polish: free rows of each tile, listed from the tile's first row (sliced: their
                           // positions, in row order)
    int32_t* free_cnt;     // polish: free rows per tile (index within the instance's tiles)
    int32_t* col_ff;       // polish: the free-column entries of a tile's free rows, packed row
    float* hi_ff;          //   after row (list order) from the start of the tile's own extent
    float* lo_ff;          //   [rowptr[row_begin], ...): row r at [start_ff[r], + cnt_ff[r])
    int32_t* cnt_ff;
    int32_t* start_ff;     //   (sliced: 32 list positions a slice, entries interleaved column by column as in
                           //   the matrix, the slice's first entry at start_ff[its first position])
    double* pc_inv;        // polish preconditioner, per free-list position: 1 / pivot of the chain factorization (1 / Q_rr on a Jacobi row)
    double* pc_e;          //   and the kept coupling to the next position (0 ends a chain)
    int32_t* pc_tile;      //   per tile (index within the instance): 1 when the tile has a chain
    unsigned long long stat_floor;  // within a running check: the largest stationarity ratio (FP64
                                    // bits) published so far; rows that cannot exceed it skip the division
    // geometry (the instance's tile range lives in View::ranges)
    int64_t nnz;
    int32_t sum_lanes;     // sliced mixed steps: the order of a row's FP32 sum (slice_sums)
    int32_t n;
    int32_t diag_gate;
    // control
    int32_t status;
    int32_t phase;
    int32_t interval;
    int32_t polish_rounds;
    int32_t precision;
    int32_t polish;        // mixed: free-set polish enabled
    int32_t arm_chunk;     // 1: admission arms the first chunk without a check of x0 (mixed)
    int32_t lip_device;    // 1: L is the device power estimate in *lprec (BQP_LIPSCHITZ_POWER)
    int32_t moved[2];      // mixed: a variable entered or left a bound in the chunk's last two steps
    float* sstep;          // mixed, preconditioned: per-row step 1 / (L' Q_ii) (null: scalar 1/L)
    double* lprec;         // L' of the preconditioned mixed engine, or the power estimate of L (device-computed at admission)
    GateResult* gate;      // the admission's convexity gate and Gershgorin bound (convexity_gate_kernel)
    int32_t lanes_res;     // polish: lanes per row of the residual pass (full rows)
    int32_t lanes_cg;      // polish: lanes per row of the CG products (free-free rows) and of the mixed checks
    int64_t it0;          // first iteration of the current chunk (beta[k] is iteration it0 + k)
    int64_t it_cur;        // iteration of the body's first step launch; a chunk may span bodies
    int64_t it_next;       // iteration of the next check
    int64_t max_iter;
    int64_t deadline_ns;   // %globaltimer deadline
    int64_t start_ns;
    int64_t end_ns;
    double L;
    double invL;
    double invL_lo;        // exact engine, sliced: 1/L - invL, and the dividends' exponent range (KnownDivisor)
    float invLf;
    int32_t div_span;
    int32_t result_src;    // where the answer lives: 0 x64, 1 x32, 2 xp
    double tol;
    double offset;
    double t;              // FISTA t_k
    double beta[kMaxInterval];
    float beta32[kMaxInterval];  // the same rounded to FP32, for the mixed steps (no per-tile conversion)
    // last check
    double objective;
    double primal_res;
    double stationarity;
    double dual_bound;
    double rel_gap;
    int32_t verified;
    int32_t stable_checks;
    int64_t iterations;
    uint64_t active_hash;
    int64_t n_active;
    double best_stat;
    // polish (CG on the free set)
    double rz;
    double alpha;
    double beta_cg;
    double cg_res;
    double cg_tol;
    double polish_switch;  // stationarity that triggers the first polish attempt
    double step_switch;    // the same after a step-stable chunk (see after_check)
    int64_t cg_it;
    int64_t cg_total;
    int64_t cg_max;
    // accounting
    int64_t fista_iters;
    int64_t checks;
    int64_t ff_nnz;        // polish: entries of the packed Q_FF of the current polish round
    int64_t ff_rows;       // polish: free rows of the current polish round
    double polish_bytes;   // polish: algorithmic bytes of the residual passes and CG iterations
};
static_assert(sizeof(InstDev) % 16 == 0, "rearm_kernel copies records as 16-byte words");

// Division by a divisor known in advance, correctly rounded: hi = RN(1/b), lo = RN(1/b - hi), then
// q = RN(a hi + RN(a lo)) is within an ulp of a/b, r = a - q b is exact (one fused operation), and
// RN(q + r hi) is RN(a/b) (P. Markstein, IBM J. Res. Dev. 34, 1990; the two-part reciprocal of
// N. Brisebarre, J.-M. Muller and S. K. Raina, IEEE Trans. Computers 53, 2004).  Four FP64
// operations, where the general division takes several times as many.  The theorem wants every
// step clear of underflow and overflow: divisors of 2^-100..2^100 and dividends of biased exponent
// kDivLow.. kDivLow + kDivSpan; span 0 (divisor outside) and other dividends take the general division
// (a zero, whose sign the remainder would lose, stays as it is).
constexpr int kDivLow = 200, kDivSpan = 1647;
struct KnownDivisor {
    double b, hi, lo;
    int32_t span;
};
inline KnownDivisor known_divisor(double b) {
    KnownDivisor d{b, 1.0 / b, 0.0, 0};
    if (b >= 0x1p-100 && b <= 0x1p100) {
        d.lo = std::fma(-d.hi, b, 1.0) / b;  // the remainder is exact
        d.span = kDivSpan;
    }
    return d;
}

struct Ctrl {
    int32_t n_inst;        // instance records in use
    int32_t n_tiles;       // tiles in use
    int32_t n_units;       // CG work units in use (View::units)
    int32_t n_passes;      // check and residual work units in use, behind those
    int32_t bodies;        // loop bodies run in the current launch
    int32_t body_cap;      // stop the device loop after this many bodies
    int32_t running;       // instances still running (written by the gate kernel)
    int32_t n_fista[3];    // instances in the FISTA phase, per precision
    int32_t n_polish;
    int32_t error;         // non-zero: a kernel detected an inconsistency
    int32_t n_cg;          // instances that may still run CG iterations in this body
    int32_t n_cg_left[kCgTurns];  // n_cg as each turn's CG vector step of the loop's body found it
    int32_t cg_iters;      // CG iterations run in this body
    long long kernels;     // engine kernels executed by this launch (counted by gate/control)
    int32_t group_begin[kStepGroups + 1];  // step groups: [begin, end) in View::group_tiles
    int32_t check_due[3];  // instances due for each check family in the next body (0: its kernel returns at once)
    int32_t step_due[3];   // per precision: step launches of this body with work (later ones return at once)
};

// What the collect kernel hands out of one solve when a launch has ended (CollectSpan: its blocks).
struct CollectJob {
    int32_t slot;
    int32_t n;          // rows of the primal to write (0: the record alone)
    InstDev* record;    // page-locked
    double* x;          // page-locked, or device memory for a primal that bqp_fetch will copy
};
constexpr int kCollectRows = 1024;  // rows per block, whole slice windows

// Everything a tile kernel needs, passed by value.
struct View {
    InstDev* inst;
    const Tile* tiles;
    Partial* partial;
    int32_t* tile_done;    // per-instance count of finished tiles (check / CG reductions)
    Ctrl* ctrl;
    const int2* ranges;      // per-instance tile range [x, y) in the tile table; empty for an instance that is
                             // not in this launch, whatever its record says
    const Tile* group_tiles;     // the tiles (sliced instances: pieces of kSlicePiece rows) ordered by step group (Ctrl::group_begin)
    const double2* momentum;     // FISTA: beta_k and t_{k+1} for k < kMomentumTable (they depend on k alone)
    const int4* units;           // work units of the CG product, then those of the sliced checks and the residual
                                 // pass: x the first tile of a run of y consecutive tiles of one
                                 // instance, z the unit's index within the instance, w its unit count
};

}  // namespace bqp
