// Launch wrappers of the box-QP kernels (definitions in kernels.cu).
#pragma once
#include "engine.cuh"

namespace bqp {

// Computes each tile kernel's full wave (SMs x resident blocks per SM); returns the largest.
// Call once before launching.  The `grid` argument of the launchers below is a cap: each
// kernel launches min(cap, its own full wave) blocks.
int tile_grid(int sms);
// resident blocks of the CG product kernel (after tile_grid)
int cg_matvec_slots();
// Tile kernels: grid-stride over the tile table (the grid size is fixed at capture).
// dependent: the first overlaps the launch before it (false behind a conditional node or nothing)
void launch_check(const View& v, int families, int grid, bool dependent, cudaStream_t s);
// Step j of a body: the step kernel of one group (step_group(precision, variant)) over the group's
// tiles, or the FP64_EXACT step over the whole table.
void launch_step_group(const View& v, int group, int j, int grid, cudaStream_t s);
void launch_step_exact(const View& v, int j, int grid, cudaStream_t s);
// Check kernels of a body: one per family that has instances (bits of kCheck*).
constexpr int kCheckFp64 = 1;    // FP64 engines over the CSR
constexpr int kCheckSlices = 2;  // FP64 engines over sliced rows
constexpr int kCheckMixed = 4;   // mixed engine over the CSR: the FP32 iterate and the polished point (two kernels)
constexpr int kCheckMixedSlices = 8;  // the same over sliced rows
constexpr int check_launches(int families) {
    return ((families & kCheckFp64) ? 1 : 0) + ((families & kCheckSlices) ? 1 : 0) + ((families & kCheckMixed) ? 2 : 0) +
           ((families & kCheckMixedSlices) ? 2 : 0);
}
// Residual and CG product kernels of a body (kCheckMixed, kCheckMixedSlices of `families`).
constexpr int polish_launches(int families) { return ((families & kCheckMixed) ? 1 : 0) + ((families & kCheckMixedSlices) ? 1 : 0); }
void launch_polish_init(const View& v, int grid, cudaStream_t s);
void launch_polish_residual(const View& v, int families, int grid, cudaStream_t s);
void launch_cg_matvec(const View& v, int families, int grid, cudaStream_t s);
// cap > 0 (inside a graph): the last of a body's kCgTurns also sets cg_loop, the WHILE handle of the CG
// loop, allowing at most `cap` iterations per polish branch.  cap = 0: no handle is touched (host-driven launches).
// products: product kernels launched before it (for the count of kernels)
void launch_cg_vector(const View& v, int products, int grid, cudaStream_t s, cudaGraphConditionalHandle cg_loop = 0, int cap = 0,
                      int turn = 0);
// Single-block kernels that steer the conditional graph nodes (in_graph; else they touch no handle).
// Kernels of a body, for the count of kernels.
struct StepLaunches {
    int n[3];          // precision-k step launches
    int checks;
    int polish;        // kernels at the head of the polish branch
    unsigned present;  // bit k: the graph has steps for precision k (bit 1: and the polish)
    unsigned always;   // bit k: outside an IF node
};
// After the steps of a body (`steps`: per instance at most): chunks advance; polish: the IF node of the polish
// branch; cg_loop: the WHILE node of its CG loop.
void launch_advance(const View& v, cudaGraphConditionalHandle polish, cudaGraphConditionalHandle cg_loop, StepLaunches body,
                    int steps, bool in_graph, bool dependent, cudaStream_t s);
// After the checks.  fista[k]: the IF node of the precision-k steps; loop: the WHILE node around the body.
void launch_gate(const View& v, const cudaGraphConditionalHandle* fista, cudaGraphConditionalHandle loop, StepLaunches body,
                 int steps, bool ends_body, bool in_graph, cudaStream_t s);
// Admission, first kernel: the convexity gate and Gershgorin bound of the uploaded full CSR
// (FP64 values `val`) into *rec.gate (cleared first), the FP64 diagonal into rec.diag and, for the
// mixed engine, the hi/lo FP32 values into rec.vhi/rec.vlo.  The later admission kernels read L there.
// position_of: the columns are positions already (launch_slice_columns); the diagonal goes there too.
void launch_gate(const InstDev& rec, int64_t n, const double* val, bool split, const uint8_t* position_of, cudaStream_t s);
// Admission of a sliced instance, three kernels: the order of its rows (slice_len, slice_row, slice_base of
// `rec`; its vectors c, l, u, diag, where given, move into that order in place) from the uploaded row
// pointers, with each row's position in its window in position_of (n bytes); the uploaded columns as
// positions, in place (below `columns`); and the entries in slice order into col_out and val_out, or,
// for the mixed engine, as FP32 pairs.
void launch_slice_order(const InstDev& rec, int64_t n, const int32_t* rowptr, uint8_t* position_of, cudaStream_t s);
void launch_slice_columns(int64_t nnz, int64_t columns, int32_t* col, const uint8_t* position_of, cudaStream_t s);
void launch_slice_entries(const InstDev& rec, int64_t n, int64_t nnz, const int32_t* rowptr, const int32_t* col,
                          const double* val, int32_t* col_out, double* val_out, cudaStream_t s);
void launch_slice_entries_split(const InstDev& rec, int64_t n, int64_t nnz, const int32_t* rowptr, const int32_t* col,
                                const double* val, int32_t* col_out, float* hi_out, float* lo_out, cudaStream_t s);
// x of a sliced instance in row order: out[row] = x[position].
void launch_unslice(int64_t n, const uint8_t* slice_row, const double* x, double* out, cudaStream_t s);
// The same pass on raw device pointers (diag, vhi, vlo may be null: not stored).
void launch_gate_raw(int64_t n, const int32_t* rowptr, const int32_t* col, const double* val, GateResult* out,
                     double* diag, float* vhi, float* vlo, const uint8_t* position_of, cudaStream_t s);
// Admission, mixed engine, after launch_gate on the same stream: 1/diag, preconditioner scales and
// the FP32 cost and bounds (nothing for the FP64 engines).
// The record is passed by value: the instance is installed in its slot later, between graph launches.
void launch_prepare_instance(const InstDev& rec, int64_t n, cudaStream_t s);
// Mixed engine: per-row FISTA steps (diagonally preconditioned when `scaled`, else 1/L), after
// launch_prepare_instance on the same stream; val = the FP64 values.  With rec.lip_device the
// power estimate replaces the Gershgorin bound (power_scratch: power_scratch_bytes()).
void launch_precondition(const InstDev& rec, int64_t n, const double* val, bool scaled, void* power_scratch,
                         cudaStream_t s);
// BQP_LIPSCHITZ_POWER: Lanczos on the power iteration's Krylov space of S Q S (S = diag(rec.s)
// when `scaled`), FP64, at admission; *rec.lprec holds the Gershgorin bound of that matrix before
// and the estimate after.  scratch: power_scratch_bytes(n) bytes of device memory, 256-aligned.
size_t power_scratch_bytes(int64_t n);
void launch_power_lipschitz(const InstDev& rec, int64_t n, const double* val, bool scaled, void* scratch, cudaStream_t s);
// Re-arm of resident solves: records staged in page-locked host memory (read from there by the kernel),
// spans (staged index, first row) of kRearmRows rows each, one block per span.
void launch_rearm(const View& v, const InstDev* stage, const int32_t* slots, const int2* spans, int n_spans,
                  cudaStream_t s);

// After a launch: statuses, the control block and, of the solves that have finished, the records and
// primals in row order, written to where `jobs` says (spans: job index, first row; all page-locked).
void launch_collect(const View& v, const CollectJob* jobs, const int2* spans, int n_spans, int32_t* statuses, Ctrl* ctrl,
                    cudaStream_t s);
// One launch in place of a copy per array: pieces of page-locked host memory,
// 4-byte multiples.
struct UploadPieces {
    static constexpr int kMost = 8;
    int count = 0;
    const uint32_t* src[kMost];
    uint32_t* dst[kMost];
    uint32_t words[kMost];
};
void launch_upload(const UploadPieces& p, cudaStream_t s);

// Standalone FP64 check on caller device arrays (one instance, block partials in scratch).
// scratch must hold check_scratch_bytes(n) bytes.
size_t check_scratch_bytes(int64_t n);
int check_grid(int64_t n);
void launch_check_standalone(int64_t n, const int32_t* rowptr, const int32_t* col, const double* val,
                             const double* x, const double* c, const double* l, const double* u,
                             double tol, double offset, int gate, void* scratch, double* result,
                             cudaStream_t s);
// Loads the standalone check kernel into the current context now (under lazy module loading
// its first launch would load it) and opts it into its shared-memory size.
cudaError_t load_check_standalone();

// Plugin-level FISTA step (reference numerics: FP64, division by L, no FMA), ping-pong w.  The
// problem over the uploaded CSR, or over sliced rows (slice_len set: every array in slice order,
// the launches of one stream chained by programmatic dependent launch).
struct BoxStep {
    int64_t n;
    const int32_t* rowptr;
    const uint8_t* slice_len;
    const int32_t* slice_base;
    const int32_t* col;
    const double* val;
    const double* c;
    const double* l;
    const double* u;
    KnownDivisor L;
};
void launch_box_step(const BoxStep& b, double beta, double* x, const double* w_in, double* w_out, cudaStream_t s);

}  // namespace bqp
