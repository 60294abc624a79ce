// Constrained-QP ADMM inner solve on the GPU: the linear system of the reference's ADMM x-update
// (02-software/solver/src/qp_admm.cpp:157-161)
//     K x = rhs,   K = H + sigma I + A' diag(rho) A
// with H (n x n) and A (m x n) resident in CSR (A' built once, by a stable transpose), solved by
// the reference's Jacobi-preconditioned CG (qp_admm.cpp:262-273): r = rhs - K x, pre = r / M,
// d = pre, then while inner < max_inner and max|r| > accuracy: alpha = r'pre / d'K d (stop when
// that denominator is not positive and finite), x += alpha d, r -= alpha K d, beta = new r'pre /
// old, d = pre + beta d.  M = diag(H) + sigma + sum_i rho_i a_ij^2 as qp_admm.cpp:153-156 forms it
// (same order of additions, no FMA contraction: the same bits).
//
// One CUDA graph per system: the set-up kernels, then a WHILE node over one CG iteration (A d,
// then H d + sigma d + A'(rho A d) with the partial sums of d'K d, then the vector updates with
// the partial sums of r'pre and the maximum of |r|, then the new direction); the last block of
// each reduction finalizes it in a fixed order and sets the loop condition, so a solve is one
// graph launch with no host round trip per iteration.  FP64 throughout (the reference's inner
// products; its long double dot accumulation is not reproduced, so iterates agree to rounding).
//
// Systems whose rows allow it (sliceable: H's and A' rows together, and A's) keep sliced rows
// (engine.cuh): row j of H and row j of A' are one row over the stacked vector [v; t], so K v is one
// product with one lane per row, its sums without shuffles and its epilogue on full warps; every
// vector is in slice order and host vectors are permuted as they come and go.  The other systems
// keep CSR with four lanes per row.
#include "boxqp.h"
#include "fpbits.h"
#include "kernels.cuh"
#include "slices.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

namespace {

constexpr int kB = 256;
constexpr int kLanes = 4;         // lanes per CSR row
constexpr int kRows = kB / kLanes;
constexpr int kSms = 152, kMaxBlocks = kSms * 4;

struct AdmmState {
    double rz, alpha, beta;
    double accuracy;
    unsigned long long rmax;  // max |r| as the bit pattern of a non-negative double
    long long max_inner;
    long long inner;
    long long inner_sum;      // inner iterations over the ADMM iterations of one bqp_admm_iterate call
    unsigned ticket;
    int stop;                 // a non-positive or non-finite d'K d ended the loop
};

__device__ __forceinline__ unsigned long long umax64(unsigned long long a, unsigned long long b) { return a < b ? b : a; }
__device__ __forceinline__ unsigned long long dbits(double v) {
    return static_cast<unsigned long long>(__double_as_longlong(v));
}
// the bits of |v| in integer arithmetic (fpbits.h: bits64)
__device__ __forceinline__ unsigned long long abs_bits(double v) { return bqp::bits64(v) & 0x7fffffffffffffffull; }

// y = M v for rows [0, rows) of a CSR matrix, kLanes lanes per row in a fixed order; returns the
// row sum in the group's lane 0 (valid for r < rows).
__device__ __forceinline__ double csr_row(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                          const double* __restrict__ va, const double* __restrict__ v, int r, int rows,
                                          int sl) {
    double s = 0;
    if (r < rows) {
        const int ks = __ldg(rp + r), ke = __ldg(rp + r + 1);
        for (int k = ks + sl; k < ke; k += kLanes) s = fma(__ldg(va + k), v[__ldg(ci + k)], s);
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Fixed-order block sums of one or two doubles (TWO) and a maximum; the last block (ticket) adds the block
// partials, all its threads strided over them and then the same fixed tree, and returns true in
// its thread 0 with the grid totals.  A sum that nobody reads is left out: its additions take the
// FP64 pipe 16 cycles per warp and level.
template <bool TWO>
__device__ __forceinline__ void block_tree(double& a, double& b, unsigned long long& mx, double* ra, double* rb,
                                           unsigned long long* rm) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        if (TWO) b += __shfl_xor_sync(0xffffffffu, b, o);
        mx = umax64(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        ra[warp] = a;
        if (TWO) rb[warp] = b;
        rm[warp] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a = 0;
        b = 0;
        mx = 0;
        for (int w = 0; w < kB / 32; ++w) {
            a += ra[w];
            if (TWO) b += rb[w];
            mx = umax64(mx, rm[w]);
        }
    }
}

template <bool TWO>
__device__ bool reduce_last(double a, double b, unsigned long long mx, double* partial, AdmmState* st, double* ta,
                            double* tb, unsigned long long* tm) {
    __shared__ double ra[kB / 32], rb[TWO ? kB / 32 : 1];
    __shared__ unsigned long long rm[kB / 32];
    __shared__ int last;
    block_tree<TWO>(a, b, mx, ra, rb, rm);
    if (threadIdx.x == 0) {
        partial[3 * blockIdx.x] = a;
        if (TWO) partial[3 * blockIdx.x + 1] = b;
        partial[3 * blockIdx.x + 2] = __longlong_as_double(static_cast<long long>(mx));
        __threadfence();
        last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1 ? 1 : 0;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double sa = 0, sb = 0;
    unsigned long long sm = 0;
    for (unsigned k = threadIdx.x; k < gridDim.x; k += kB) {
        sa += __ldcg(partial + 3 * k);
        if (TWO) sb += __ldcg(partial + 3 * k + 1);
        sm = umax64(sm, dbits(__ldcg(partial + 3 * k + 2)));
    }
    block_tree<TWO>(sa, sb, sm, ra, rb, rm);  // thread 0 read the first tree's ra/rb/rm before the barrier above
    if (threadIdx.x != 0) return false;
    st->ticket = 0;
    *ta = sa;
    *tb = sb;
    *tm = sm;
    return true;
}

struct Sys {
    int n, m;
    const int32_t *hrp, *hci, *arp, *aci, *trp, *tci;
    const double *hva, *ava, *tva;
    const double* rho;
    double sigma;
    const double* precond;
    double* t;      // rho .* (A v), m
};

// t = rho .* (A v)
__global__ void __launch_bounds__(kB) admm_a_kernel(Sys s, const double* __restrict__ v, const AdmmState* st) {
    if (st->stop) return;
    const int sl = threadIdx.x % kLanes;
    for (int base = blockIdx.x * kRows; base < s.m; base += gridDim.x * kRows) {
        const int r = base + static_cast<int>(threadIdx.x) / kLanes;
        const double y = csr_row(s.arp, s.aci, s.ava, v, r, s.m, sl);
        if (r < s.m && sl == 0) s.t[r] = s.rho[r] * y;
    }
}

// out = H v + sigma v + A' t, then by mode:
//   0 (apply): nothing more;
//   1 (set-up, v = x): r = rhs - out, pre = r / M, d = pre; rz = r'pre, max|r|; the loop runs while
//     max_inner > 0 and max|r| > accuracy;
//   2 (iteration, v = d): d'out -> alpha = rz / d'out, or stop.
__global__ void __launch_bounds__(kB) admm_k_kernel(Sys s, const double* __restrict__ v, double* __restrict__ out,
                                                    int mode, const double* __restrict__ rhs, double* __restrict__ r,
                                                    double* __restrict__ pre, double* __restrict__ d, double* partial,
                                                    AdmmState* st, cudaGraphConditionalHandle loop) {
    if (mode == 2 && st->stop) return;
    const int sl = threadIdx.x % kLanes;
    double acc_a = 0, acc_b = 0;
    unsigned long long acc_m = 0;
    for (int base = blockIdx.x * kRows; base < s.n; base += gridDim.x * kRows) {
        const int j = base + static_cast<int>(threadIdx.x) / kLanes;
        const double hv = csr_row(s.hrp, s.hci, s.hva, v, j, s.n, sl);
        const double at = csr_row(s.trp, s.tci, s.tva, s.t, j, s.n, sl);
        if (j < s.n && sl == 0) {
            // the reference's expression, output[j] += sigma v[j] + product[j], unfused
            const double o = __dadd_rn(hv, __dadd_rn(__dmul_rn(s.sigma, v[j]), at));
            out[j] = o;
            if (mode == 1) {
                const double rr = __dsub_rn(rhs[j], o);
                const double pp = __ddiv_rn(rr, s.precond[j]);
                r[j] = rr;
                pre[j] = pp;
                d[j] = pp;
                acc_a = fma(rr, pp, acc_a);
                acc_m = umax64(acc_m, dbits(fabs(rr)));
            } else if (mode == 2) {
                acc_a = fma(v[j], o, acc_a);
            }
        }
    }
    if (mode == 0) return;
    double ta, tb;
    unsigned long long tm;
    if (!reduce_last<true>(acc_a, acc_b, acc_m, partial, st, &ta, &tb, &tm)) return;
    if (mode == 1) {
        st->rz = ta;
        st->rmax = tm;
        st->inner = 0;
        st->stop = 0;
        cudaGraphSetConditional(loop, (st->max_inner > 0 && __longlong_as_double(static_cast<long long>(tm)) > st->accuracy) ? 1u : 0u);
    } else {
        if (!(ta > 0) || !isfinite(ta)) st->stop = 1;
        else st->alpha = st->rz / ta;
    }
}

// x += alpha d, r -= alpha K d, pre = r / M; then rz, beta and the loop condition
__global__ void __launch_bounds__(kB) admm_update_kernel(Sys s, double* __restrict__ x, double* __restrict__ r,
                                                         double* __restrict__ pre, const double* __restrict__ d,
                                                         const double* __restrict__ kd, double* partial, AdmmState* st,
                                                         cudaGraphConditionalHandle loop) {
    if (st->stop) {
        if (blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(loop, 0u);
        return;
    }
    const double alpha = st->alpha;
    double acc_a = 0;
    unsigned long long acc_m = 0;
    for (int j = blockIdx.x * kB + threadIdx.x; j < s.n; j += gridDim.x * kB) {
        x[j] = __dadd_rn(x[j], __dmul_rn(alpha, d[j]));
        const double rr = __dsub_rn(r[j], __dmul_rn(alpha, kd[j]));
        const double pp = __ddiv_rn(rr, s.precond[j]);
        r[j] = rr;
        pre[j] = pp;
        acc_a = fma(rr, pp, acc_a);
        acc_m = umax64(acc_m, dbits(fabs(rr)));
    }
    double ta, tb;
    unsigned long long tm;
    if (!reduce_last<false>(acc_a, 0.0, acc_m, partial, st, &ta, &tb, &tm)) return;
    st->beta = ta / st->rz;
    st->rz = ta;
    st->rmax = tm;
    st->inner += 1;
    cudaGraphSetConditional(loop, (st->inner < st->max_inner && __longlong_as_double(static_cast<long long>(tm)) > st->accuracy) ? 1u : 0u);
}

// d = pre + beta d
__global__ void __launch_bounds__(kB) admm_direction_kernel(int n, double* __restrict__ d, const double* __restrict__ pre,
                                                            const AdmmState* st) {
    if (st->stop) return;
    const double beta = st->beta;
    for (int j = blockIdx.x * kB + threadIdx.x; j < n; j += gridDim.x * kB) d[j] = __dadd_rn(pre[j], __dmul_rn(beta, d[j]));
}

// ---- the same over sliced rows ------------------------------------------------------------------
// Bounds of an iteration on 1M variables, 15M + 2 x 4M entries: 23M random gathers (92 us at the
// 250 G/s this GPU gathers), 276 MB of entries (41 us), on the FP64 pipe 23M products and about
// eight operations a row (50 us); the L2 hands out a 32-byte sector per gathered number, which with
// the entries makes 104 us.  Now 152: A d 22, K d 100, update 20, direction and the loop 11 (two
// iterations per body of the loop: 157).  Four lanes per CSR row spent as much FP64 time again on tree
// additions and quarter-warp epilogues, and a general division per row: 217 us an iteration.
// Columns of a row in flight: 5 on large systems (64 registers; 4: 183, 8: 167 us an iteration), whole
// rows on small ones, which are bound by the latency of their loads.
constexpr int kAhead = 5, kAheadSmall = 16;
constexpr int64_t kSmallRows = 65536;
constexpr int kSliceBlocks = kMaxBlocks;  // their partial sums share the buffer of kMaxBlocks
struct SliceRows {
    int n;
    const uint8_t* len;
    const uint8_t* row;
    const int32_t* base;
    const int32_t* col;
    const double* val;
};
struct SliceSys {
    SliceRows k, a;       // [H, A'] over [v; t], and A over v
    int t0;               // where t begins in a stacked vector
    const double* rho;    // in A's slice order
    double sigma;
    const double* minv;   // 1 / M
};

// A warp's first slice, of a stride of gridDim.x * kB / 32: a block's warps take neighbours, or, where
// there are fewer slices than warps, the blocks share them out.
__device__ __forceinline__ int first_slice(int slices) {
    const int warp = threadIdx.x >> 5, blocks = gridDim.x;
    return slices < blocks * (kB / 32) ? warp * blocks + static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x) * (kB / 32) + warp;
}

// A lane's row of slice s: its sum (0 past the last row).  The first columns are loaded before
// `wait`, the wait for the launch that wrote the vector.
template <int AHEAD, class Wait>
__device__ __forceinline__ double slice_row_sum(const SliceRows& R, int s, const double* v, Wait wait) {
    const int p = s * 32 + static_cast<int>(threadIdx.x & 31);
    const int len = p < R.n ? __ldg(R.len + p) : 0;
    int k = __ldg(R.base + s) + static_cast<int>(threadIdx.x & 31);
    const int longest = __shfl_sync(0xffffffffu, len, 0);
    bqp::SliceColumns<AHEAD> e;
    e.load(R.col, R.val, len, k);
    wait();
    double acc = e.add<false>(v, longest, 0.0);
    for (int j = AHEAD; j < longest; j += AHEAD) {
        e.load(R.col, R.val, len - j, k);
        acc = e.add<false>(v, longest - j, acc);
    }
    return acc;
}

// Waits once for the launch before; then whether an earlier kernel ended the loop.
struct WaitOnce {
    bool waited = false;
    __device__ __forceinline__ void operator()() {
        if (!waited) bqp::wait_for_previous_launch();
        waited = true;
    }
};

// t = rho .* (A v), t behind v
template <int AHEAD>
__global__ void __launch_bounds__(kB, AHEAD > 8 ? 2 : 4) admm_a_slice_kernel(SliceSys S, double* v) {
    bqp::let_next_launch_begin();
    WaitOnce wait;
    const int slices = (S.a.n + 31) / 32;
    for (int s = first_slice(slices); s < slices; s += gridDim.x * (kB / 32)) {
        const double y = slice_row_sum<AHEAD>(S.a, s, v, wait);
        const int p = s * 32 + static_cast<int>(threadIdx.x & 31);
        if (p < S.a.n) v[S.t0 + p] = __ldg(S.rho + p) * y;
    }
    wait();
}

// out = K v by the modes of admm_k_kernel (0 apply, 1 set-up: v = x, 2 iteration: v = d)
template <int AHEAD>
__global__ void __launch_bounds__(kB, AHEAD > 8 ? 2 : 4) admm_k_slice_kernel(SliceSys S, const double* v, double* out, int mode, const double* rhs,
                                                         double* r, double* pre, double* d, double* partial, AdmmState* st,
                                                         cudaGraphConditionalHandle loop) {
    bqp::let_next_launch_begin();
    WaitOnce wait;
    double acc_a = 0;
    unsigned long long acc_m = 0;
    const int slices = (S.k.n + 31) / 32;
    for (int s = first_slice(slices); s < slices; s += gridDim.x * (kB / 32)) {
        const double sum = slice_row_sum<AHEAD>(S.k, s, v, wait);
        const int p = s * 32 + static_cast<int>(threadIdx.x & 31);
        if (p >= S.k.n) continue;
        const double vp = v[p], o = fma(S.sigma, vp, sum);
        out[p] = o;
        if (mode == 1) {
            const double rr = rhs[p] - o, pp = rr * __ldg(S.minv + p);
            r[p] = rr;
            pre[p] = pp;
            d[p] = pp;
            acc_a = fma(rr, pp, acc_a);
            acc_m = umax64(acc_m, abs_bits(rr));
        } else if (mode == 2) {
            acc_a = fma(vp, o, acc_a);
        }
    }
    wait();
    if (mode == 0) return;
    double ta, tb;
    unsigned long long tm;
    if (!reduce_last<false>(acc_a, 0.0, acc_m, partial, st, &ta, &tb, &tm)) return;
    if (mode == 1) {
        st->rz = ta;
        st->rmax = tm;
        st->inner = 0;
        st->stop = 0;
        cudaGraphSetConditional(loop, (st->max_inner > 0 && __longlong_as_double(static_cast<long long>(tm)) > st->accuracy) ? 1u : 0u);
    } else {
        if (!(ta > 0) || !isfinite(ta)) st->stop = 1;
        else st->alpha = st->rz / ta;
    }
}

// x += alpha d, r -= alpha K d, pre = r / M; then rz, beta and the loop condition
__global__ void __launch_bounds__(kB) admm_update_slice_kernel(int n, const double* __restrict__ minv, double* x, double* r,
                                                               double* pre, const double* d, const double* kd, double* partial,
                                                               AdmmState* st, cudaGraphConditionalHandle loop) {
    bqp::let_next_launch_begin();
    bqp::wait_for_previous_launch();
    if (st->stop) {
        if (blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(loop, 0u);
        return;
    }
    const double alpha = st->alpha;
    double acc_a = 0;
    unsigned long long acc_m = 0;
    for (int j = blockIdx.x * kB + threadIdx.x; j < n; j += gridDim.x * kB) {
        x[j] = fma(alpha, d[j], x[j]);
        const double rr = fma(-alpha, kd[j], r[j]), pp = rr * __ldg(minv + j);
        r[j] = rr;
        pre[j] = pp;
        acc_a = fma(rr, pp, acc_a);
        acc_m = umax64(acc_m, abs_bits(rr));
    }
    double ta, tb;
    unsigned long long tm;
    if (!reduce_last<false>(acc_a, 0.0, acc_m, partial, st, &ta, &tb, &tm)) return;
    st->beta = ta / st->rz;
    st->rz = ta;
    st->rmax = tm;
    st->inner += 1;
    cudaGraphSetConditional(loop, (st->inner < st->max_inner && __longlong_as_double(static_cast<long long>(tm)) > st->accuracy) ? 1u : 0u);
}

// d = pre + beta d
__global__ void __launch_bounds__(kB) admm_direction_slice_kernel(int n, double* d, const double* pre, const AdmmState* st) {
    bqp::let_next_launch_begin();
    bqp::wait_for_previous_launch();
    if (st->stop) return;
    const double beta = st->beta;
    for (int j = blockIdx.x * kB + threadIdx.x; j < n; j += gridDim.x * kB) d[j] = fma(beta, d[j], pre[j]);
}

// 1 / M, M as admm_precond_kernel forms it: a row holds its H entries, then its A' entries in increasing i
__global__ void __launch_bounds__(kB) admm_precond_slice_kernel(SliceSys S, double* __restrict__ minv) {
    const int slices = (S.k.n + 31) / 32;
    for (int s = first_slice(slices); s < slices; s += gridDim.x * (kB / 32)) {
        const int p = s * 32 + static_cast<int>(threadIdx.x & 31);
        const int len = p < S.k.n ? __ldg(S.k.len + p) : 0;
        const int longest = __shfl_sync(0xffffffffu, len, 0);
        int k = __ldg(S.k.base + s) + static_cast<int>(threadIdx.x & 31);
        double dg = 0, m = 0;
        bool head = true;
        for (int j = 0; j < longest; ++j) {
            const bool in = j < len;
            if (in) {
                const int c = __ldg(S.k.col + k);
                const double a = __ldg(S.k.val + k);
                if (c == p) dg = a;
                if (c >= S.t0) {
                    if (head) m = __dadd_rn(dg, S.sigma);
                    head = false;
                    m = __dadd_rn(m, __dmul_rn(__dmul_rn(__ldg(S.rho + c - S.t0), a), a));
                }
            }
            k += __popc(__ballot_sync(0xffffffffu, in));
        }
        if (head) m = __dadd_rn(dg, S.sigma);
        if (p < S.k.n) minv[p] = __ddiv_rn(1.0, m);
    }
}

// rhs = A'(rho z - y) + (sigma x - c), in two kernels: yz into t, then the A' part of the stacked rows
// (a row's H entries are skipped; its A' entries follow them)
__global__ void __launch_bounds__(kB) admm_yz_kernel(int m, const double* __restrict__ rho, const double* __restrict__ z,
                                                     const double* __restrict__ y, double* __restrict__ t) {
    for (int i = blockIdx.x * kB + threadIdx.x; i < m; i += gridDim.x * kB)
        t[i] = __dsub_rn(__dmul_rn(__ldg(rho + i), z[i]), y[i]);  // the reference's yz[i]
}

__global__ void __launch_bounds__(kB) admm_rhs_slice_kernel(SliceSys S, const double* __restrict__ stacked,
                                                            const double* __restrict__ xa, const double* __restrict__ c,
                                                            double* __restrict__ rhs, double* __restrict__ x0, double* partial,
                                                            AdmmState* st, double iteration_factor) {
    unsigned long long mx = 0;
    const int slices = (S.k.n + 31) / 32;
    for (int s = first_slice(slices); s < slices; s += gridDim.x * (kB / 32)) {
        const int p = s * 32 + static_cast<int>(threadIdx.x & 31);
        const int len = p < S.k.n ? __ldg(S.k.len + p) : 0;
        const int longest = __shfl_sync(0xffffffffu, len, 0);
        int k = __ldg(S.k.base + s) + static_cast<int>(threadIdx.x & 31);
        double acc = 0;
        for (int j = 0; j < longest; ++j) {
            const bool in = j < len;
            const int col = in ? __ldg(S.k.col + k) : 0;
            if (col >= S.t0) acc = fma(__ldg(S.k.val + k), __ldg(stacked + col), acc);
            k += __popc(__ballot_sync(0xffffffffu, in));
        }
        if (p < S.k.n) {
            const double v = __dadd_rn(acc, __dsub_rn(__dmul_rn(S.sigma, xa[p]), c[p]));
            rhs[p] = v;
            x0[p] = xa[p];
            mx = umax64(mx, abs_bits(v));
        }
    }
    double ta, tb;
    unsigned long long tm;
    if (!reduce_last<false>(0.0, 0.0, mx, partial, st, &ta, &tb, &tm)) return;
    const double rmax = __longlong_as_double(static_cast<long long>(tm));
    st->accuracy = __dmul_rn(iteration_factor, __dadd_rn(1.0, rmax));
    st->max_inner = S.k.n * 2LL + 20 < 4000 ? S.k.n * 2LL + 20 : 4000;
    st->stop = 0;  // a breakdown of the previous inner solve does not carry over
}

// admm_zy_kernel over sliced rows of A
__global__ void __launch_bounds__(kB, 4) admm_zy_slice_kernel(SliceSys S, const double* next, double* __restrict__ z,
                                                           double* __restrict__ y, const double* __restrict__ lo,
                                                           const double* __restrict__ up, AdmmState* st) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->inner_sum += st->inner;
    const int slices = (S.a.n + 31) / 32;
    for (int s = first_slice(slices); s < slices; s += gridDim.x * (kB / 32)) {
        const double ax = slice_row_sum<kAhead>(S.a, s, next, [] {});
        const int i = s * 32 + static_cast<int>(threadIdx.x & 31);
        if (i >= S.a.n) continue;
        const double zi = z[i], yi = y[i], ri = S.rho[i];
        const double relaxed = __dsub_rn(__dmul_rn(1.6, ax), __dmul_rn(.6, zi));
        const double w = __dadd_rn(relaxed, __ddiv_rn(yi, ri));
        const double t = w < up[i] ? w : up[i];  // std::max(lo, std::min(up, w))
        const double nz = lo[i] < t ? t : lo[i];
        y[i] = __dadd_rn(yi, __dmul_rn(ri, __dsub_rn(relaxed, nz)));
        z[i] = nz;
    }
}

// Row j of H, then row j of A' (its columns moved behind the variables, at t0), as one CSR row
__global__ void __launch_bounds__(kB) admm_stack_kernel(int n, int t0, const int32_t* __restrict__ hrp,
                                                        const int32_t* __restrict__ hci, const double* __restrict__ hva,
                                                        const int32_t* __restrict__ trp, const int32_t* __restrict__ tci,
                                                        const double* __restrict__ tva, int32_t* __restrict__ rp,
                                                        int32_t* __restrict__ ci, double* __restrict__ va) {
    const int lane = threadIdx.x % 8;
    if (blockIdx.x == 0 && threadIdx.x == 0) rp[n] = hrp[n] + trp[n];
    for (int j = (blockIdx.x * kB + static_cast<int>(threadIdx.x)) / 8; j < n; j += gridDim.x * kB / 8) {
        const int h0 = hrp[j], h = hrp[j + 1] - h0, t_at = trp[j], t = trp[j + 1] - t_at, o = h0 + t_at;
        if (lane == 0) rp[j] = o;
        for (int k = lane; k < h; k += 8) {
            ci[o + k] = hci[h0 + k];
            va[o + k] = hva[h0 + k];
        }
        for (int k = lane; k < t; k += 8) {
            ci[o + h + k] = t0 + tci[t_at + k];
            va[o + h + k] = tva[t_at + k];
        }
    }
}

// M = diag(H) + sigma + sum_i rho_i a_ij^2, row j of A' in increasing i (the reference's order)
__global__ void __launch_bounds__(kB) admm_precond_kernel(Sys s, double* __restrict__ precond) {
    for (int j = blockIdx.x * kB + threadIdx.x; j < s.n; j += gridDim.x * kB) {
        double dg = 0;
        for (int k = s.hrp[j]; k < s.hrp[j + 1]; ++k)
            if (s.hci[k] == j) dg = s.hva[k];
        double p = __dadd_rn(dg, s.sigma);
        for (int k = s.trp[j]; k < s.trp[j + 1]; ++k) {
            const double a = s.tva[k];
            p = __dadd_rn(p, __dmul_rn(__dmul_rn(s.rho[s.tci[k]], a), a));
        }
        precond[j] = p;
    }
}

// ---- the ADMM iteration around the inner solve (qp_admm.cpp:255-279) --------------------------
// rhs = A'(rho z - y) + (sigma x - c); the inner accuracy min(1e-7, .05 / (it+1)^1.6) (1 + max|rhs|)
// and the inner iteration cap go to the state the inner solve's set-up reads; x0 of the inner
// solve = x.
__global__ void __launch_bounds__(kB) admm_rhs_kernel(Sys s, const double* __restrict__ z, const double* __restrict__ y,
                                                      const double* __restrict__ xa, const double* __restrict__ c,
                                                      double* __restrict__ rhs, double* __restrict__ x0, double* partial,
                                                      AdmmState* st, double iteration_factor) {
    const int sl = threadIdx.x % kLanes;
    unsigned long long mx = 0;
    for (int base = blockIdx.x * kRows; base < s.n; base += gridDim.x * kRows) {
        const int j = base + static_cast<int>(threadIdx.x) / kLanes;
        double acc = 0;
        if (j < s.n) {
            const int ks = __ldg(s.trp + j), ke = __ldg(s.trp + j + 1);
            for (int k = ks + sl; k < ke; k += kLanes) {
                const int i = __ldg(s.tci + k);
                const double yz = __dsub_rn(__dmul_rn(s.rho[i], z[i]), y[i]);  // the reference's yz[i]
                acc = fma(__ldg(s.tva + k), yz, acc);
            }
        }
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (j < s.n && sl == 0) {
            const double v = __dadd_rn(acc, __dsub_rn(__dmul_rn(s.sigma, xa[j]), c[j]));
            rhs[j] = v;
            x0[j] = xa[j];
            mx = umax64(mx, dbits(fabs(v)));
        }
    }
    double ta, tb;
    unsigned long long tm;
    if (!reduce_last<false>(0.0, 0.0, mx, partial, st, &ta, &tb, &tm)) return;
    const double rmax = __longlong_as_double(static_cast<long long>(tm));
    st->accuracy = __dmul_rn(iteration_factor, __dadd_rn(1.0, rmax));
    st->max_inner = s.n * 2LL + 20 < 4000 ? s.n * 2LL + 20 : 4000;
    st->stop = 0;  // a breakdown of the previous inner solve does not carry over
}

// ax = A next; relaxed = 1.6 ax - .6 z; z+ = clip(relaxed + y / rho, lo, up); y += rho (relaxed - z+)
__global__ void __launch_bounds__(kB) admm_zy_kernel(Sys s, const double* __restrict__ next, double* __restrict__ z,
                                                     double* __restrict__ y, const double* __restrict__ lo,
                                                     const double* __restrict__ up, AdmmState* st) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->inner_sum += st->inner;
    const int sl = threadIdx.x % kLanes;
    for (int base = blockIdx.x * kRows; base < s.m; base += gridDim.x * kRows) {
        const int i = base + static_cast<int>(threadIdx.x) / kLanes;
        const double ax = csr_row(s.arp, s.aci, s.ava, next, i, s.m, sl);
        if (i < s.m && sl == 0) {
            const double zi = z[i], yi = y[i], ri = s.rho[i];
            const double relaxed = __dsub_rn(__dmul_rn(1.6, ax), __dmul_rn(.6, zi));
            const double w = __dadd_rn(relaxed, __ddiv_rn(yi, ri));
            const double t = w < up[i] ? w : up[i];  // std::max(lo, std::min(up, w))
            const double nz = lo[i] < t ? t : lo[i];
            y[i] = __dadd_rn(yi, __dmul_rn(ri, __dsub_rn(relaxed, nz)));
            z[i] = nz;
        }
    }
}

// x = 1.6 next - .6 x
__global__ void __launch_bounds__(kB) admm_x_kernel(int n, const double* __restrict__ next, double* __restrict__ xa) {
    for (int j = blockIdx.x * kB + threadIdx.x; j < n; j += gridDim.x * kB)
        xa[j] = __dsub_rn(__dmul_rn(1.6, next[j]), __dmul_rn(.6, xa[j]));
}

int grid_for(int rows, int per_block) {
    int g = (rows + per_block - 1) / per_block;
    return std::max(1, std::min(g, kMaxBlocks));
}

}  // namespace

struct bqp_admm {
    int device = 0;
    int64_t n = 0, m = 0;
    cudaStream_t stream = nullptr;
    // device arrays
    int32_t *hrp = nullptr, *hci = nullptr, *arp = nullptr, *aci = nullptr, *trp = nullptr, *tci = nullptr;
    double *hva = nullptr, *ava = nullptr, *tva = nullptr;
    double *rho = nullptr, *t = nullptr, *precond = nullptr;
    double *rhs = nullptr, *x = nullptr, *r = nullptr, *pre = nullptr, *d = nullptr, *kd = nullptr, *v = nullptr;
    double* partial = nullptr;
    AdmmState* st = nullptr;
    AdmmState* h_st = nullptr;
    // ADMM state of bqp_admm_iterate (allocated on first use): x, the cost, z, y and the
    // constraint bounds (one per row of A)
    double *xa = nullptr, *c = nullptr, *z = nullptr, *y = nullptr, *lo = nullptr, *up = nullptr;
    double sigma = 0;
    bool rho_set = false;
    // sliced rows (engine.cuh); x, d and v are then stacked vectors (t0 + m entries), rhs, r, pre, kd, xa, c
    // in the variables' slice order and rho, z, y, lo, up in the rows' of A
    bool sliced = false;
    int64_t t0 = 0;
    uint8_t *k_len = nullptr, *k_row = nullptr, *a_len = nullptr, *a_row = nullptr;
    int32_t *k_base = nullptr, *a_base = nullptr, *k_col = nullptr, *a_col = nullptr;
    double *k_val = nullptr, *a_val = nullptr, *stage = nullptr;  // stage: a host vector in its own order
    cudaGraph_t graph = nullptr, apply_graph = nullptr;
    cudaGraphExec_t exec = nullptr, apply_exec = nullptr;
    std::string error;

    Sys sys() const {
        Sys s;
        s.n = static_cast<int>(n);
        s.m = static_cast<int>(m);
        s.hrp = hrp; s.hci = hci; s.hva = hva;
        s.arp = arp; s.aci = aci; s.ava = ava;
        s.trp = trp; s.tci = tci; s.tva = tva;
        s.rho = rho;
        s.sigma = sigma;
        s.precond = precond;
        s.t = t;
        return s;
    }
    SliceSys slices() const {
        SliceSys s;
        s.k = SliceRows{static_cast<int>(n), k_len, k_row, k_base, k_col, k_val};
        s.a = SliceRows{static_cast<int>(m), a_len, a_row, a_base, a_col, a_val};
        s.t0 = static_cast<int>(t0);
        s.rho = rho;
        s.sigma = sigma;
        s.minv = precond;
        return s;
    }
    // host vectors of the variables (of the rows of A) to the device and back, through the slice order
    void put(double* dst, const double* src, int64_t count, const uint8_t* row) {
        if (count <= 0) return;
        cudaMemcpyAsync(sliced ? stage : dst, src, sizeof(double) * static_cast<size_t>(count), cudaMemcpyHostToDevice, stream);
        if (sliced) bqp::launch_slice_vector(count, row, stage, dst, stream);
    }
    void get(double* dst, const double* src, int64_t count, const uint8_t* row) {
        if (count <= 0) return;
        if (sliced) bqp::launch_unslice(count, row, src, stage, stream);
        cudaMemcpyAsync(dst, sliced ? stage : src, sizeof(double) * static_cast<size_t>(count), cudaMemcpyDeviceToHost, stream);
    }
    cudaError_t slice(int64_t hz, int64_t az);
    // K x (mode as admm_k_kernel), preceded by t = rho .* (A x); dependent: overlapping the launch before
    void launch_product(double* x_in, double* out, int mode, cudaGraphConditionalHandle h, bool dependent, cudaStream_t s) {
        const SliceSys S = slices();
        const bool small = n <= kSmallRows;
        if (m) launch(small ? admm_a_slice_kernel<kAheadSmall> : admm_a_slice_kernel<kAhead>, slice_grid(m, small), dependent, s, S, x_in);
        launch(small ? admm_k_slice_kernel<kAheadSmall> : admm_k_slice_kernel<kAhead>, slice_grid(n, small), m != 0 || dependent, s, S, static_cast<const double*>(x_in), out, mode,
               static_cast<const double*>(rhs), r, pre, d, partial, st, h);
    }
    template <class... P, class... A>
    static void launch(void (*kernel)(P...), int grid, bool dependent, cudaStream_t s, A... args) {
        cudaLaunchAttribute overlap;
        overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        overlap.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(static_cast<unsigned>(grid));
        config.blockDim = dim3(kB);
        config.stream = s;
        config.attrs = &overlap;
        config.numAttrs = dependent ? 1 : 0;
        cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
    }
    // A slice per warp as far as the resident blocks go (two of the small kernels on an SM), the same number of
    // blocks on each SM, no more than that takes: 38k rows 2.89 ms per 77 iterations with 608 blocks in
    // two rounds, 2.32 with 304, 2.05 with 152.
    static int slice_grid(int64_t rows, bool small = false) {
        const int64_t slices = (rows + 31) / 32, per_sm = (slices + kSms * (kB / 32) - 1) / (kSms * (kB / 32));
        const int64_t blocks = kSms * std::min<int64_t>(per_sm, small ? 2 : kSliceBlocks / kSms);
        return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(slices, blocks)));
    }
    bool ok(cudaError_t e, const char* what) {
        if (e == cudaSuccess) return true;
        error = std::string("CUDA: ") + what + ": " + cudaGetErrorString(e);
        return false;
    }
    // graphs are built once rho and sigma are known (sigma is a kernel argument)
    bool build() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (apply_exec) cudaGraphExecDestroy(apply_exec);
        if (apply_graph) cudaGraphDestroy(apply_graph);
        exec = nullptr; graph = nullptr; apply_exec = nullptr; apply_graph = nullptr;
        const Sys s = sys();
        const int gm = grid_for(static_cast<int>(m), kRows), gn = grid_for(static_cast<int>(n), kRows);
        const int gv = grid_for(static_cast<int>(n), kB);
        if (!ok(cudaGraphCreate(&graph, 0), "graph")) return false;
        cudaGraphConditionalHandle h;
        if (!ok(cudaGraphConditionalHandleCreate(&h, graph, 0, cudaGraphCondAssignDefault), "conditional handle")) return false;
        // set-up: sys = K x, r, pre, d, rz, max|r|, the loop condition
        cudaStream_t cap = nullptr;
        if (!ok(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking), "capture stream")) return false;
        bool good = ok(cudaStreamBeginCaptureToGraph(cap, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal), "capture");
        cudaGraphNode_t tail = nullptr;
        if (good) {
            if (sliced) {
                launch_product(x, kd, 1, h, false, cap);
            } else {
                admm_a_kernel<<<gm, kB, 0, cap>>>(s, x, st);
                admm_k_kernel<<<gn, kB, 0, cap>>>(s, x, kd, 1, rhs, r, pre, d, partial, st, h);
            }
            cudaStreamCaptureStatus cs;
            const cudaGraphNode_t* last = nullptr;
            size_t nlast = 0;
            good = ok(cudaStreamGetCaptureInfo(cap, &cs, nullptr, nullptr, &last, nullptr, &nlast), "capture info");
            if (good && nlast) tail = last[0];
            cudaGraph_t out = nullptr;
            good = ok(cudaStreamEndCapture(cap, &out), "end capture") && good && tail;
        }
        if (good) {
            cudaGraphNodeParams p = {cudaGraphNodeTypeConditional};
            p.conditional.handle = h;
            p.conditional.type = cudaGraphCondTypeWhile;
            p.conditional.size = 1;
            cudaGraphNode_t wnode;
            good = ok(cudaGraphAddNode(&wnode, graph, &tail, nullptr, 1, &p), "while node");
            if (good) {
                cudaGraph_t body = p.conditional.phGraph_out[0];
                good = ok(cudaStreamBeginCaptureToGraph(cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal), "capture");
                if (good) {
                    if (sliced) {
                        launch_product(d, kd, 2, h, false, cap);
                        launch(admm_update_slice_kernel, gv, true, cap, s.n, static_cast<const double*>(precond), x, r, pre,
                               static_cast<const double*>(d), static_cast<const double*>(kd), partial, st, h);
                        launch(admm_direction_slice_kernel, gv, true, cap, s.n, d, static_cast<const double*>(pre),
                               static_cast<const AdmmState*>(st));
                    } else {
                        admm_a_kernel<<<gm, kB, 0, cap>>>(s, d, st);
                        admm_k_kernel<<<gn, kB, 0, cap>>>(s, d, kd, 2, rhs, r, pre, d, partial, st, h);
                        admm_update_kernel<<<gv, kB, 0, cap>>>(s, x, r, pre, d, kd, partial, st, h);
                        admm_direction_kernel<<<gv, kB, 0, cap>>>(s.n, d, pre, st);
                    }
                    cudaGraph_t out = nullptr;
                    good = ok(cudaStreamEndCapture(cap, &out), "end capture");
                }
            }
        }
        if (good) good = ok(cudaGraphInstantiate(&exec, graph, 0), "graph instantiate");
        // K v alone
        if (good) good = ok(cudaGraphCreate(&apply_graph, 0), "graph");
        if (good) good = ok(cudaStreamBeginCaptureToGraph(cap, apply_graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal), "capture");
        if (good) {
            if (sliced) {
                launch_product(v, kd, 0, 0, false, cap);
            } else {
                admm_a_kernel<<<gm, kB, 0, cap>>>(s, v, st);
                admm_k_kernel<<<gn, kB, 0, cap>>>(s, v, kd, 0, rhs, r, pre, d, partial, st, 0);
            }
            cudaGraph_t out = nullptr;
            good = ok(cudaStreamEndCapture(cap, &out), "end capture");
        }
        if (good) good = ok(cudaGraphInstantiate(&apply_exec, apply_graph, 0), "graph instantiate");
        cudaStreamDestroy(cap);
        return good && ok(cudaGetLastError(), "admm kernels");
    }
    ~bqp_admm() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (apply_exec) cudaGraphExecDestroy(apply_exec);
        if (apply_graph) cudaGraphDestroy(apply_graph);
        for (void* p : {static_cast<void*>(hrp), static_cast<void*>(hci), static_cast<void*>(arp), static_cast<void*>(aci),
                        static_cast<void*>(trp), static_cast<void*>(tci), static_cast<void*>(hva), static_cast<void*>(ava),
                        static_cast<void*>(tva), static_cast<void*>(rho), static_cast<void*>(t), static_cast<void*>(precond),
                        static_cast<void*>(rhs), static_cast<void*>(x), static_cast<void*>(r), static_cast<void*>(pre),
                        static_cast<void*>(d), static_cast<void*>(kd), static_cast<void*>(v), static_cast<void*>(partial),
                        static_cast<void*>(st), static_cast<void*>(xa), static_cast<void*>(c), static_cast<void*>(z),
                        static_cast<void*>(y), static_cast<void*>(lo), static_cast<void*>(up), static_cast<void*>(k_len),
                        static_cast<void*>(k_row), static_cast<void*>(a_len), static_cast<void*>(a_row),
                        static_cast<void*>(k_base), static_cast<void*>(a_base), static_cast<void*>(k_col),
                        static_cast<void*>(a_col), static_cast<void*>(k_val), static_cast<void*>(a_val),
                        static_cast<void*>(stage)})
            if (p) cudaFree(p);
        if (h_st) cudaFreeHost(h_st);
        if (stream) cudaStreamDestroy(stream);
    }
};

// Brings the uploaded system (H, A, A' in CSR) into slice order and gives the CSR back.  Without memory
// for the second copy the system stays in CSR.
cudaError_t bqp_admm::slice(int64_t hz, int64_t az) {
    const size_t N = static_cast<size_t>(n), M = static_cast<size_t>(std::max<int64_t>(m, 1));
    t0 = (n + bqp::kSliceWindow - 1) / bqp::kSliceWindow * bqp::kSliceWindow;
    const size_t stacked = static_cast<size_t>(t0 + m), kz = static_cast<size_t>(hz + az), Z = static_cast<size_t>(az);
    int32_t *rp = nullptr, *ci = nullptr;  // the stacked rows in CSR
    double *va = nullptr, *x2 = nullptr, *d2 = nullptr, *v2 = nullptr;
    uint8_t* position_of = nullptr;
    struct Want {
        void** p;
        size_t bytes;
    };
    auto at = [](auto** p) { return reinterpret_cast<void**>(p); };
    const Want kept[] = {{at(&k_len), N}, {at(&k_row), N}, {at(&k_base), (N + 31) / 32 * 4}, {at(&k_col), kz * 4 + 16},
                         {at(&k_val), kz * 8 + 16}, {at(&a_len), M}, {at(&a_row), M}, {at(&a_base), (M + 31) / 32 * 4},
                         {at(&a_col), Z * 4 + 16}, {at(&a_val), Z * 8 + 16}, {at(&stage), std::max(N, M) * 8},
                         {at(&x2), stacked * 8}, {at(&d2), stacked * 8}, {at(&v2), stacked * 8}};
    const Want scratch[] = {{at(&rp), (N + 1) * 4}, {at(&ci), kz * 4 + 16}, {at(&va), kz * 8 + 16}, {at(&position_of), stacked}};
    auto release = [](const Want& w) {
        cudaFree(*w.p);
        *w.p = nullptr;
    };
    cudaError_t e = cudaSuccess;
    for (const Want& w : kept) if (!e) e = cudaMalloc(w.p, w.bytes);
    for (const Want& w : scratch) if (!e) e = cudaMalloc(w.p, w.bytes);
    if (!e) {
        admm_stack_kernel<<<kMaxBlocks, kB, 0, stream>>>(static_cast<int>(n), static_cast<int>(t0), hrp, hci, hva, trp, tci, tva,
                                                        rp, ci, va);
        bqp::InstDev k{}, a{};
        k.slice_len = k_len; k.slice_row = k_row; k.slice_base = k_base;
        a.slice_len = a_len; a.slice_row = a_row; a.slice_base = a_base;
        bqp::launch_slice_order(k, n, rp, position_of, stream);
        if (m) bqp::launch_slice_order(a, m, arp, position_of + t0, stream);
        bqp::launch_slice_columns(hz + az, t0 + m, ci, position_of, stream);
        bqp::launch_slice_entries(k, n, hz + az, rp, ci, va, k_col, k_val, stream);
        if (m) {
            // into a copy: without success the CSR stays in use
            cudaMemcpyAsync(ci, aci, Z * 4, cudaMemcpyDeviceToDevice, stream);
            bqp::launch_slice_columns(az, n, ci, position_of, stream);
            bqp::launch_slice_entries(a, m, az, arp, ci, ava, a_col, a_val, stream);
        }
        e = cudaGetLastError();
        const cudaError_t done = cudaStreamSynchronize(stream);
        if (!e) e = done;
    }
    for (const Want& w : scratch) release(w);
    if (e) {
        for (const Want& w : kept) release(w);
        if (e != cudaErrorMemoryAllocation) return e;
        cudaGetLastError();  // not sticky
        return cudaSuccess;
    }
    for (void* p : {static_cast<void*>(hrp), static_cast<void*>(hci), static_cast<void*>(hva), static_cast<void*>(trp),
                    static_cast<void*>(tci), static_cast<void*>(tva), static_cast<void*>(arp), static_cast<void*>(aci),
                    static_cast<void*>(ava), static_cast<void*>(t), static_cast<void*>(x), static_cast<void*>(d),
                    static_cast<void*>(v)})
        cudaFree(p);
    hrp = hci = trp = tci = arp = aci = nullptr;
    hva = tva = ava = t = nullptr;
    x = x2;
    d = d2;
    v = v2;
    sliced = true;
    return cudaSuccess;
}

namespace {
std::string g_admm_error;

bool valid_csr(int64_t rows, int64_t cols, int64_t nnz, const int32_t* rp, const int32_t* ci, const double* va) {
    if (rows < 0 || nnz < 0 || !rp || (nnz && (!ci || !va)) || rp[0] != 0 || rp[rows] != nnz) return false;
    for (int64_t i = 0; i < rows; ++i)
        if (rp[i + 1] < rp[i]) return false;
    for (int64_t k = 0; k < nnz; ++k)
        if (ci[k] < 0 || ci[k] >= cols || !std::isfinite(va[k])) return false;
    return true;
}
}  // namespace

extern "C" {

bqp_admm* bqp_admm_create(int device, int64_t n, int64_t m, const int32_t* h_rowptr, const int32_t* h_col,
                          const double* h_val, const int32_t* a_rowptr, const int32_t* a_col, const double* a_val) {
    if (n <= 0 || m < 0 || n > 2000000000LL || m > 2000000000LL || !h_rowptr || !a_rowptr) {
        g_admm_error = "Invalid ADMM system dimensions";
        return nullptr;
    }
    const int64_t hz = h_rowptr[n], az = a_rowptr[m];
    if (!valid_csr(n, n, hz, h_rowptr, h_col, h_val) || !valid_csr(m, n, az, a_rowptr, a_col, a_val)) {
        g_admm_error = "Invalid CSR arrays of H or A";
        return nullptr;
    }
    // A' by a stable counting sort: row j of A' lists the rows i of A in increasing order
    std::vector<int32_t> trp(static_cast<size_t>(n) + 1, 0), tci(static_cast<size_t>(az));
    std::vector<double> tva(static_cast<size_t>(az));
    for (int64_t k = 0; k < az; ++k) trp[static_cast<size_t>(a_col[k]) + 1]++;
    for (int64_t j = 0; j < n; ++j) trp[j + 1] += trp[j];
    {
        std::vector<int32_t> next(trp.begin(), trp.end() - 1);
        for (int64_t i = 0; i < m; ++i)
            for (int64_t k = a_rowptr[i]; k < a_rowptr[i + 1]; ++k) {
                const int32_t pos = next[a_col[k]]++;
                tci[pos] = static_cast<int32_t>(i);
                tva[pos] = a_val[k];
            }
    }
    std::unique_ptr<bqp_admm> s(new (std::nothrow) bqp_admm);
    if (!s) {
        g_admm_error = "host memory";
        return nullptr;
    }
    s->device = device;
    s->n = n;
    s->m = m;
    int prev = -1;
    cudaGetDevice(&prev);
    auto fail = [&](const char* what, cudaError_t e) {
        g_admm_error = std::string("CUDA: ") + what + ": " + cudaGetErrorString(e);
        if (prev >= 0) cudaSetDevice(prev);
        return static_cast<bqp_admm*>(nullptr);
    };
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return fail("set device", e);
    const size_t N = static_cast<size_t>(n), M = static_cast<size_t>(std::max<int64_t>(m, 1));
    auto alloc = [&](auto** p, size_t count) {
        return cudaMalloc(reinterpret_cast<void**>(p), sizeof(**p) * std::max<size_t>(count, 1));
    };
    if ((e = alloc(&s->hrp, N + 1)) || (e = alloc(&s->hci, static_cast<size_t>(hz))) || (e = alloc(&s->hva, static_cast<size_t>(hz))) ||
        (e = alloc(&s->arp, M + 1)) || (e = alloc(&s->aci, static_cast<size_t>(az))) || (e = alloc(&s->ava, static_cast<size_t>(az))) ||
        (e = alloc(&s->trp, N + 1)) || (e = alloc(&s->tci, static_cast<size_t>(az))) || (e = alloc(&s->tva, static_cast<size_t>(az))) ||
        (e = alloc(&s->rho, M)) || (e = alloc(&s->t, M)) || (e = alloc(&s->precond, N)) || (e = alloc(&s->rhs, N)) ||
        (e = alloc(&s->x, N)) || (e = alloc(&s->r, N)) || (e = alloc(&s->pre, N)) || (e = alloc(&s->d, N)) ||
        (e = alloc(&s->kd, N)) || (e = alloc(&s->v, N)) || (e = alloc(&s->partial, 3 * static_cast<size_t>(kMaxBlocks))) ||
        (e = alloc(&s->st, 1)))
        return fail("allocate", e);
    if ((e = cudaMallocHost(reinterpret_cast<void**>(&s->h_st), sizeof(AdmmState)))) return fail("allocate", e);
    if ((e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking))) return fail("stream", e);
    cudaMemcpy(s->hrp, h_rowptr, sizeof(int32_t) * (N + 1), cudaMemcpyHostToDevice);
    if (hz) cudaMemcpy(s->hci, h_col, sizeof(int32_t) * static_cast<size_t>(hz), cudaMemcpyHostToDevice);
    if (hz) cudaMemcpy(s->hva, h_val, sizeof(double) * static_cast<size_t>(hz), cudaMemcpyHostToDevice);
    cudaMemcpy(s->arp, a_rowptr, sizeof(int32_t) * (static_cast<size_t>(m) + 1), cudaMemcpyHostToDevice);
    if (az) cudaMemcpy(s->aci, a_col, sizeof(int32_t) * static_cast<size_t>(az), cudaMemcpyHostToDevice);
    if (az) cudaMemcpy(s->ava, a_val, sizeof(double) * static_cast<size_t>(az), cudaMemcpyHostToDevice);
    cudaMemcpy(s->trp, trp.data(), sizeof(int32_t) * (N + 1), cudaMemcpyHostToDevice);
    if (az) cudaMemcpy(s->tci, tci.data(), sizeof(int32_t) * static_cast<size_t>(az), cudaMemcpyHostToDevice);
    if (az) cudaMemcpy(s->tva, tva.data(), sizeof(double) * static_cast<size_t>(az), cudaMemcpyHostToDevice);
    cudaMemset(s->st, 0, sizeof(AdmmState));
    if ((e = cudaDeviceSynchronize())) return fail("upload", e);
    int64_t longest_k = 0, longest_a = 0;
    for (int64_t j = 0; j < n; ++j)
        longest_k = std::max<int64_t>(longest_k, static_cast<int64_t>(h_rowptr[j + 1]) - h_rowptr[j] + trp[j + 1] - trp[j]);
    for (int64_t i = 0; i < m; ++i) longest_a = std::max<int64_t>(longest_a, static_cast<int64_t>(a_rowptr[i + 1]) - a_rowptr[i]);
    const bool fits = hz + az <= 2000000000LL && n + m <= 2000000000LL;  // 32-bit entries and stacked columns
    if (fits && bqp::sliceable(n, hz + az, longest_k) && (m == 0 || bqp::sliceable(m, az, longest_a)))
        if ((e = s->slice(hz, az))) return fail("slice rows", e);
    if (prev >= 0) cudaSetDevice(prev);
    return s.release();
}

int bqp_admm_set_rho(bqp_admm* s, const double* rho, double sigma) {
    if (!s || (s->m && !rho) || !std::isfinite(sigma) || sigma < 0) return BQP_ERR_INVALID;
    for (int64_t i = 0; i < s->m; ++i)
        if (!(rho[i] > 0) || !std::isfinite(rho[i])) return BQP_ERR_INVALID;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(s->device);
    s->put(s->rho, rho, s->m, s->a_row);
    s->sigma = sigma;
    if (s->sliced) admm_precond_slice_kernel<<<bqp_admm::slice_grid(s->n), kB, 0, s->stream>>>(s->slices(), s->precond);
    else admm_precond_kernel<<<grid_for(static_cast<int>(s->n), kB), kB, 0, s->stream>>>(s->sys(), s->precond);
    bool good = s->ok(cudaStreamSynchronize(s->stream), "preconditioner") && s->build();
    s->rho_set = good;
    if (prev >= 0) cudaSetDevice(prev);
    if (!good) {
        g_admm_error = s->error;
        return BQP_ERR_CUDA;
    }
    return BQP_OK;
}

int bqp_admm_apply(bqp_admm* s, const double* v, double* out) {
    if (!s || !v || !out) return BQP_ERR_INVALID;
    if (!s->rho_set) return BQP_ERR_NOT_READY;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(s->device);
    const size_t N = static_cast<size_t>(s->n);
    s->put(s->v, v, s->n, s->k_row);
    cudaMemsetAsync(s->st, 0, sizeof(AdmmState), s->stream);
    cudaGraphLaunch(s->apply_exec, s->stream);
    s->get(out, s->kd, s->n, s->k_row);
    const bool good = s->ok(cudaStreamSynchronize(s->stream), "apply");
    if (prev >= 0) cudaSetDevice(prev);
    if (!good) {
        g_admm_error = s->error;
        return BQP_ERR_CUDA;
    }
    return BQP_OK;
}

int bqp_admm_solve(bqp_admm* s, const double* rhs, double* x, double accuracy, int64_t max_inner, int64_t* inner_out,
                   double* residual_out) {
    if (!s || !rhs || !x || !(accuracy >= 0) || max_inner < 0) return BQP_ERR_INVALID;
    if (!s->rho_set) return BQP_ERR_NOT_READY;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(s->device);
    const size_t N = static_cast<size_t>(s->n);
    std::memset(s->h_st, 0, sizeof(AdmmState));
    s->h_st->accuracy = accuracy;
    s->h_st->max_inner = max_inner;
    s->put(s->rhs, rhs, s->n, s->k_row);
    s->put(s->x, x, s->n, s->k_row);
    cudaMemcpyAsync(s->st, s->h_st, sizeof(AdmmState), cudaMemcpyHostToDevice, s->stream);
    cudaGraphLaunch(s->exec, s->stream);
    s->get(x, s->x, s->n, s->k_row);
    cudaMemcpyAsync(s->h_st, s->st, sizeof(AdmmState), cudaMemcpyDeviceToHost, s->stream);
    const bool good = s->ok(cudaStreamSynchronize(s->stream), "solve");
    if (prev >= 0) cudaSetDevice(prev);
    if (!good) {
        g_admm_error = s->error;
        return BQP_ERR_CUDA;
    }
    if (inner_out) *inner_out = s->h_st->inner;
    if (residual_out) std::memcpy(residual_out, &s->h_st->rmax, sizeof(double));
    return BQP_OK;
}

int bqp_admm_iterate(bqp_admm* s, const double* c, const double* lo, const double* up, double* x, double* z, double* y,
                     int64_t first_iteration, int64_t iterations, int64_t* inner_total) {
    if (!s || !c || !x || (s->m && (!lo || !up || !z || !y)) || first_iteration < 0 || iterations < 0)
        return BQP_ERR_INVALID;
    if (!s->rho_set) return BQP_ERR_NOT_READY;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(s->device);
    const size_t N = static_cast<size_t>(s->n), M = static_cast<size_t>(std::max<int64_t>(s->m, 1));
    cudaError_t e = cudaSuccess;
    if (!s->xa) {
        if ((e = cudaMalloc(&s->xa, sizeof(double) * N)) || (e = cudaMalloc(&s->c, sizeof(double) * N)) ||
            (e = cudaMalloc(&s->z, sizeof(double) * M)) || (e = cudaMalloc(&s->y, sizeof(double) * M)) ||
            (e = cudaMalloc(&s->lo, sizeof(double) * M)) || (e = cudaMalloc(&s->up, sizeof(double) * M))) {
            s->ok(e, "allocate ADMM state");
            if (prev >= 0) cudaSetDevice(prev);
            g_admm_error = s->error;
            return BQP_ERR_NO_MEMORY;
        }
    }
    s->put(s->xa, x, s->n, s->k_row);
    s->put(s->c, c, s->n, s->k_row);
    s->put(s->z, z, s->m, s->a_row);
    s->put(s->y, y, s->m, s->a_row);
    s->put(s->lo, lo, s->m, s->a_row);
    s->put(s->up, up, s->m, s->a_row);
    cudaMemsetAsync(s->st, 0, sizeof(AdmmState), s->stream);
    const Sys sy = s->sys();
    const int gn = grid_for(static_cast<int>(s->n), kRows), gm = grid_for(static_cast<int>(s->m), kRows);
    const int gv = grid_for(static_cast<int>(s->n), kB);
    for (int64_t k = 0; k < iterations; ++k) {
        const double it = static_cast<double>(first_iteration + k + 1);
        const double factor = std::min(1e-7, .05 / std::pow(it, 1.6));
        if (s->sliced) {
            const SliceSys S = s->slices();
            const int sn = bqp_admm::slice_grid(s->n), sm = bqp_admm::slice_grid(s->m);
            if (s->m) admm_yz_kernel<<<gv, kB, 0, s->stream>>>(S.a.n, s->rho, s->z, s->y, s->v + s->t0);
            admm_rhs_slice_kernel<<<sn, kB, 0, s->stream>>>(S, s->v, s->xa, s->c, s->rhs, s->x, s->partial, s->st, factor);
            cudaGraphLaunch(s->exec, s->stream);
            admm_zy_slice_kernel<<<sm, kB, 0, s->stream>>>(S, s->x, s->z, s->y, s->lo, s->up, s->st);
        } else {
            admm_rhs_kernel<<<gn, kB, 0, s->stream>>>(sy, s->z, s->y, s->xa, s->c, s->rhs, s->x, s->partial, s->st, factor);
            cudaGraphLaunch(s->exec, s->stream);
            admm_zy_kernel<<<gm, kB, 0, s->stream>>>(sy, s->x, s->z, s->y, s->lo, s->up, s->st);
        }
        admm_x_kernel<<<gv, kB, 0, s->stream>>>(static_cast<int>(s->n), s->x, s->xa);
    }
    s->get(x, s->xa, s->n, s->k_row);
    s->get(z, s->z, s->m, s->a_row);
    s->get(y, s->y, s->m, s->a_row);
    cudaMemcpyAsync(s->h_st, s->st, sizeof(AdmmState), cudaMemcpyDeviceToHost, s->stream);
    const bool good = s->ok(cudaStreamSynchronize(s->stream), "iterate") && s->ok(cudaGetLastError(), "ADMM kernels");
    if (prev >= 0) cudaSetDevice(prev);
    if (!good) {
        g_admm_error = s->error;
        return BQP_ERR_CUDA;
    }
    if (inner_total) *inner_total = s->h_st->inner_sum;
    return BQP_OK;
}

const char* bqp_admm_last_error(void) { return g_admm_error.c_str(); }

void bqp_admm_destroy(bqp_admm* s) {
    if (!s) return;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(s->device);
    delete s;
    if (prev >= 0) cudaSetDevice(prev);
}

}  // extern "C"
