// Device helpers of the kernels over sliced rows (engine.cuh: VAR_SLICE).
#pragma once
#include "engine.cuh"

namespace bqp {

// Programmatic dependent launch: the next launch of the stream may begin once every block has
// called let_next_launch_begin; wait_for_previous_launch returns once the launch before has ended
// and its writes are visible.  A kernel that reads what a launch before wrote waits in every
// block, the idle ones too, so that a launch that has ended implies that those before it have.
__device__ __forceinline__ void wait_for_previous_launch() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_launch_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Loads of a matrix that a launch reads once: no line of L1 for them, which the gathers of the vector
// then have to themselves (what bounds a random matrix is its gathers, a request and a 32-byte sector
// each: the L1s are 83 % busy with them): FP64 step of the random graph 1M 71.5 -> 70.9 us with it.
__device__ __forceinline__ int load_once(const int32_t* p) {
    int v;
    asm("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float load_once(const float* p) {
    float v;
    asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double load_once(const double* p) {
    double v;
    asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// One slice, one row per lane: the sum of the row's products in column order.  `len` is the lane's
// row length (descending over the lanes), `base` the slice's first entry.  At column j the rows
// still active are the first lanes, so the column's entries are base + the entries of the columns
// before it + lane: the lane's address advances by the count of active lanes.  AHEAD columns
// are loaded together (entries, then gathers) before the first product.
// EXACT: products and sums rounded separately from 0.0, the reference loop's arithmetic.
template <int AHEAD, class T = double>
struct SliceColumns {  // AHEAD columns of a slice: this lane's columns (-1: the row has ended) and values
    int c[AHEAD];
    T a[AHEAD];
    __device__ __forceinline__ void load(const int32_t* __restrict__ col, const T* __restrict__ val, int left, int& k) {
#pragma unroll
        for (int q = 0; q < AHEAD; ++q) {
            const bool in = q < left;
            c[q] = in ? load_once(col + k) : -1;
            a[q] = in ? load_once(val + k) : T(0);
            k += __popc(__ballot_sync(0xffffffffu, in));
        }
    }
    // adds the first `columns` (warp-uniform) of them; a column past the slice's longest row costs
    // no FP64 issue slot
    template <bool EXACT>
    __device__ __forceinline__ T add(const T* x, int columns, T acc) const {
        T xv[AHEAD];
#pragma unroll
        for (int q = 0; q < AHEAD; ++q) xv[q] = c[q] >= 0 ? x[c[q]] : T(0);
        return sum<EXACT, 0>(xv, columns, acc);
    }

private:
    template <bool EXACT, int Q>
    __device__ __forceinline__ T sum(const T* xv, int columns, T acc) const {
        if constexpr (Q < AHEAD) {
            if (Q >= columns) return acc;
            if constexpr (EXACT) {
                if (c[Q] >= 0) acc = __dadd_rn(acc, __dmul_rn(a[Q], xv[Q]));
            } else {
                if (c[Q] >= 0) acc = fma(a[Q], xv[Q], acc);
            }
            return sum<EXACT, Q + 1>(xv, columns, acc);
        } else {
            return acc;
        }
    }
};
template <bool EXACT, int AHEAD>
__device__ __forceinline__ double slice_dot(const int32_t* __restrict__ col, const double* __restrict__ val,
                                            const double* x, int base, int len) {
    const int longest = __shfl_sync(0xffffffffu, len, 0);
    int k = base + (threadIdx.x & 31);
    double acc = 0.0;
    SliceColumns<AHEAD> e;
    for (int j = 0; j < longest; j += AHEAD) {  // warp-uniform
        e.load(col, val, len - j, k);
        acc = e.template add<EXACT>(x, longest - j, acc);
    }
    return acc;
}

}  // namespace bqp
