// Device helpers shared by the factor and solve kernels: reciprocal, FP64 tensor-core product,
// children's vectors, programmatic dependent launches, asynchronous copies, prefix searches.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "plan.h"

namespace rfg {

// 1/p for a positive normal p: one step of Chebyshev's iteration (third order) for f(r) = 1/r − p from the
// hardware's approximate reciprocal r0, r0·(1 + e + e²) with e = 1 − p·r0, which leaves the relative error
// e³. rcp.approx.ftz.f64 reads 20 mantissa bits of p and gives 20 of r0 (its documentation), so
// |e| < 2^-19 and e³ < 2^-57, a sixteenth of the last place beside the half of the last fused multiply-add's
// rounding: at most 0.57 units in the last place of 1/p (0.508 in 8·10⁶ values, root mean square that of
// the correctly rounded quotient, 0.2887). Three dependent operations after r0, a fraction of the
// IEEE division's chain.
__device__ __forceinline__ double recip_chebyshev(double p) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(p));
    const double e = fma(-p, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// D = A·B + D on the FP64 tensor-core path for one 8×8×4 block (mma.sync m8n8k4 f64):
// lane l holds A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2·(l % 4) + {0, 1}].
__device__ __forceinline__ void dmma_884(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// x plus the children's update-vector entries of local row p of front f, right-hand side j,
// child 0 before child 1. imap holds, per front with children, the child row (or −1) of each of
// its rows for either child.
__device__ __forceinline__ double kids_add(double x, const double* V, const int32_t* __restrict__ imap,
                                           const DFront& f, int64_t p, int nrhs, int j) {
    if (f.imap_off < 0) return x;
    const int32_t i0 = imap[f.imap_off + p], i1 = imap[f.imap_off + f.m + p];
    if (i0 >= 0) x += __ldcg(V + (f.kv0 + i0) * nrhs + j);
    if (i1 >= 0) x += __ldcg(V + (f.kv1 + i1) * nrhs + j);
    return x;
}

// Programmatic dependent launch (PDL): a kernel launched with the programmatic
// stream-serialization attribute may start while its predecessor in the stream still
// runs. pdl_wait() blocks until the predecessor grid has completed and its memory is
// visible (it returns at once for a kernel launched without the attribute), so a kernel
// reads or writes nothing that its predecessors produce or consume before it;
// pdl_launch_dependents() lets the next kernel start once every CTA of this grid has
// issued it.
// A kernel that starts early shares its lifetime with the kernels that write its inputs. What an
// earlier kernel of the chain wrote therefore never comes in as `const T* __restrict__` and is never
// read by __ldg (either lets the compiler take the non-coherent path, which holds only for data that
// nobody writes while the kernel lives): such parameters carry no __restrict__, and values that are
// read once or staged in shared memory are read from L2 (__ldcg, cp.async.cg), whatever an SM's L1
// kept from a kernel before. const __restrict__ stays on what is constant for the whole chain: the
// plan's arrays and, in the sweeps, the factor.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// cp.async of 16 bytes global -> shared (cached in L2 only), src_bytes ∈ [0, 16] read and
// the rest of the 16 bytes zero-filled; both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// cp.async of the tile src[rr·ld + c] (rr < nr, c < ncol) into dst[rr·pitch + c] for
// rr < rows, c < cols, zero-filled outside (cols a multiple of 16 bytes, pitch·sizeof(T)
// a multiple of 16 bytes, src rows 16-byte aligned). Threads [0, nt) issue the copies.
template <typename T>
__device__ __forceinline__ void cp_async_tile(T* dst, int pitch, const T* src, int64_t ld, int nr, int ncol, int rows,
                                              int cols, int nt) {
    constexpr int VEC = 16 / (int)sizeof(T);
    const int per_row = cols / VEC;
    // (row, chunk) of this thread's first copy, then advanced by nt chunks without division
    int rr = (int)threadIdx.x / per_row, cc = (int)threadIdx.x - rr * per_row;
    const int dr = nt / per_row, dc = nt - dr * per_row;
    for (; rr < rows; rr += dr) {
        const int c = cc * VEC;
        int bytes = 0;
        const T* s = src;
        if (rr < nr && c < ncol) {
            bytes = min(VEC, ncol - c) * (int)sizeof(T);
            s = src + (int64_t)rr * ld + c;
        }
        cp_async16(dst + (int64_t)rr * pitch + c, s, bytes);
        cc += dc;
        if (cc >= per_row) {
            cc -= per_row;
            rr++;
        }
    }
}

// cp.async of n contiguous 16-byte chunks (both ends 16-byte aligned), threads [0, nt).
__device__ __forceinline__ void cp_async_flat(void* dst, const void* src, int n, int nt) {
    for (int i = threadIdx.x; i < n; i += nt)
        cp_async16(static_cast<char*>(dst) + 16 * (size_t)i, static_cast<const char*>(src) + 16 * (size_t)i, 16);
}
// Index i of the segment that holds item b: pre[i] <= b < pre[i+1], i in [0, n) (pre
// nondecreasing, pre[0] = 0, pre[n] > b). Warp-cooperative: every round the 32 lanes
// probe 32 evenly spaced entries and the ballot narrows the range 32-fold, so a launch
// over thousands of segments pays ~3 dependent loads per CTA instead of ~13. Must be
// called by all 32 lanes of a warp with the same b.
__device__ __forceinline__ int64_t find_slot_warp(const int64_t* __restrict__ pre, int64_t n, int64_t b) {
    const int lane = threadIdx.x & 31;
    int64_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const int64_t step = (hi - lo + 31) / 32;
        const int64_t idx = lo + lane * step;
        const bool ok = idx < hi && pre[idx] <= b;
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        const int k = 31 - __clz(m);  // lane 0 probes lo, where pre[lo] <= b
        lo += k * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// The tile of CTA b in a part of a step's outer update: pre (and pre_a of it, the tiles of the next
// outer block's columns, first in each front's list) are the prefix sums over the fronts. Part 0:
// all tiles, 1: those of pre_a, 2: the others. Returns the front's slot and its tile index in
// *tile. All 32 lanes of a warp with the same b.
__device__ __forceinline__ int64_t find_tile_warp(const int64_t* __restrict__ pre, const int64_t* __restrict__ pre_a,
                                                  int part, int64_t n, int64_t b, int64_t* tile) {
    if (part == 0) {
        const int64_t i = find_slot_warp(pre, n, b);
        *tile = b - pre[i];
        return i;
    }
    if (part == 1) {
        const int64_t i = find_slot_warp(pre_a, n, b);
        *tile = b - pre_a[i];
        return i;
    }
    const int lane = threadIdx.x & 31;
    int64_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const int64_t step = (hi - lo + 31) / 32;
        const int64_t idx = lo + lane * step;
        const bool ok = idx < hi && pre[idx] - pre_a[idx] <= b;
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        const int k = 31 - __clz(m);
        lo += k * step;
        hi = min(hi, lo + step);
    }
    *tile = b - (pre[lo] - pre_a[lo]) + (pre_a[lo + 1] - pre_a[lo]);
    return lo;
}

}  // namespace rfg
