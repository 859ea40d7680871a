// Solve chains (chain.h): the forward and backward sweeps of the levels with few fronts
// in one launch per level and direction.
//
// A level at the top of the tree has one to a few fronts of thousands of pivots. Stepped
// the usual way (solve.cu) each WS-wide block costs a launch for its diagonal block on one
// CTA and a launch for the rows below, and the GPU waits on the first. Here the level's
// work items are WS-wide diagonal blocks (and, forward, WS-row pieces of the later rows),
// each done by a cluster of four CTAs:
//   forward, block B of a front, CTA s owning the rows B·WS + 64s ... + 63:
//       x_s = X[rows] + (children's V) − Σ_{J < B} L[rows, J]·y_J   (tile J as soon as block
//             J's flag is up)
//       y of the block (below), then the block's flag is raised;
//   forward, later rows: V[rows] = (children's V) − Σ_J L[rows, J]·y_J over all blocks J;
//   backward, block B, CTA s owning the columns B·WS + 64s ... + 63:
//       z_s = Y[cols]/D − Σ_{r later} L[r, cols]·y_r − Σ_{J > B} L[J, cols]ᵀ·y_J,
//       y of the block.
// The tiles of a block stream through a ring of four cp.async stages while the CTA waits
// for the flags; the dependency chain from block to block is one flag wait, the last
// tile and the solve with the block's diagonal block, for which two ways stand:
//   FP32 factor: x_B (z_B) gathered from the cluster's CTAs (distributed shared memory) and one
//       product with the explicit WS × WS inverse of L_BB (k_chain_inverse);
//   FP64 factor: substitution over the CTAs in turn, forward y_s = inv(L_ss)·x_s with the
//       factorization's 64 × 64 inverse, y_s to the CTAs after s, x_t −= L_ts·y_s there (backward
//       the same from the last one, transposed). Three cluster barriers more in the chain from block to
//       block (a solve call of the 33³ cube 1.55 ms, 1.42 with the inverse), for the rounding of the
//       stepped sweeps: an FP64 solve is not refined unless the caller asks, and with the WS × WS
//       inverse its residuals were 1.02 to 1.10 times as large in the 2-norm and up to 1.5 times in the
//       maximum norm (means over right-hand sides; hex8 17³ to 45³, hex20 20³, one and six of them). Now
//       0.98 to 1.003 and 0.95 to 1.06 times.
//
// Items are taken in the plan's order from a counter, by the first CTA of a cluster when
// its previous item is done. Every item depends only on items before it in that order and
// an item is only taken by a running cluster, so the launch progresses with any number of
// resident clusters. Waits are bounded: a wait that gives up sets *err, the CTA goes on
// with the values it finds, every later wait of the launch returns at once, and the host
// reports the error (Engine::chain_check).
//
// One to four right-hand sides run on the CUDA cores. Five and more run the same chains in
// groups of eight right-hand sides (the _mm kernels): the eight columns are the N of the FP64
// tensor-core product, a group is a chain of its own with its own flags, and the later rows take
// all groups in one CTA so that L21 is read once.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "chain.h"
#include "engine.h"
#include "tiles.cuh"

namespace cg = cooperative_groups;

namespace rfg {
namespace {

constexpr int CT = 256;             // threads per CTA
constexpr int CQ = WS / 4;          // rows (forward) or columns (backward) of a block per CTA
constexpr int CL = WS / CQ;         // CTAs per cluster: one block
// The tiles of a block stream in pieces of 256-byte rows, so that the ring is the same size for
// an FP32 and an FP64 factor: forward 64 rows × FQC columns, backward BRC rows × 64 columns.
template <typename T>
constexpr int FQC = 256 / (int)sizeof(T);         // columns of a forward piece
template <typename T>
constexpr int FQP = FQC<T> + 64 / (int)sizeof(T); // its pitch: 16-byte row reads without conflicts
template <typename T>
constexpr int FPB = WS / FQC<T>;                  // forward pieces of a block
template <typename T>
constexpr int BRC = 256 / (int)sizeof(T);         // rows of a backward piece
template <typename T>
constexpr int BPB = WS / BRC<T>;                  // backward pieces of a block
constexpr int FLP = WS + 4;         // pitch (doubles) of the forward inverse rows
constexpr int BTP = CQ;             // pitch of a backward piece
constexpr long CHAIN_SPIN = 1L << 22;  // polls of a flag (about a second) before a wait gives up

static_assert(CL == 4 && CT == 4 * CQ, "four CTAs of 256 threads per block");
static_assert(CQ == CHAIN_PIECE, "the later-row pieces of the plan are one CTA's rows or columns");

constexpr size_t fwd_smem(int R) {
    return (size_t)CQ * FLP * 8 + (size_t)4 * CQ * FQP<float> * sizeof(float) + (size_t)2 * WS * R * 8;
}
constexpr size_t bwd_smem(int R) {
    return (size_t)WS * CQ * 8 + (size_t)4 * BRC<float> * BTP * sizeof(float) + (size_t)4 * CQ * R * 8 + (size_t)2 * WS * R * 8;
}
static_assert(FQP<float> * sizeof(float) == FQP<double> * sizeof(double) && BRC<float> * sizeof(float) == BRC<double> * sizeof(double),
              "the rings of both precisions have one size");
static_assert(fwd_smem(4) <= 232448 && bwd_smem(4) <= 232448, "shared memory of a CTA");

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ld_relaxed(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// One thread: waits until *flag >= target, at most CHAIN_SPIN polls.
__device__ void chain_wait(const int* flag, int target, int* err) {
    if (ld_acquire(flag) >= target) return;
    for (long it = 0; it < CHAIN_SPIN; it++) {
        if (ld_relaxed(err) != 0) return;
        __nanosleep(32);
        if (ld_acquire(flag) >= target) return;
    }
    atomicExch(err, 1);
}

// The CTA's writes before this call are visible to any thread that sees the flag count it.
__device__ __forceinline__ void chain_signal(int* flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(flag, 1);
    }
}

// cp.async of 8 bytes, global -> shared (the source written by an earlier launch)
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait_upto(int n) {
    if (n <= 0)
        cp_async_wait<0>();
    else if (n == 1)
        cp_async_wait<1>();
    else if (n == 2)
        cp_async_wait<2>();
    else
        cp_async_wait<3>();
}

// The cluster's next item: the first CTA takes it from the counter and writes it into the
// shared word of every CTA of the cluster.
__device__ __forceinline__ int64_t grab(cg::cluster_group& cluster, int64_t* s_item, int* counter) {
    if (cluster.block_rank() == 0 && threadIdx.x == 0) {
        const int64_t v = atomicAdd(counter, 1);
        for (int r = 0; r < CL; r++) *cluster.map_shared_rank(s_item, r) = v;
    }
    cluster.sync();
    return *s_item;
}

// Sum over the four lanes of a row (lanes 4i .. 4i+3); every lane gets the same value.
template <int R>
__device__ __forceinline__ void quad_sum(double (&a)[R]) {
#pragma unroll
    for (int r = 0; r < R; r++) {
        a[r] += __shfl_xor_sync(0xffffffffu, a[r], 1);
        a[r] += __shfl_xor_sync(0xffffffffu, a[r], 2);
    }
}

// a += b, b = 0. The products of each block of WS rows or columns are summed by themselves before they
// join the others: one running sum over thousands of terms rounds at the size of the whole sum each time
// (hex20 20³, six right-hand sides, FP64: residual 2-norms 1.04 times those of the stepped sweeps so,
// 1.00 now).
template <int R>
__device__ __forceinline__ void fold(double (&a)[R], double (&b)[R]) {
#pragma unroll
    for (int r = 0; r < R; r++) {
        a[r] += b[r];
        b[r] = 0.0;
    }
}
template <int N>
__device__ __forceinline__ void fold(double (&a)[N][2], double (&b)[N][2]) {
#pragma unroll
    for (int n = 0; n < N; n++) fold(a[n], b[n]);
}

// Forward tiles: acc (thread (i, q): row i, 16-byte groups q, q + 4, ... of each piece's row)
// += Σ_{Q < nq} L[r0 + i, piece Q]·y over the pieces of the blocks 0, 1, ...; piece Q in
// ring slot Q & 3, three pieces in flight. yload(j) fills yb with y_j (all threads,
// starting with a barrier that ends the previous block's use of yb).
template <typename T, int R, typename YLoad>
__device__ __forceinline__ void fwd_tiles(double (&acc)[R], T* ring, double* yb, const T* prow, int64_t ldp,
                                          int64_t k, int nr, int nq, YLoad&& yload) {
    constexpr int QC = FQC<T>, QP = FQP<T>, PB = FPB<T>, VEC = 16 / (int)sizeof(T);
    using VT = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
    const int tid = threadIdx.x, i = tid >> 2, q = tid & 3;
    auto issue = [&](int Q) {
        const int64_t c0 = (int64_t)Q * QC;
        const int ncol = (int)max((int64_t)0, min((int64_t)QC, k - c0));
        if (ncol > 0 && nr > 0) cp_async_tile<T>(ring + (Q & 3) * CQ * QP, QP, prow + c0, ldp, nr, ncol, CQ, QC, CT);
        cp_async_commit();
    };
    for (int Q = 0; Q < min(3, nq); Q++) issue(Q);
    double tot[R] = {};
    for (int Q = 0; Q < nq; Q++) {
        const int64_t j = Q / PB;
        const int qq = Q % PB;
        if (qq == 0) {
            fold(tot, acc);
            yload(j);
        }
        cp_wait_upto(min(2, nq - 1 - Q));
        __syncthreads();  // piece Q and y_j visible; every thread is done with piece Q − 1
        if (Q + 3 < nq) issue(Q + 3);
        if ((int64_t)Q * QC < k) {
            const T* Lt = ring + (Q & 3) * CQ * QP + i * QP;
            const double* yq = yb + qq * QC * R;
#pragma unroll
            for (int v = 0; v < QC / (4 * VEC); v++) {
                const int c = VEC * (q + 4 * v);
                const VT l4 = *reinterpret_cast<const VT*>(Lt + c);
                const T* l = reinterpret_cast<const T*>(&l4);
#pragma unroll
                for (int e = 0; e < VEC; e++)
#pragma unroll
                    for (int r = 0; r < R; r++) acc[r] = fma((double)l[e], yq[(c + e) * R + r], acc[r]);
            }
        }
    }
    fold(acc, tot);
}

// What CTA s of a forward block needs of the diagonal block, into Lv. FP32 factor: its rows of the
// WS × WS inverse. FP64: its rows of L left of the diagonal (from prow) and inv(L_ss) after them.
template <typename T>
__device__ __forceinline__ void load_fwd_block(double* Lv, const double* inv, const T* prow, const DFront& f, int64_t cb,
                                               int64_t b, int s, int nr) {
    if constexpr (sizeof(T) == 4) {
        const int cmax = CQ * (s + 1);  // inverse row 64s + i ends at the diagonal
        cp_async_tile<double>(Lv, FLP, inv + (cb * WS + s * CQ) * (int64_t)WS, WS, CQ, cmax, CQ, cmax, CT);
    } else {
        if (nr <= 0) return;
        if (s > 0) cp_async_tile<double>(Lv, FLP, prow, f.ldp, nr, CQ * s, CQ, CQ * s, CT);
        cp_async_tile<double>(Lv + CQ * s, FLP, inv + (f.blk_off + CL * b + s) * (int64_t)(NB * NB), NB, NB, NB, NB, NB, CT);
    }
}

// The same for the columns of a backward block, into Lc (rows of pitch P): FP32 its columns of the
// inverse from the diagonal on; FP64 inv(L_ss), then its columns of L below (from pcol, nrr rows).
template <typename T, int P>
__device__ __forceinline__ void load_bwd_block(double* Lc, const double* inv, const T* pcol, const DFront& f, int64_t cb,
                                               int64_t b, int s, int nc, int nrr) {
    if constexpr (sizeof(T) == 4) {
        const int ninv = WS - s * CQ;  // inverse column 64s + c starts at its diagonal row
        cp_async_tile<double>(Lc, P, inv + (cb * WS + s * CQ) * (int64_t)WS + s * CQ, WS, ninv, CQ, ninv, CQ, CT);
    } else {
        if (nc <= 0) return;
        cp_async_tile<double>(Lc, P, inv + (f.blk_off + CL * b + s) * (int64_t)(NB * NB), NB, NB, NB, NB, NB, CT);
        if (nrr > 0) cp_async_tile<double>(Lc + CQ * P, P, pcol, f.ldp, nrr, nc, WS - CQ * (s + 1), CQ, CT);
    }
}

template <typename T, int R>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CT, 1)
    k_chain_fwd(const double* X, double* __restrict__ Y, const T* __restrict__ panel,
                const double* V, const int32_t* __restrict__ imap,
                const double* __restrict__ inv, const DFront* __restrict__ fr, const int64_t* __restrict__ chain_blk,
                const int64_t* __restrict__ items, int64_t nitems, int* __restrict__ flags, int* __restrict__ counter,
                int* __restrict__ err) {
    pdl_launch_dependents();
    pdl_wait();
    cg::cluster_group cluster = cg::this_cluster();
    const int s = (int)cluster.block_rank();
    extern __shared__ __align__(16) double sm[];
    double* Lv = sm;                                                   // [CQ][FLP]: inverse rows 64s .., or L_st and inv(L_ss)
    T* ring = reinterpret_cast<T*>(sm + CQ * FLP);                     // [4][CQ][FQP]: tile pieces
    double* yb = reinterpret_cast<double*>(ring + 4 * CQ * FQP<T>);    // [WS][R]: y_J, then x_B
    double* xo = yb + WS * R;                                          // [CQ][R]: this CTA's rows of x_B
    double* yr = xo + CQ * R;                                          // [WS - CQ][R]: y_t of the cluster's other CTAs
    __shared__ int64_t s_item;
    const int tid = threadIdx.x, i = tid >> 2, q = tid & 3;
    for (;;) {
        const int64_t it = grab(cluster, &s_item, counter);
        if (it >= nitems) break;
        const int64_t t = items[2 * it], b = items[2 * it + 1];
        const DFront f = fr[t];
        const int64_t cb0 = chain_blk[t];
        const int64_t r0 = b * WS + s * CQ;
        const int nr = (int)max((int64_t)0, min((int64_t)CQ, f.k - r0));
        load_fwd_block<T>(Lv, inv, panel + f.poff + r0 * f.ldp + b * WS, f, cb0 + b, b, s, nr);
        cp_async_commit();
        double acc[R];
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = 0.0;
        fwd_tiles<T, R>(acc, ring, yb, panel + f.poff + r0 * f.ldp, f.ldp, f.k, nr, FPB<T> * (int)b, [&](int64_t j) {
            if (tid == 0) chain_wait(&flags[cb0 + j], CL, err);
            __syncthreads();
            const int wbj = (int)min((int64_t)WS, f.k - j * WS);
            const double* ys = Y + (f.start + j * WS) * R;
            for (int e = tid; e < WS * R; e += CT) yb[e] = e < wbj * R ? __ldcg(ys + e) : 0.0;
        });
        quad_sum<R>(acc);
        if (q == 0) {
#pragma unroll
            for (int r = 0; r < R; r++)
                xo[i * R + r] =
                    i < nr ? kids_add(__ldcg(X + (f.start + r0 + i) * R + r), V, imap, f, r0 + i, R, r) - acc[r] : 0.0;
        }
        // a = Σ_c Lv[i, c0 + c]·v[c] over n columns, a multiple of CQ
        auto row_product = [&](double (&a)[R], int c0, int n, const double* v) {
            double a2[R] = {};
#pragma unroll
            for (int r = 0; r < R; r++) a[r] = 0.0;
            for (int cb = 0; cb < n; cb += CQ) {
#pragma unroll
                for (int u = 0; u < CQ / 4; u += 2) {
                    const int c = cb + q + 4 * u;
                    const double l0 = Lv[i * FLP + c0 + c], l1 = Lv[i * FLP + c0 + c + 4];
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        a[r] = fma(l0, v[c * R + r], a[r]);
                        a2[r] = fma(l1, v[(c + 4) * R + r], a2[r]);
                    }
                }
            }
            fold(a, a2);
            quad_sum<R>(a);
        };
        auto put_y = [&](const double (&a)[R]) {
            if (q == 0 && i < nr) {
#pragma unroll
                for (int r = 0; r < R; r++) Y[(f.start + r0 + i) * R + r] = a[r];
            }
        };
        double a[R];
        if constexpr (sizeof(T) == 4) {
            cluster.sync();
            for (int e = tid; e < WS * R; e += CT) {
                const int rk = e / (CQ * R);
                yb[e] = cluster.map_shared_rank(xo, rk)[e - rk * CQ * R];
            }
            cp_async_wait<0>();
            __syncthreads();
            row_product(a, 0, CQ * (s + 1), yb);  // inverse row 64s + i ends at the diagonal
            put_y(a);
        } else {
            cp_async_wait<0>();
            __syncthreads();
            const int nsub = (int)min((int64_t)CL, (f.k - b * WS + CQ - 1) / CQ);
            for (int t = 0; t < nsub; t++) {
                if (s == t) {
                    row_product(a, CQ * t, CQ, xo);
                    if (q > t) {  // the lanes of a row take a rank each
                        double* o = cluster.map_shared_rank(yr, q) + (CQ * t + i) * R;
#pragma unroll
                        for (int r = 0; r < R; r++) o[r] = a[r];
                    }
                }
                // Y after the barrier: its release would wait for stores to global memory too
                if (t + 1 < nsub) cluster.sync();
                if (s == t) put_y(a);
                if (t + 1 == nsub) break;
                if (s > t && s < nsub) {
                    row_product(a, CQ * t, CQ, yr + CQ * t * R);
                    if (q == 0) {
#pragma unroll
                        for (int r = 0; r < R; r++) xo[i * R + r] -= a[r];
                    }
                    __syncthreads();
                }
            }
        }
        chain_signal(&flags[cb0 + b]);
        cluster.sync();  // the cluster's x_B pieces may be overwritten after this
    }
}

// The later rows of a chain level's fronts after the level's chain: V[rows] = (children's V) −
// L21·y over all the front's pivots, one CTA per CHAIN_PIECE rows.
template <typename T, int R>
__global__ void __launch_bounds__(CT) k_chain_rows(const double* Y, double* __restrict__ V,
                                                   const int32_t* __restrict__ imap, const T* __restrict__ panel,
                                                   const DFront* __restrict__ fr, const int64_t* __restrict__ items) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) double sm[];
    T* ring = reinterpret_cast<T*>(sm);                              // [4][CQ][FQP]
    double* yb = reinterpret_cast<double*>(ring + 4 * CQ * FQP<T>);  // [WS][R]
    const int tid = threadIdx.x, i = tid >> 2, q = tid & 3;
    const int64_t t = items[2 * blockIdx.x], c = items[2 * blockIdx.x + 1];
    const DFront f = fr[t];
    const int64_t r0 = f.k + c * CQ;
    const int nr = (int)min((int64_t)CQ, f.m - r0);
    double acc[R];
#pragma unroll
    for (int r = 0; r < R; r++) acc[r] = 0.0;
    fwd_tiles<T, R>(acc, ring, yb, panel + f.poff + r0 * f.ldp, f.ldp, f.k, nr, FPB<T> * (int)((f.k + WS - 1) / WS),
                    [&](int64_t j) {
                        __syncthreads();
                        const int wbj = (int)min((int64_t)WS, f.k - j * WS);
                        const double* ys = Y + (f.start + j * WS) * R;
                        for (int e = tid; e < WS * R; e += CT) yb[e] = e < wbj * R ? __ldcg(ys + e) : 0.0;
                    });
    quad_sum<R>(acc);
    if (q == 0 && i < nr) {
        double* vt = V + (f.vuoff + c * CQ + i) * R;
#pragma unroll
        for (int r = 0; r < R; r++) vt[r] = kids_add(0.0, V, imap, f, r0 + i, R, r) - acc[r];
    }
}

// Backward chunks: acc (thread (c, g): column c, rows g, g + 4, ... of each BRC-row chunk)
// += Σ_{h < nh} L[rows of chunk h, col0 + c]·y(rows); chunk h in ring slot h & 3, three in
// flight. rows_of(h, ra) gives the chunk's first row and row count; yload(h) runs before
// chunk h (all threads) and returns where the chunk's y values are in shared memory;
// issue_y(h) queues the chunk's y values with its tile (cp.async) when it can.
template <typename T, int R, typename Rows, typename YLoad, typename IssueY>
__device__ __forceinline__ void bwd_tiles(double (&acc)[R], T* ring, const T* pcol, int64_t ldp, int nc, int nh,
                                          Rows&& rows_of, YLoad&& yload, IssueY&& issue_y) {
    const int tid = threadIdx.x, c = tid & (CQ - 1), g = tid >> 6;
    auto issue = [&](int h) {
        int64_t ra;
        const int nrr = rows_of(h, ra);
        if (nrr > 0 && nc > 0)
            cp_async_tile<T>(ring + (h & 3) * BRC<T> * BTP, BTP, pcol + ra * ldp, ldp, nrr, nc, BRC<T>, CQ, CT);
        issue_y(h, ra, nrr);
        cp_async_commit();
    };
    for (int h = 0; h < min(3, nh); h++) issue(h);
    double tot[R] = {};
    for (int h = 0; h < nh; h++) {
        int64_t ra;
        const int nrr = rows_of(h, ra);
        if (h % BPB<T> == 0) fold(tot, acc);
        const double* yv = yload(h);
        cp_wait_upto(min(2, nh - 1 - h));
        __syncthreads();  // chunk h visible; every thread is done with chunk h − 1
        if (h + 3 < nh) issue(h + 3);
        if (nrr > 0) {
            const T* Lt = ring + (h & 3) * BRC<T> * BTP + c;
#pragma unroll 4
            for (int u = 0; u < BRC<T> / 4; u++) {
                const int rr = g + 4 * u;
                const double l = Lt[rr * BTP];
#pragma unroll
                for (int r = 0; r < R; r++) acc[r] = fma(l, yv[rr * R + r], acc[r]);
            }
        }
    }
    fold(acc, tot);
}

// Σ over the four row groups of a column, in group order (threads tid < CQ get the total
// of column tid); red [4][CQ][R] in shared memory.
template <int R>
__device__ __forceinline__ void col_sum(double (&acc)[R], double* red) {
    const int tid = threadIdx.x, c = tid & (CQ - 1), g = tid >> 6;
#pragma unroll
    for (int r = 0; r < R; r++) red[(g * CQ + c) * R + r] = acc[r];
    __syncthreads();
    if (tid < CQ) {
#pragma unroll
        for (int r = 0; r < R; r++)
            acc[r] = ((red[c * R + r] + red[(CQ + c) * R + r]) + red[(2 * CQ + c) * R + r]) + red[(3 * CQ + c) * R + r];
    }
}

// z of pivot column col of a front before the chain's own products: the forward result over D
// minus the later rows' part (the row groups of k_chain_cols in order; cb < 0: no later rows).
__device__ __forceinline__ double chain_z(const double* Y, const double* d, const double* part, int64_t cb,
                                          const DFront& f, int64_t col, int nrhs, int r) {
    double z = __ldcg(Y + (f.start + col) * nrhs + r) / d[f.start + col];
    if (cb >= 0) {
        const double* p = part + ((cb + col / CQ) * CHAIN_GROUPS * CQ + col % CQ) * (int64_t)nrhs + r;
        double sum = 0.0;
#pragma unroll
        for (int g = 0; g < CHAIN_GROUPS; g++) sum += __ldcg(p + (int64_t)g * CQ * nrhs);
        z -= sum;
    }
    return z;
}

template <typename T, int R>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CT, 1)
    k_chain_bwd(double* __restrict__ Y, const T* __restrict__ panel, const double* __restrict__ inv,
                const double* __restrict__ d, const double* part, const int64_t* __restrict__ colbase,
                const DFront* __restrict__ fr, const int64_t* __restrict__ chain_blk, const int64_t* __restrict__ items,
                int64_t nitems, int* __restrict__ flags, int* __restrict__ counter, int* __restrict__ err) {
    pdl_launch_dependents();
    pdl_wait();
    cg::cluster_group cluster = cg::this_cluster();
    const int s = (int)cluster.block_rank();
    extern __shared__ __align__(16) double sm[];
    double* Lc = sm;                                               // [WS][CQ]: rows 64s .. of inverse columns 64s .., or inv(L_ss) and L_ts
    T* ring = reinterpret_cast<T*>(sm + WS * CQ);                  // [4][BRC][BTP]: tile chunks
    double* yp = reinterpret_cast<double*>(ring + 4 * BRC<T> * BTP);  // [WS][R]: y of a later block; then z_B
    double* red = yp + WS * R;                                     // [4][CQ][R]
    double* zo = red + 4 * CQ * R;                                 // [CQ][R]: this CTA's columns of z_B
    double* yr = zo + CQ * R;                                      // [WS - CQ][R]: y_t of the cluster's other CTAs
    __shared__ int64_t s_item;
    const int tid = threadIdx.x, c = tid & (CQ - 1), g = tid >> 6;
    for (;;) {
        const int64_t it = grab(cluster, &s_item, counter);
        if (it >= nitems) break;
        const int64_t t = items[2 * it], b = items[2 * it + 1];
        const DFront f = fr[t];
        const int64_t cb0 = chain_blk[t];
        const int64_t col0 = b * WS + s * CQ;
        const int nc = (int)max((int64_t)0, min((int64_t)CQ, f.k - col0));
        const int64_t nb = (f.k + WS - 1) / WS;
        const int wb = (int)min((int64_t)WS, f.k - b * WS);
        load_bwd_block<T, CQ>(Lc, inv, panel + f.poff + (b * WS + CQ * (s + 1)) * f.ldp + col0, f, cb0 + b, b, s, nc,
                              wb - CQ * (s + 1));
        cp_async_commit();
        double acc[R];
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = 0.0;
        // the chunks of blocks nb − 1, ..., b + 1, BPB per block
        bwd_tiles<T, R>(
            acc, ring, panel + f.poff + col0, f.ldp, nc, BPB<T> * (int)(nb - 1 - b),
            [&](int h, int64_t& ra) -> int {
                ra = (nb - 1 - h / BPB<T>) * WS + (h % BPB<T>) * BRC<T>;
                return (int)max((int64_t)0, min((int64_t)BRC<T>, f.k - ra));
            },
            [&](int h) -> const double* {
                if (h % BPB<T> == 0) {
                    const int64_t bb = nb - 1 - h / BPB<T>;
                    if (tid == 0) chain_wait(&flags[cb0 + bb], CL, err);
                    __syncthreads();
                    const int wbb = (int)min((int64_t)WS, f.k - bb * WS);
                    const double* src = Y + (f.start + bb * WS) * R;
                    for (int e = tid; e < WS * R; e += CT) yp[e] = e < wbb * R ? __ldcg(src + e) : 0.0;
                }
                return yp + (h % BPB<T>) * BRC<T> * R;
            },
            [](int, int64_t, int) {});
        col_sum<R>(acc, red);
        if (tid < CQ) {
#pragma unroll
            for (int r = 0; r < R; r++)
                zo[c * R + r] = c < nc ? chain_z(Y, d, part, colbase[t], f, col0 + c, R, r) - acc[r] : 0.0;
        }
        // threads tid < CQ: a = Σ_rr Lc[r0 + rr, c]·v[rr] over n rows, a multiple of CQ
        auto col_product = [&](double (&a)[R], int r0, int n, const double* v) {
            double a2[R] = {};
#pragma unroll
            for (int r = 0; r < R; r++) a[r] = 0.0;
            for (int rb = 0; rb < n; rb += CQ) {
#pragma unroll
                for (int u = 0; u < CQ / 4; u += 2) {
                    const int rr = rb + g + 4 * u;
                    const double l0 = Lc[(r0 + rr) * CQ + c], l1 = Lc[(r0 + rr + 4) * CQ + c];
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        a[r] = fma(l0, v[rr * R + r], a[r]);
                        a2[r] = fma(l1, v[(rr + 4) * R + r], a2[r]);
                    }
                }
            }
            fold(a, a2);
            col_sum<R>(a, red);
        };
        auto put_y = [&](const double (&a)[R]) {
            if (tid < nc) {
#pragma unroll
                for (int r = 0; r < R; r++) Y[(f.start + col0 + c) * R + r] = a[r];
            }
        };
        double a[R];
        if constexpr (sizeof(T) == 4) {
            cluster.sync();
            double* zf = yp;
            for (int e = tid; e < WS * R; e += CT) {
                const int rk = e / (CQ * R);
                zf[e] = cluster.map_shared_rank(zo, rk)[e - rk * CQ * R];
            }
            cp_async_wait<0>();
            __syncthreads();
            col_product(a, 0, WS - s * CQ, zf + s * CQ * R);
            put_y(a);
        } else {
            cp_async_wait<0>();
            __syncthreads();
            for (int t = (wb + CQ - 1) / CQ - 1; t >= 0; t--) {
                if (s == t) {
                    col_product(a, 0, CQ, zo);
                    if (tid < CQ) {
                        for (int rk = 0; rk < t; rk++) {
                            double* o = cluster.map_shared_rank(yr, rk) + (CQ * (t - 1) + c) * R;
#pragma unroll
                            for (int r = 0; r < R; r++) o[r] = a[r];
                        }
                    }
                }
                if (t > 0) cluster.sync();
                if (s == t) put_y(a);
                if (t == 0) break;
                if (s < t) {
                    col_product(a, CQ * (t - s), CQ, yr + CQ * (t - 1) * R);
                    if (tid < CQ) {
#pragma unroll
                        for (int r = 0; r < R; r++) zo[c * R + r] -= a[r];
                    }
                    __syncthreads();
                }
            }
        }
        chain_signal(&flags[cb0 + b]);
        cluster.sync();  // the cluster's z_B pieces may be overwritten after this
    }
}

// y of the later rows of a chain level's fronts into V (contiguous per front), before the
// level's backward: V[vuoff + i] = Y[rows[rows_off + i]], one CTA per CHAIN_PIECE rows.
__global__ void __launch_bounds__(CT) k_chain_gather(const double* Y, double* __restrict__ V,
                                                     const DFront* __restrict__ fr, const int64_t* __restrict__ rows,
                                                     const int64_t* __restrict__ items, int nrhs) {
    pdl_launch_dependents();
    const int64_t t = items[2 * blockIdx.x], c = items[2 * blockIdx.x + 1];
    const DFront f = fr[t];
    const int64_t i0 = c * CQ;
    pdl_wait();
    const int nr = (int)min((int64_t)CQ, f.u - i0);
    for (int e = threadIdx.x; e < nr * nrhs; e += CT) {
        const int ii = e / nrhs, r = e - ii * nrhs;
        V[(f.vuoff + i0 + ii) * nrhs + r] = __ldcg(Y + rows[f.rows_off + i0 + ii] * nrhs + r);
    }
}

// The later rows' part of a chain level's backward, before its chain: the partial sums
// L21ᵀ·y of the front's later rows (their y in V, from k_chain_gather), one CTA per
// CHAIN_PIECE pivot columns and group of rows (blockIdx.y of CHAIN_GROUPS), into
// part[(item · CHAIN_GROUPS + group) · CHAIN_PIECE + column]; the chain subtracts them in
// group order (chain_z).
template <typename T, int R>
__global__ void __launch_bounds__(CT) k_chain_cols(double* __restrict__ part, const double* V,
                                                   const T* __restrict__ panel, const DFront* __restrict__ fr,
                                                   const int64_t* __restrict__ items) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) double sm[];
    constexpr int RC = BRC<T>;
    T* ring = reinterpret_cast<T*>(sm);                           // [4][RC][BTP]
    double* ys = reinterpret_cast<double*>(ring + 4 * RC * BTP);  // [4][RC][R]: y of a chunk, by slot
    double* red = ys + 4 * RC * R;                                // [4][CQ][R]
    const int tid = threadIdx.x, c = tid & (CQ - 1);
    const int64_t t = items[2 * blockIdx.x], cc = items[2 * blockIdx.x + 1];
    const DFront f = fr[t];
    const int64_t col0 = cc * CQ;
    const int nc = (int)min((int64_t)CQ, f.k - col0);
    const int nchunk = (int)((f.u + RC - 1) / RC), g = blockIdx.y;
    const int h0 = nchunk * g / CHAIN_GROUPS, h1 = nchunk * (g + 1) / CHAIN_GROUPS;
    double acc[R];
#pragma unroll
    for (int r = 0; r < R; r++) acc[r] = 0.0;
    bwd_tiles<T, R>(
        acc, ring, panel + f.poff + col0, f.ldp, nc, h1 - h0,
        [&](int h, int64_t& ra) -> int {
            ra = f.k + (int64_t)(h0 + h) * RC;
            return (int)min((int64_t)RC, f.m - ra);
        },
        [&](int h) -> const double* { return ys + (h & 3) * RC * R; },
        [&](int h, int64_t ra, int nrr) {
            if (tid < RC * R) {
                const int rr = tid / R, r = tid - rr * R;
                double* dst = ys + ((h & 3) * RC + rr) * R + r;
                if (rr < nrr)
                    cp_async8(dst, V + (f.vuoff + ra - f.k + rr) * R + r);
                else
                    *dst = 0.0;
            }
        });
    col_sum<R>(acc, red);
    if (tid < CQ) {
        double* out = part + (((int64_t)blockIdx.x * CHAIN_GROUPS + g) * CQ + c) * R;
#pragma unroll
        for (int r = 0; r < R; r++) out[r] = acc[r];
    }
}

// ---------------------------------------------------------------------------
// Five to 32 right-hand sides: groups of eight (MG) on the FP64 tensor-core path (m8n8k4).
// Warp w owns rows (forward) or columns (backward) 8w ... of the CTA's 64. The vectors of a
// group are rows of eight doubles with the halves swapped on every second pair of rows (vsw),
// so that a fragment load (four rows, eight columns) meets every bank once per half-warp.
// Before, the wide steps ran one by one with the products on the CUDA cores and eight
// right-hand sides per CTA of the diagonal kernels: 47.3 ms per refined solve of the hex20 20³
// cube with 32 right-hand sides (four sweeps), now 11.7 ms.
// ---------------------------------------------------------------------------
constexpr int MG = 8;
template <typename T>
constexpr int MFP = FQC<T> + 4;                    // pitch of a forward piece: conflict-free row fragments
template <typename T>
constexpr int MBP = CQ + (sizeof(T) == 4 ? 8 : 4); // pitch of a backward piece: conflict-free column fragments
constexpr int MLP = CQ + 4;                        // pitch of the backward inverse columns
template <typename T>
constexpr size_t mm_fwd_smem = (size_t)CQ * FLP * 8 + (size_t)4 * CQ * MFP<T> * sizeof(T) + (size_t)WS * MG * 8;
template <typename T>
constexpr size_t mm_bwd_smem = (size_t)WS * MLP * 8 + (size_t)4 * BRC<T> * MBP<T> * sizeof(T) + (size_t)WS * MG * 8;
static_assert(mm_fwd_smem<float> <= 232000 && mm_fwd_smem<double> <= 232000 && mm_bwd_smem<float> <= 232000 &&
                  mm_bwd_smem<double> <= 232000,
              "shared memory of a CTA");

__device__ __forceinline__ int vsw(int k, int n) { return k * MG + (n ^ ((k & 2) << 1)); }

template <typename T>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CT, 1)
    k_chain_fwd_mm(const double* X, double* __restrict__ Y, const T* __restrict__ panel,
                   const double* V, const int32_t* __restrict__ imap, const double* __restrict__ inv,
                   const DFront* __restrict__ fr, const int64_t* __restrict__ chain_blk,
                   const int64_t* __restrict__ items, int64_t nitems, int nrhs, int64_t nblocks,
                   int* __restrict__ flags0, int* __restrict__ counter, int* __restrict__ err) {
    pdl_launch_dependents();
    pdl_wait();
    cg::cluster_group cluster = cg::this_cluster();
    const int s = (int)cluster.block_rank(), ngrp = (nrhs + MG - 1) / MG;
    extern __shared__ __align__(16) double sm[];
    constexpr int QC = FQC<T>, QP = MFP<T>, PB = FPB<T>;
    double* Lv = sm;                                             // [CQ][FLP]: inverse rows 64s ..
    T* ring = reinterpret_cast<T*>(sm + CQ * FLP);               // [4][CQ][QP]
    double* yb = reinterpret_cast<double*>(ring + 4 * CQ * QP);  // [WS][MG]: y_J, then x_B
    double* xo = reinterpret_cast<double*>(ring);                // [CQ][MG]: this CTA's rows of x_B (ring idle)
    __shared__ int64_t s_item;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    for (;;) {
        const int64_t it = grab(cluster, &s_item, counter);
        if (it >= nitems * ngrp) break;
        const int64_t item = it / ngrp;
        const int jg = (int)(it - item * ngrp), j0 = jg * MG, rc = min(MG, nrhs - j0);
        const int64_t t = items[2 * item], b = items[2 * item + 1];
        const DFront f = fr[t];
        int* flags = flags0 + jg * nblocks + chain_blk[t];
        const int64_t r0 = b * WS + s * CQ;
        const int nr = (int)max((int64_t)0, min((int64_t)CQ, f.k - r0));
        load_fwd_block<T>(Lv, inv, panel + f.poff + r0 * f.ldp + b * WS, f, chain_blk[t] + b, b, s, nr);
        cp_async_commit();
        const T* prow = panel + f.poff + r0 * f.ldp;
        const int nq = PB * (int)b;
        auto issue = [&](int Q) {
            if (nr > 0) cp_async_tile<T>(ring + (Q & 3) * CQ * QP, QP, prow + (int64_t)Q * QC, f.ldp, nr, QC, CQ, QC, CT);
            cp_async_commit();
        };
        double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0}, tot[2] = {0.0, 0.0};
        for (int Q = 0; Q < min(3, nq); Q++) issue(Q);
        for (int Q = 0; Q < nq; Q++) {
            if (Q % PB == 0) {
                fold(a0, a1);
                fold(tot, a0);
                const int64_t j = Q / PB;
                if (tid == 0) chain_wait(&flags[j], CL, err);
                __syncthreads();
                const double* ys = Y + (f.start + j * WS) * nrhs + j0;
                for (int e = tid; e < WS * MG; e += CT) {
                    const int k = e / MG, n = e % MG;
                    yb[vsw(k, n)] = n < rc ? __ldcg(ys + (int64_t)k * nrhs + n) : 0.0;
                }
            }
            cp_wait_upto(min(2, nq - 1 - Q));
            __syncthreads();  // piece Q and y_j visible; every thread is done with piece Q − 1
            if (Q + 3 < nq) issue(Q + 3);
            if (nr > 8 * w) {
                const T* Lt = ring + (Q & 3) * CQ * QP + (8 * w + g) * QP + q;
                const int kb = (Q % PB) * QC + q;
#pragma unroll
                for (int k = 0; k < QC; k += 8) {
                    dmma_884(a0[0], a0[1], (double)Lt[k], yb[vsw(kb + k, g)]);
                    dmma_884(a1[0], a1[1], (double)Lt[k + 4], yb[vsw(kb + k + 4, g)]);
                }
            }
        }
        double x[2];  // row 8w + g of x_s, right-hand sides 2q, 2q + 1
        const int i = 8 * w + g;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int n = 2 * q + e;
            x[e] = 0.0;
            if (i < nr && n < rc)
                x[e] = kids_add(__ldcg(X + (f.start + r0 + i) * nrhs + j0 + n), V, imap, f, r0 + i, nrhs, j0 + n) - (tot[e] + (a0[e] + a1[e]));
        }
        // y = Σ_k Lv[i, k0 + k]·yb[k0 + k] over n columns
        double y[2];
        auto row_product = [&](int k0, int n) {
            double acc[2][2] = {};
            const double* Lr = Lv + (8 * w + g) * FLP + q + k0;
            for (int k = 0; k < n; k += 8) {
                dmma_884(acc[0][0], acc[0][1], Lr[k], yb[vsw(k0 + k + q, g)]);
                dmma_884(acc[1][0], acc[1][1], Lr[k + 4], yb[vsw(k0 + k + 4 + q, g)]);
            }
            y[0] = acc[0][0] + acc[1][0];
            y[1] = acc[0][1] + acc[1][1];
        };
        auto put_y = [&] {
#pragma unroll
            for (int e = 0; e < 2; e++)
                if (i < nr && 2 * q + e < rc) Y[(f.start + r0 + i) * nrhs + j0 + 2 * q + e] = y[e];
        };
        __syncthreads();  // the ring is idle: it takes x_s
        if constexpr (sizeof(T) == 4) {
            xo[i * MG + 2 * q] = x[0];
            xo[i * MG + 2 * q + 1] = x[1];
            cluster.sync();
            for (int e = tid; e < WS * MG; e += CT) {
                const int k = e / MG;
                yb[vsw(k, e % MG)] = cluster.map_shared_rank(xo, k / CQ)[e - (k / CQ) * CQ * MG];
            }
            cp_async_wait<0>();
            __syncthreads();
            row_product(0, s * CQ + 8 * w + 8);  // the inverse rows 8w .. 8w+7 end at their diagonal
            put_y();
        } else {
            cp_async_wait<0>();
            cluster.sync();  // every CTA is past its tiles: y_t comes into the rows 64t of yb, x_s stands in its own
            const int nsub = (int)min((int64_t)CL, (f.k - b * WS + CQ - 1) / CQ);
            for (int t = 0; t < nsub; t++) {
                if (s == t) {
                    yb[vsw(CQ * t + i, 2 * q)] = x[0];
                    yb[vsw(CQ * t + i, 2 * q + 1)] = x[1];
                    __syncthreads();
                    row_product(CQ * t, 8 * w + 8);
                    for (int rk = t + 1; rk < nsub; rk++) {
                        double* o = cluster.map_shared_rank(yb, rk);
                        o[vsw(CQ * t + i, 2 * q)] = y[0];
                        o[vsw(CQ * t + i, 2 * q + 1)] = y[1];
                    }
                }
                if (t + 1 < nsub) cluster.sync();
                if (s == t) put_y();
                if (t + 1 == nsub) break;
                if (s > t && s < nsub) {
                    row_product(CQ * t, CQ);
                    x[0] -= y[0];
                    x[1] -= y[1];
                }
            }
        }
        chain_signal(&flags[b]);
        cluster.sync();  // the cluster's x_B pieces may be overwritten after this
    }
}

template <typename T>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CT, 1)
    k_chain_bwd_mm(double* __restrict__ Y, const T* __restrict__ panel, const double* __restrict__ inv,
                   const double* __restrict__ d, const double* part, const int64_t* __restrict__ colbase,
                   const DFront* __restrict__ fr, const int64_t* __restrict__ chain_blk,
                   const int64_t* __restrict__ items, int64_t nitems, int nrhs, int64_t nblocks,
                   int* __restrict__ flags0, int* __restrict__ counter, int* __restrict__ err) {
    pdl_launch_dependents();
    pdl_wait();
    cg::cluster_group cluster = cg::this_cluster();
    const int s = (int)cluster.block_rank(), ngrp = (nrhs + MG - 1) / MG;
    extern __shared__ __align__(16) double sm[];
    constexpr int RC = BRC<T>, BP = MBP<T>, PB = BPB<T>;
    double* Lc = sm;                                             // [WS][MLP]: rows 64s .. of inverse columns 64s ..
    T* ring = reinterpret_cast<T*>(sm + WS * MLP);               // [4][RC][BP]
    double* yp = reinterpret_cast<double*>(ring + 4 * RC * BP);  // [WS][MG]: y of a later block; then z_B
    double* zo = reinterpret_cast<double*>(ring);                // [CQ][MG]: this CTA's columns of z_B (ring idle)
    __shared__ int64_t s_item;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    for (;;) {
        const int64_t it = grab(cluster, &s_item, counter);
        if (it >= nitems * ngrp) break;
        const int64_t item = it / ngrp;
        const int jg = (int)(it - item * ngrp), j0 = jg * MG, rc = min(MG, nrhs - j0);
        const int64_t t = items[2 * item], b = items[2 * item + 1];
        const DFront f = fr[t];
        int* flags = flags0 + jg * nblocks + chain_blk[t];
        const int64_t col0 = b * WS + s * CQ;
        const int nc = (int)max((int64_t)0, min((int64_t)CQ, f.k - col0));
        const int64_t nb = (f.k + WS - 1) / WS;
        const int wb = (int)min((int64_t)WS, f.k - b * WS);
        load_bwd_block<T, MLP>(Lc, inv, panel + f.poff + (b * WS + CQ * (s + 1)) * f.ldp + col0, f, chain_blk[t] + b, b, s,
                               nc, wb - CQ * (s + 1));
        cp_async_commit();
        // the chunks of blocks nb − 1, ..., b + 1, PB per block
        const T* pcol = panel + f.poff + col0;
        const int nh = PB * (int)(nb - 1 - b);
        auto issue = [&](int h) {
            const int64_t ra = (nb - 1 - h / PB) * WS + (h % PB) * RC;
            const int nrr = (int)max((int64_t)0, min((int64_t)RC, f.k - ra));
            if (nc > 0)
                cp_async_tile<T>(ring + (h & 3) * RC * BP, BP, nrr > 0 ? pcol + ra * f.ldp : pcol, f.ldp, nrr, nc, RC, CQ,
                                 CT);
            cp_async_commit();
        };
        double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0}, tot[2] = {0.0, 0.0};
        for (int h = 0; h < min(3, nh); h++) issue(h);
        for (int h = 0; h < nh; h++) {
            if (h % PB == 0) {
                fold(a0, a1);
                fold(tot, a0);
                const int64_t bb = nb - 1 - h / PB;
                if (tid == 0) chain_wait(&flags[bb], CL, err);
                __syncthreads();
                const int wbb = (int)min((int64_t)WS, f.k - bb * WS);
                const double* src = Y + (f.start + bb * WS) * nrhs + j0;
                for (int e = tid; e < WS * MG; e += CT) {
                    const int k = e / MG, n = e % MG;
                    yp[vsw(k, n)] = (k < wbb && n < rc) ? __ldcg(src + (int64_t)k * nrhs + n) : 0.0;
                }
            }
            cp_wait_upto(min(2, nh - 1 - h));
            __syncthreads();  // chunk h visible; every thread is done with chunk h − 1
            if (h + 3 < nh) issue(h + 3);
            if (nc > 8 * w) {
                const T* Lt = ring + (h & 3) * RC * BP + q * BP + 8 * w + g;
                const int kb = (h % PB) * RC + q;
#pragma unroll
                for (int k = 0; k < RC; k += 8) {
                    dmma_884(a0[0], a0[1], (double)Lt[k * BP], yp[vsw(kb + k, g)]);
                    dmma_884(a1[0], a1[1], (double)Lt[(k + 4) * BP], yp[vsw(kb + k + 4, g)]);
                }
            }
        }
        double z[2];  // column 8w + g of z_s, right-hand sides 2q, 2q + 1
        const int c = 8 * w + g;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int n = 2 * q + e;
            z[e] = c < nc && n < rc ? chain_z(Y, d, part, colbase[t], f, col0 + c, nrhs, j0 + n) - (tot[e] + (a0[e] + a1[e])) : 0.0;
        }
        // y = Σ_k Lc[k, c]·yp[64s + k] over the rows [k0, k1) (relative to 64s)
        double y[2];
        auto col_product = [&](int k0, int k1) {
            double acc[2][2] = {};
            const double* Lq = Lc + q * MLP + 8 * w + g;
            for (int k = k0; k < k1; k += 8) {
                dmma_884(acc[0][0], acc[0][1], Lq[k * MLP], yp[vsw(s * CQ + k + q, g)]);
                dmma_884(acc[1][0], acc[1][1], Lq[(k + 4) * MLP], yp[vsw(s * CQ + k + 4 + q, g)]);
            }
            y[0] = acc[0][0] + acc[1][0];
            y[1] = acc[0][1] + acc[1][1];
        };
        auto put_y = [&] {
#pragma unroll
            for (int e = 0; e < 2; e++)
                if (c < nc && 2 * q + e < rc) Y[(f.start + col0 + c) * nrhs + j0 + 2 * q + e] = y[e];
        };
        __syncthreads();  // the ring is idle: it takes z_s
        if constexpr (sizeof(T) == 4) {
            zo[c * MG + 2 * q] = z[0];
            zo[c * MG + 2 * q + 1] = z[1];
            cluster.sync();
            for (int e = tid; e < WS * MG; e += CT) {
                const int k = e / MG;
                yp[vsw(k, e % MG)] = cluster.map_shared_rank(zo, k / CQ)[e - (k / CQ) * CQ * MG];
            }
            cp_async_wait<0>();
            __syncthreads();
            col_product(8 * w, WS - s * CQ);  // the inverse's columns start at their diagonal
            put_y();
        } else {
            cp_async_wait<0>();
            cluster.sync();  // every CTA is past its tiles: y_t comes into the rows 64t of yp, z_s stands in its own
            for (int t = (wb + CQ - 1) / CQ - 1; t >= 0; t--) {
                if (s == t) {
                    yp[vsw(CQ * t + c, 2 * q)] = z[0];
                    yp[vsw(CQ * t + c, 2 * q + 1)] = z[1];
                    __syncthreads();
                    col_product(8 * w, CQ);
                    for (int rk = 0; rk < t; rk++) {
                        double* o = cluster.map_shared_rank(yp, rk);
                        o[vsw(CQ * t + c, 2 * q)] = y[0];
                        o[vsw(CQ * t + c, 2 * q + 1)] = y[1];
                    }
                }
                if (t > 0) cluster.sync();
                if (s == t) put_y();
                if (t == 0) break;
                if (s < t) {
                    col_product(CQ * (t - s), CQ * (t - s) + CQ);
                    z[0] -= y[0];
                    z[1] -= y[1];
                }
            }
        }
        chain_signal(&flags[b]);
        cluster.sync();  // the cluster's z_B pieces may be overwritten after this
    }
}

// Later rows, NT groups in one CTA: pieces of L and of the vectors (pitch 8·NT + 4 doubles)
// stream together through a four-slot ring.
template <int NT>
constexpr int MVP = MG * NT + 4;
template <typename T, int NT>
constexpr size_t mm_rows_smem = (size_t)4 * CQ * MFP<T> * sizeof(T) + (size_t)4 * FQC<T> * MVP<NT> * 8;
template <typename T, int NT>
constexpr size_t mm_cols_smem = (size_t)4 * BRC<T> * MBP<T> * sizeof(T) + (size_t)4 * BRC<T> * MVP<NT> * 8;

// cp.async of n rows of nrhs contiguous values into rows of pitch MVP, zero beyond the rows and
// beyond nrhs; src rows are contiguous
template <int NT>
__device__ __forceinline__ void vec_piece(double* dst, const double* src, int n, int nrhs, int rows) {
    for (int e = threadIdx.x; e < rows * MG * NT; e += CT) {
        const int k = e / (MG * NT), c = e % (MG * NT);
        double* o = dst + k * MVP<NT> + c;
        if (k < n && c < nrhs)
            cp_async8(o, src + (int64_t)k * nrhs + c);
        else
            *o = 0.0;
    }
}

template <typename T, int NT>
__global__ void __launch_bounds__(CT) k_chain_rows_mm(const double* Y, double* __restrict__ V,
                                                      const int32_t* __restrict__ imap, const T* __restrict__ panel,
                                                      const DFront* __restrict__ fr, const int64_t* __restrict__ items,
                                                      int nrhs) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) double sm[];
    constexpr int QC = FQC<T>, QP = MFP<T>, VP = MVP<NT>;
    double* yr = sm;                                         // [4][QC][VP]
    T* ring = reinterpret_cast<T*>(sm + 4 * QC * VP);        // [4][CQ][QP]
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int64_t t = items[2 * blockIdx.x], c = items[2 * blockIdx.x + 1];
    const DFront f = fr[t];
    const int64_t r0 = f.k + c * CQ;
    const int nr = (int)min((int64_t)CQ, f.m - r0);
    const int nq = (int)((f.k + QC - 1) / QC);
    const T* prow = panel + f.poff + r0 * f.ldp;
    auto issue = [&](int Q) {
        const int64_t c0 = (int64_t)Q * QC;
        const int ncol = (int)min((int64_t)QC, f.k - c0);
        cp_async_tile<T>(ring + (Q & 3) * CQ * QP, QP, prow + c0, f.ldp, nr, ncol, CQ, QC, CT);
        vec_piece<NT>(yr + (Q & 3) * QC * VP, Y + (f.start + c0) * nrhs, ncol, nrhs, QC);
        cp_async_commit();
    };
    double acc[NT][2] = {}, tot[NT][2] = {};
    for (int Q = 0; Q < min(3, nq); Q++) issue(Q);
    for (int Q = 0; Q < nq; Q++) {
        if (Q % FPB<T> == 0) fold(tot, acc);
        cp_wait_upto(min(2, nq - 1 - Q));
        __syncthreads();
        if (Q + 3 < nq) issue(Q + 3);
        const T* Lt = ring + (Q & 3) * CQ * QP + (8 * w + g) * QP + q;
        const double* yq = yr + (Q & 3) * QC * VP + q * VP + g;
#pragma unroll 4
        for (int k = 0; k < QC; k += 4) {
            const double a = (double)Lt[k];
#pragma unroll
            for (int n = 0; n < NT; n++) dmma_884(acc[n][0], acc[n][1], a, yq[k * VP + n * MG]);
        }
    }
    const int i = 8 * w + g;
    if (i < nr) {
        double* vt = V + (f.vuoff + c * CQ + i) * nrhs;
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int j = n * MG + 2 * q + e;
                if (j < nrhs) vt[j] = kids_add(0.0, V, imap, f, r0 + i, nrhs, j) - (tot[n][e] + acc[n][e]);
            }
    }
}

template <typename T, int NT>
__global__ void __launch_bounds__(CT) k_chain_cols_mm(double* __restrict__ part, const double* V,
                                                      const T* __restrict__ panel, const DFront* __restrict__ fr,
                                                      const int64_t* __restrict__ items, int nrhs) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) double sm[];
    constexpr int RC = BRC<T>, BP = MBP<T>, VP = MVP<NT>;
    double* yr = sm;                                   // [4][RC][VP]
    T* ring = reinterpret_cast<T*>(sm + 4 * RC * VP);  // [4][RC][BP]
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int64_t t = items[2 * blockIdx.x], cc = items[2 * blockIdx.x + 1];
    const DFront f = fr[t];
    const int64_t col0 = cc * CQ;
    const int nc = (int)min((int64_t)CQ, f.k - col0);
    const int nchunk = (int)((f.u + RC - 1) / RC), grp = blockIdx.y;
    const int h0 = nchunk * grp / CHAIN_GROUPS, nh = nchunk * (grp + 1) / CHAIN_GROUPS - h0;
    auto issue = [&](int h) {
        const int64_t ra = (int64_t)(h0 + h) * RC;
        const int nrr = (int)min((int64_t)RC, f.u - ra);
        cp_async_tile<T>(ring + (h & 3) * RC * BP, BP, panel + f.poff + (f.k + ra) * f.ldp + col0, f.ldp, nrr, nc, RC, CQ,
                         CT);
        vec_piece<NT>(yr + (h & 3) * RC * VP, V + (f.vuoff + ra) * nrhs, nrr, nrhs, RC);
        cp_async_commit();
    };
    double acc[NT][2] = {}, tot[NT][2] = {};
    for (int h = 0; h < min(3, nh); h++) issue(h);
    for (int h = 0; h < nh; h++) {
        if (h % BPB<T> == 0) fold(tot, acc);
        cp_wait_upto(min(2, nh - 1 - h));
        __syncthreads();
        if (h + 3 < nh) issue(h + 3);
        const T* Lt = ring + (h & 3) * RC * BP + q * BP + 8 * w + g;
        const double* yq = yr + (h & 3) * RC * VP + q * VP + g;
#pragma unroll 4
        for (int k = 0; k < RC; k += 4) {
            const double a = (double)Lt[k * BP];
#pragma unroll
            for (int n = 0; n < NT; n++) dmma_884(acc[n][0], acc[n][1], a, yq[k * VP + n * MG]);
        }
    }
    double* out = part + (((int64_t)blockIdx.x * CHAIN_GROUPS + grp) * CQ + 8 * w + g) * nrhs;
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int j = n * MG + 2 * q + e;
            if (j < nrhs) out[j] = tot[n][e] + acc[n][e];
        }
}

// The inverse of a chain block's unit-lower diagonal block, by block columns of NB:
// M_jj = inv(L_jj) (from the factorization), M_ij = −inv(L_ii)·Σ_{j ≤ t < i} L_it·M_tj.
// The block columns are independent: one CTA (8 warps of 32×16 outputs) each, its M_tj kept
// in shared memory, the products on the FP64 tensor-core path. It is bound by the chain of
// 64³ products of block column 0 (nine for a full block) and by the loads of L between them.
// For an FP32 factor; an FP64 one is solved by substitution (the head of this file).
constexpr int IVP = NB + 4;  // pitch (doubles): fragment loads of both operands without conflicts
constexpr size_t INV_SMEM = (size_t)5 * NB * IVP * sizeof(double);

__global__ void __launch_bounds__(256) k_chain_inverse(double* __restrict__ cinv, const float* __restrict__ panel,
                                                       const double* __restrict__ linv, const DFront* __restrict__ fr,
                                                       const int64_t* __restrict__ chain_blk,
                                                       const int64_t* __restrict__ chain_bfront) {
    extern __shared__ __align__(16) double sm[];
    double* A = sm;                  // [NB][IVP]: L_it, then inv(L_ii)
    double* B = sm + NB * IVP;       // [NB][IVP]: the sum
    double* Mt = sm + 2 * NB * IVP;  // [3][NB][IVP]: M_jj, M_{j+1,j}, M_{j+2,j}
    const int64_t cb = blockIdx.x, ft = chain_bfront[cb];
    const int j = blockIdx.y;
    const DFront f = fr[ft];
    const int64_t b = cb - chain_blk[ft], J0 = b * WS;
    const int wb = (int)min((int64_t)WS, f.k - J0), nbw = (wb + NB - 1) / NB;
    double* M = cinv + cb * (int64_t)WS * WS + j * NB;  // the block column
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int wm = warp & 1, wn = warp >> 1;
    // zero above the diagonal block and beyond the block's width
    for (int e = tid; e < WS * NB / 2; e += 256) {
        const int r = e / (NB / 2), c = 2 * (e % (NB / 2));
        if (j >= nbw || r < j * NB || r >= nbw * NB)
            *reinterpret_cast<double2*>(M + (int64_t)r * WS + c) = make_double2(0.0, 0.0);
    }
    if (j >= nbw) return;
    const double* li = linv + (f.blk_off + 4 * b) * (int64_t)(NB * NB);
    for (int e = tid; e < NB * NB; e += 256) {
        const double v = li[j * NB * NB + e];
        Mt[(e / NB) * IVP + e % NB] = v;
        M[(int64_t)(j * NB + e / NB) * WS + e % NB] = v;
    }
    // acc += A·B over NB: rows 32·wm + 8a + g, columns 16·wn + 8c + 2q + {0, 1}
    auto gemm = [&](double (&acc)[4][2][2], const double* Bt) {
        const double* a0 = A + (wm * 32 + g) * IVP + q;
        const double* b0 = Bt + q * IVP + wn * 16 + g;
#pragma unroll 4
        for (int k = 0; k < NB; k += 4) {
            double fa[4], fb[2];
#pragma unroll
            for (int a = 0; a < 4; a++) fa[a] = a0[a * 8 * IVP + k];
#pragma unroll
            for (int c = 0; c < 2; c++) fb[c] = b0[k * IVP + c * 8];
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int c = 0; c < 2; c++) dmma_884(acc[a][c][0], acc[a][c][1], fa[a], fb[c]);
        }
    };
    for (int i = j + 1; i < nbw; i++) {
        double acc[4][2][2] = {};
        for (int t = j; t < i; t++) {
            __syncthreads();  // A is read
            for (int e = tid; e < NB * NB; e += 256) {
                const int row = i * NB + e / NB;
                A[(e / NB) * IVP + e % NB] =
                    row < wb ? (double)panel[f.poff + (J0 + row) * f.ldp + J0 + t * NB + e % NB] : 0.0;
            }
            __syncthreads();
            gemm(acc, Mt + (t - j) * NB * IVP);
        }
        __syncthreads();
        for (int e = tid; e < NB * NB; e += 256) A[(e / NB) * IVP + e % NB] = li[i * NB * NB + e];
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    B[(wm * 32 + a * 8 + g) * IVP + wn * 16 + c * 8 + 2 * q + e] = acc[a][c][e];
        __syncthreads();
        double acc2[4][2][2] = {};
        gemm(acc2, B);
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int r = wm * 32 + a * 8 + g, cc = wn * 16 + c * 8 + 2 * q + e;
                    M[(int64_t)(i * NB + r) * WS + cc] = -acc2[a][c][e];
                    if (i - j < 3) Mt[((i - j) * NB + r) * IVP + cc] = -acc2[a][c][e];
                }
    }
}

// per device: attributes set, the number of clusters that fit at once (forward, backward;
// by right-hand sides 1 .. 4)
struct ChainDev {
    bool done = false;
    int fwd[2][5] = {}, bwd[2][5] = {};  // [0] FP32, [1] FP64 factor; by right-hand sides 1 .. 4, [0] the groups
};
template <typename T>
constexpr int chain_kind = sizeof(T) == 8 ? 1 : 0;

template <typename K>
int fit_clusters(K kern, size_t smem) {
    RFG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CL * 64);
    cfg.blockDim = dim3(CT);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    RFG_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
    return n;
}

constexpr size_t rows_smem(int R) { return (size_t)4 * CQ * FQP<float> * sizeof(float) + (size_t)WS * R * 8; }
constexpr size_t cols_smem(int R) { return (size_t)4 * BRC<float> * BTP * sizeof(float) + (size_t)8 * CQ * R * 8; }

template <typename K>
void set_smem(K kern, size_t bytes) {
    RFG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}
template <typename T, int R>
void set_chain_attrs(ChainDev& d) {
    d.fwd[chain_kind<T>][R] = fit_clusters(k_chain_fwd<T, R>, fwd_smem(R));
    d.bwd[chain_kind<T>][R] = fit_clusters(k_chain_bwd<T, R>, bwd_smem(R));
    set_smem(k_chain_rows<T, R>, rows_smem(R));
    set_smem(k_chain_cols<T, R>, cols_smem(R));
    set_smem(k_chain_rows_mm<T, R>, mm_rows_smem<T, R>);
    set_smem(k_chain_cols_mm<T, R>, mm_cols_smem<T, R>);
}
template <typename T>
void set_chain_attrs_all(ChainDev& d) {
    set_chain_attrs<T, 1>(d);
    set_chain_attrs<T, 2>(d);
    set_chain_attrs<T, 3>(d);
    set_chain_attrs<T, 4>(d);
    d.fwd[chain_kind<T>][0] = fit_clusters(k_chain_fwd_mm<T>, mm_fwd_smem<T>);
    d.bwd[chain_kind<T>][0] = fit_clusters(k_chain_bwd_mm<T>, mm_bwd_smem<T>);
}

const ChainDev& chain_dev() {
    static std::mutex mu;
    static ChainDev devs[64];
    int dev = 0;
    RFG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) throw CudaError("solve chain: device ordinal out of range");
    std::lock_guard<std::mutex> lock(mu);
    ChainDev& d = devs[dev];
    if (!d.done) {
        set_smem(k_chain_inverse, INV_SMEM);
        set_chain_attrs_all<float>(d);
        set_chain_attrs_all<double>(d);
        d.done = true;
    }
    return d;
}

unsigned grid_for_items(int fit, int64_t nitems) {
    if (fit <= 0) throw CudaError("solve chain: no cluster of four CTAs fits on this device");
    return (unsigned)(std::min<int64_t>(fit, nitems) * CL);
}

// what the chains multiply by in a block's solve
template <typename T>
const double* block_inverses(const ChainArgs& c) {
    return sizeof(T) == 8 ? c.linv : c.cinv;
}

void check_nrhs(int nrhs) {
    if (nrhs < 1 || nrhs > 4 * MG) throw CudaError("solve chain: 1 to 32 right-hand sides");
}

}  // namespace

void launch_chain_inverse(double* cinv, const float* panel, const double* linv, const DFront* fronts,
                          const int64_t* chain_blk, const int64_t* chain_bfront, int64_t nblocks, cudaStream_t st) {
    if (nblocks <= 0) return;
    chain_dev();
    k_chain_inverse<<<dim3((unsigned)nblocks, CL), 256, INV_SMEM, st>>>(cinv, panel, linv, fronts, chain_blk,
                                                                       chain_bfront);
    RFG_CUDA(cudaGetLastError());
}

// one of four instantiations (by the number of right-hand sides or of groups)
#define RFG_CHAIN_BY_R(num, CALL) \
    do {                          \
        if ((num) == 1) {         \
            constexpr int R = 1;  \
            CALL;                 \
        } else if ((num) == 2) {  \
            constexpr int R = 2;  \
            CALL;                 \
        } else if ((num) == 3) {  \
            constexpr int R = 3;  \
            CALL;                 \
        } else {                  \
            constexpr int R = 4;  \
            CALL;                 \
        }                         \
    } while (0)

template <typename T>
void launch_chain_fwd(int nrhs, int64_t nitems, const double* X, double* Y, const double* V, const T* panel,
                      const ChainArgs& c, const int64_t* items, int* flags, int* counter, cudaStream_t st) {
    if (nitems <= 0) return;
    check_nrhs(nrhs);
    const ChainDev& d = chain_dev();
    if (nrhs > 4) {
        const int64_t n = nitems * ((nrhs + MG - 1) / MG);
        launch_pdl(true, k_chain_fwd_mm<T>, dim3(grid_for_items(d.fwd[chain_kind<T>][0], n)), dim3(CT), mm_fwd_smem<T>,
                   st, X, Y, panel, V, c.imap, block_inverses<T>(c), c.fronts, c.blk, items, nitems, nrhs, c.nblocks, flags, counter,
                   c.err);
        return;
    }
    RFG_CHAIN_BY_R(nrhs, launch_pdl(true, k_chain_fwd<T, R>, dim3(grid_for_items(d.fwd[chain_kind<T>][R], nitems)),
                                    dim3(CT), fwd_smem(R), st, X, Y, panel, V, c.imap, block_inverses<T>(c), c.fronts, c.blk, items,
                                    nitems, flags, counter, c.err));
}

template <typename T>
void launch_chain_rows(int nrhs, int64_t nitems, const double* Y, double* V, const T* panel, const ChainArgs& c,
                       const int64_t* items, cudaStream_t st) {
    if (nitems <= 0) return;
    check_nrhs(nrhs);
    chain_dev();
    if (nrhs > 4) {
        RFG_CHAIN_BY_R((nrhs + MG - 1) / MG,
                       launch_pdl(true, k_chain_rows_mm<T, R>, dim3((unsigned)nitems), dim3(CT), mm_rows_smem<T, R>, st,
                                  Y, V, c.imap, panel, c.fronts, items, nrhs));
        return;
    }
    RFG_CHAIN_BY_R(nrhs, launch_pdl(true, k_chain_rows<T, R>, dim3((unsigned)nitems), dim3(CT), rows_smem(R), st, Y, V,
                                    c.imap, panel, c.fronts, items));
}

template <typename T>
void launch_chain_cols(int nrhs, int64_t ngather, const int64_t* gather_items, int64_t nitems, const int64_t* items,
                       const double* Y, double* V, double* part, const T* panel, const ChainArgs& c, cudaStream_t st) {
    if (nitems <= 0) return;
    check_nrhs(nrhs);
    chain_dev();
    if (ngather > 0)
        launch_pdl(true, k_chain_gather, dim3((unsigned)ngather), dim3(CT), 0, st, Y, V, c.fronts, c.rows, gather_items,
                   nrhs);
    const dim3 grid((unsigned)nitems, CHAIN_GROUPS);
    if (nrhs > 4) {
        RFG_CHAIN_BY_R((nrhs + MG - 1) / MG,
                       launch_pdl(true, k_chain_cols_mm<T, R>, grid, dim3(CT), mm_cols_smem<T, R>, st, part,
                                  (const double*)V, panel, c.fronts, items, nrhs));
        return;
    }
    RFG_CHAIN_BY_R(nrhs, launch_pdl(true, k_chain_cols<T, R>, grid, dim3(CT), cols_smem(R), st, part, (const double*)V,
                                    panel, c.fronts, items));
}

template <typename T>
void launch_chain_bwd(int nrhs, int64_t nitems, double* Y, const double* part, const T* panel, const ChainArgs& c,
                      const int64_t* items, int* flags, int* counter, cudaStream_t st) {
    if (nitems <= 0) return;
    check_nrhs(nrhs);
    const ChainDev& d = chain_dev();
    if (nrhs > 4) {
        const int64_t n = nitems * ((nrhs + MG - 1) / MG);
        launch_pdl(true, k_chain_bwd_mm<T>, dim3(grid_for_items(d.bwd[chain_kind<T>][0], n)), dim3(CT), mm_bwd_smem<T>,
                   st, Y, panel, block_inverses<T>(c), c.d, part, c.colbase, c.fronts, c.blk, items, nitems, nrhs, c.nblocks, flags,
                   counter, c.err);
        return;
    }
    RFG_CHAIN_BY_R(nrhs, launch_pdl(true, k_chain_bwd<T, R>, dim3(grid_for_items(d.bwd[chain_kind<T>][R], nitems)),
                                    dim3(CT), bwd_smem(R), st, Y, panel, block_inverses<T>(c), c.d, part, c.colbase, c.fronts, c.blk,
                                    items, nitems, flags, counter, c.err));
}

#undef RFG_CHAIN_BY_R

#define RFG_CHAIN_INSTANCE(T)                                                                                        \
    template void launch_chain_fwd<T>(int, int64_t, const double*, double*, const double*, const T*,                 \
                                      const ChainArgs&, const int64_t*, int*, int*, cudaStream_t);                   \
    template void launch_chain_rows<T>(int, int64_t, const double*, double*, const T*, const ChainArgs&,             \
                                       const int64_t*, cudaStream_t);                                                \
    template void launch_chain_cols<T>(int, int64_t, const int64_t*, int64_t, const int64_t*, const double*,         \
                                       double*, double*, const T*, const ChainArgs&, cudaStream_t);                  \
    template void launch_chain_bwd<T>(int, int64_t, double*, const double*, const T*, const ChainArgs&,              \
                                      const int64_t*, int*, int*, cudaStream_t);
RFG_CHAIN_INSTANCE(float)
RFG_CHAIN_INSTANCE(double)
#undef RFG_CHAIN_INSTANCE

}  // namespace rfg
