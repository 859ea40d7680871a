// Triangular solves over the elimination tree, and FP64 iterative refinement.
//
// The solve follows the level schedule of the factor (plan.h) in steps of WS = 4·NB
// pivots (WStep), for nrhs right-hand sides stored as X[q·nrhs + j] (internal
// numbering):
//  forward  (leaves up)   per level and step, a diagonal kernel solves the step's diagonal
//                         block with its four stored NB×NB inverse blocks (y_B → Y) and a
//                         rows kernel subtracts L[r, J0:J1]·y_B from the rows below (X or the
//                         front's update vector V_t). The first step of a front adds the
//                         children's update vectors on the way, through the map of each row
//                         to the children's rows (kids_add: child 0 before child 1);
//  backward (root down)   per step, last first: partial sums of Lᵀ·y over row chunks
//                         below the block, then the diagonal block backwards from
//                         z = Y/D − Σ partials.
// One to four right-hand sides run the _pf (FP32 factor) and _pd (FP64) kernels, five to 32
// the _mm kernels on the FP64 tensor-core path; the levels at the top run as chains (chain.h).
// Every kernel of a sweep is launched as a programmatic dependent of the one before
// (PDL): the kernels copy their factor data into shared memory before they wait for
// the vectors of the previous kernel.
// This is the multifrontal form of Factor::solve (src/sparse.rs:615-652): the same
// three sweeps, with the updates of each front gathered in its update vector instead
// of being subtracted from x row by row.

#include <cuda_runtime.h>


#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "chain.h"
#include "engine.h"
#include "par.h"
#include "tiles.cuh"

// Scratch of rfg_solve_device_noalloc: a fixed array in the library's device image,
// so that solves through that entry point allocate nothing. The driver reserves it
// when the library's kernels are loaded on a device, once per process and device.
static __device__ __align__(256) unsigned char g_noalloc_scratch[rfg::NOALLOC_SCRATCH_BYTES];

namespace rfg {

namespace {

constexpr int MAXR = 32;  // right-hand sides per sweep
__device__ __forceinline__ int64_t find_slot2(const int64_t* pre, int64_t n, int64_t b) {
    int64_t lo = 0, hi = n;
    while (hi - lo > 1) {
        int64_t mid = (lo + hi) >> 1;
        if (pre[mid] <= b)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// Prefetching step kernels for at most PF_MAXR right-hand sides.
// Every kernel of a sweep is launched as a programmatic dependent of the one before it:
// it starts while its predecessor runs, copies the factor data it needs (unchanged
// during a solve) into shared memory with cp.async, and only then waits for the
// predecessor's results. At the top of the tree, where a wide step is a chain of small
// launches, a step then costs its arithmetic instead of one global-memory round trip per
// stage plus a launch gap per kernel. The backward step is split in two: k_wbwd_part
// (partial sums of Lᵀ·y over row chunks) and k_wbwd_diag (one CTA per front: the sum of
// the partials in chunk order, then the diagonal block backwards). Shared memory is
// sized per step from the widest front of the step, so the many small fronts of the
// lower levels keep several CTAs per SM.
// ---------------------------------------------------------------------------
constexpr int PF_MAXR = 4;

// row tile of the rows / partial kernels: PF_RPC rows (half of a PR-row chunk of the plan)
// × cols floats (cols = the step's widest block rounded up to 32), row pitch cols + 8
// (16-byte rows, conflict-free row reads); three such CTAs fit on an SM
constexpr int PF_RPC = PR / 2;
// The rows kernel takes 64 rows of an FP32 factor per CTA and 32 of an FP64 one (the same bytes);
// the partial sums take 64 in both, so that the partial blocks of a chunk stay two.
template <typename T>
constexpr int PF_ROWS = PF_RPC * 4 / (int)sizeof(T);
// row pitch: the lanes of a row (two for FP32, four for FP64) read its 16-byte groups in turn, and the
// pitch keeps eight lanes' reads in different banks. (FP32 rows read in two halves at a pitch of
// cols + 4 met every bank twice: the refined solve of the 60³ cube 17.93 ms, now 17.56.)
template <typename T>
__host__ __device__ inline int pf_pitch(int cols) { return cols + 8; }
inline int pf_cols(int64_t wb_max) { return (int)((wb_max + 31) / 32 * 32); }
template <typename T>
size_t pf_rows_smem(int cols, int nrhs) {
    return (size_t)PF_ROWS<T> * pf_pitch<T>(cols) * sizeof(T) + (size_t)WS * nrhs * sizeof(double);
}
template <typename T>
size_t pf_part_smem(int cols, int nrhs) {
    return (size_t)PF_RPC * pf_pitch<T>(cols) * sizeof(T) + (size_t)PF_RPC * nrhs * sizeof(double) +
           (size_t)256 * nrhs * sizeof(double);
}
// diagonal kernels: min(nbw, 3) inverse blocks, nbw(nbw−1)/2 panel pieces (NB×NB), the
// block's vectors; nbw = the step's largest number of NB sub-blocks
__host__ __device__ inline int pf_nli(int nbw) { return nbw < 3 ? nbw : 3; }
__host__ __device__ inline int pf_npc(int nbw) { return nbw * (nbw - 1) / 2; }
// FP64 factor: the inverse blocks and pieces are tiles of one size, at most PD_SLOTS of them
// resident (all ten of a full block are 320 KB)
constexpr int PD_SLOTS = 6;
__host__ __device__ inline int pd_slots(int nbw) { return nbw + pf_npc(nbw) < PD_SLOTS ? nbw + pf_npc(nbw) : PD_SLOTS; }
inline size_t pd_diag_smem(int nbw, int nrhs) {
    return (size_t)pd_slots(nbw) * NB * NB * sizeof(double) + (size_t)(WS + NB + 4 * NB) * nrhs * sizeof(double);
}
inline size_t pf_diag_smem(int nbw, int nrhs) {
    return (size_t)pf_nli(nbw) * NB * NB * sizeof(double) + (size_t)pf_npc(nbw) * NB * NB * sizeof(float) +
           (size_t)(WS + NB + 4 * NB) * nrhs * sizeof(double);
}

// Sums of eight rows across a warp: v[i] holds lane's partial of row i; on return every
// lane holds the total of row (lane >> 2) & 7 (three exchange steps that halve the rows
// held, then two plain steps).
template <int R>
__device__ __forceinline__ void warp_sum8(const double (&v)[8][R], double (&out)[R]) {
    const int lane = threadIdx.x & 31;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    double w4[4][R], w2[2][R];
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int r = 0; r < R; r++) {
            const double send = b4 ? v[j][r] : v[j + 4][r], keep = b4 ? v[j + 4][r] : v[j][r];
            w4[j][r] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
        for (int r = 0; r < R; r++) {
            const double send = b3 ? w4[j][r] : w4[j + 2][r], keep = b3 ? w4[j + 2][r] : w4[j][r];
            w2[j][r] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
#pragma unroll
    for (int r = 0; r < R; r++) {
        const double send = b2 ? w2[0][r] : w2[1][r], keep = b2 ? w2[1][r] : w2[0][r];
        double o = keep + __shfl_xor_sync(0xffffffffu, send, 4);
        o += __shfl_xor_sync(0xffffffffu, o, 2);
        out[r] = o + __shfl_xor_sync(0xffffffffu, o, 1);
    }
}

// Forward diagonal block of a wide step: one CTA (256 threads) per active front. Pieces
// in column-block order ((1,0) (2,0) (3,0) (2,1) (3,1) (3,2) for four sub-blocks); with
// four sub-blocks the inverse block of sub-block 3 is copied into the space of column
// block 0 once stage 0 is done.
template <int R>
__global__ void __launch_bounds__(256) k_wfwd_diag_pf(const double* X, double* __restrict__ Y,
                                                      const float* __restrict__ panel, const double* __restrict__ linv,
                                                      const DFront* __restrict__ fr, const int64_t* __restrict__ order,
                                                      int64_t fr_off, int64_t S, int nbw_max,
                                                      const double* V, const int32_t* __restrict__ imap) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    double* Li = sm;                                                     // [nli][NB][NB]
    float* Pc = reinterpret_cast<float*>(sm + pf_nli(nbw_max) * NB * NB);  // [npc][NB][NB]
    double* xB = sm + pf_nli(nbw_max) * NB * NB + pf_npc(nbw_max) * NB * NB / 2;  // [WS][R]
    double* yb = xB + WS * R;                                                  // [NB][R]
    const DFront f = fr[order[fr_off + blockIdx.x]];
    const int64_t J0 = S * WS;
    const int wb = (int)min((int64_t)WS, f.k - J0), nbw = (wb + NB - 1) / NB;
    const double* lsrc = linv + (f.blk_off + S * 4) * (int64_t)(NB * NB);
    cp_async_flat(Li, lsrc, min(nbw, 3) * NB * NB / 2, 256);
    for (int b = 0; b + 1 < nbw; b++)
        for (int b2 = b + 1; b2 < nbw; b2++) {
            const int pi = b * (nbw - 1) - b * (b - 1) / 2 + (b2 - b - 1);
            cp_async_tile<float>(Pc + pi * NB * NB, NB, panel + f.poff + (J0 + b2 * NB) * f.ldp + J0 + b * NB, f.ldp,
                                 min(NB, wb - b2 * NB), NB, NB, NB, 256);
        }
    cp_async_commit();
    pdl_wait();
    const double* xs = X + (f.start + J0) * R;
    if (threadIdx.x < nbw * NB) {
        const int p = threadIdx.x;
#pragma unroll
        for (int r = 0; r < R; r++) {
            double x = p < wb ? __ldcg(xs + p * R + r) : 0.0;
            if (S == 0 && p < wb) x = kids_add(x, V, imap, f, p, R, r);
            xB[p * R + r] = x;
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sel = (lane >> 2) & 7;
    for (int b = 0; b < nbw; b++) {
        const int jbb = min(NB, wb - b * NB);
        if (b == 0 || b == 3) cp_async_wait<0>();
        __syncthreads();
        // y_b = L_bb⁻¹·x_b: warp w takes rows 8w..8w+7, lanes the columns q and q+32
        {
            const double* L = b < 3 ? Li + b * NB * NB : reinterpret_cast<const double*>(Pc);
            double x0[R], x1[R], v[8][R], out[R];
#pragma unroll
            for (int j = 0; j < R; j++) {
                x0[j] = xB[(b * NB + lane) * R + j];
                x1[j] = xB[(b * NB + lane + 32) * R + j];
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const double l0 = L[(8 * warp + i) * NB + lane], l1 = L[(8 * warp + i) * NB + lane + 32];
#pragma unroll
                for (int j = 0; j < R; j++) v[i][j] = fma(l0, x0[j], l1 * x1[j]);
            }
            warp_sum8<R>(v, out);
            if ((lane & 3) == 0) {
                const int p = 8 * warp + sel;
#pragma unroll
                for (int j = 0; j < R; j++) {
                    yb[p * R + j] = out[j];
                    if (p < jbb) Y[(f.start + J0 + b * NB + p) * R + j] = out[j];
                }
            }
        }
        __syncthreads();
        if (b + 1 < nbw) {
            // x_b2 −= L[b2, b]·y_b for the sub-blocks below, eight rows per warp at a time
            double y0[R], y1[R];
#pragma unroll
            for (int j = 0; j < R; j++) {
                y0[j] = yb[lane * R + j];
                y1[j] = yb[(lane + 32) * R + j];
            }
            const int first = b * (nbw - 1) - b * (b - 1) / 2;  // column block b's first piece
            const int ngrp = (nbw - 1 - b) * NB / 8;
            for (int g = warp; g < ngrp; g += 8) {
                double v[8][R], out[R];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float* row = Pc + (first * NB + 8 * g + i) * NB;
                    const double l0 = row[lane], l1 = row[lane + 32];
#pragma unroll
                    for (int j = 0; j < R; j++) v[i][j] = fma(l0, y0[j], l1 * y1[j]);
                }
                warp_sum8<R>(v, out);
                if ((lane & 3) == 0) {
#pragma unroll
                    for (int j = 0; j < R; j++) xB[((b + 1) * NB + 8 * g + sel) * R + j] -= out[j];
                }
            }
            if (b == 0 && nbw == 4) {
                __syncthreads();  // column block 0's pieces are read: the last inverse block goes there
                cp_async_flat(Pc, lsrc + 3 * NB * NB, NB * NB / 2, 256);
                cp_async_commit();
            }
        }
    }
}

// Rows below a wide block: X (pivot rows) or V (later rows) −= L[r, J0:J1]·y_B. PF_ROWS rows
// per CTA (two or four CTAs per PR-row chunk), two (FP32) or four (FP64) threads per row, the
// row tile prefetched before the wait for y_B.
template <typename T, int R>
__global__ void __launch_bounds__(PR) k_wfwd_rows_pf(double* __restrict__ X, double* __restrict__ V,
                                                     const double* Y, const T* __restrict__ panel,
                                                     const DFront* __restrict__ fr, const int2* __restrict__ slots,
                                                     const int64_t* __restrict__ pre,
                                                     int64_t S, int cols, const int32_t* __restrict__ imap) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    constexpr int RPC = PF_ROWS<T>, SUB = PR / RPC, TPR = PR / RPC, VEC = 16 / (int)sizeof(T);
    using VT = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
    const int pitch = pf_pitch<T>(cols);
    T* Lt = reinterpret_cast<T*>(sm);                              // [RPC][pitch]
    double* yB = sm + RPC * pitch * sizeof(T) / sizeof(double);    // [WS][R]
    const int64_t b = blockIdx.x / SUB;
    const int2 sf = __ldg(slots + b);
    const int64_t i = sf.x, chunk = b - pre[i];
    const DFront f = fr[sf.y];
    const int64_t J0 = S * WS, J1 = min(J0 + WS, f.k);
    const int wb = (int)(J1 - J0);
    const int64_t r0 = J1 + chunk * PR + (blockIdx.x % SUB) * RPC;
    const int nr = (int)max((int64_t)0, min((int64_t)RPC, f.m - r0));
    if (nr > 0) cp_async_tile<T>(Lt, pitch, panel + f.poff + r0 * f.ldp + J0, f.ldp, nr, wb, nr, cols, PR);
    cp_async_commit();
    pdl_wait();
    if (nr == 0) return;
    const double* ys = Y + (f.start + J0) * R;
    for (int idx = threadIdx.x; idx < cols * R; idx += PR) yB[idx] = idx < wb * R ? __ldcg(ys + idx) : 0.0;
    cp_async_wait<0>();
    __syncthreads();
    const int rr = threadIdx.x / TPR, h = threadIdx.x % TPR;
    double acc[R][2];
#pragma unroll
    for (int j = 0; j < R; j++) acc[j][0] = acc[j][1] = 0.0;
    const int nq = cols / (VEC * TPR);
    const VT* row = reinterpret_cast<const VT*>(Lt + rr * pitch);
#pragma unroll 4
    for (int u = 0; u < nq; u++) {
        const int q = h + u * TPR;
        const VT lv = row[q];
        const T* l = reinterpret_cast<const T*>(&lv);
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
            for (int e = 0; e < VEC; e++)
                acc[j][e & 1] = fma((double)l[e], yB[(VEC * q + e) * R + j], acc[j][e & 1]);
    }
    double v[R];
#pragma unroll
    for (int j = 0; j < R; j++) {
        v[j] = acc[j][0] + acc[j][1];
        v[j] += __shfl_xor_sync(0xffffffffu, v[j], 1);
        if (TPR == 4) v[j] += __shfl_xor_sync(0xffffffffu, v[j], 2);
    }
    if (h == 0 && rr < nr) {
        const int64_t r = r0 + rr;
        double* tgt = r < f.k ? X + (f.start + r) * R : V + (f.vuoff + r - f.k) * R;
        if (S == 0) {
            // the first step of the front: the children's part on the way (V starts from it)
#pragma unroll
            for (int j = 0; j < R; j++) tgt[j] = kids_add(r < f.k ? __ldcg(tgt + j) : 0.0, V, imap, f, r, R, j) - v[j];
        } else {
#pragma unroll
            for (int j = 0; j < R; j++) tgt[j] = __ldcg(tgt + j) - v[j];
        }
    }
}

// Backward partial sums: out[p][j] = Σ_rr L[r0+rr][J0+p]·y(r0+rr)[j] over the CTA's PF_RPC
// rows (two CTAs per PR-row chunk, each with its own block of partials); G = 256/cols
// thread groups take every G-th row, their sums added in group order.
template <typename T, int R>
__global__ void __launch_bounds__(256) k_wbwd_part_pf(const double* Y, const T* __restrict__ panel,
                                                      const DFront* __restrict__ fr, const int2* __restrict__ slots,
                                                      const int64_t* __restrict__ pre,
                                                      const int64_t* __restrict__ pre_part,
                                                      const int64_t* __restrict__ rows, int64_t S,
                                                      double* __restrict__ partial, int cols) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    const int pitch = pf_pitch<T>(cols);
    T* Lt = reinterpret_cast<T*>(sm);                               // [PF_RPC][pitch]
    double* yr = sm + PF_RPC * pitch * sizeof(T) / sizeof(double);  // [PF_RPC][R]
    double* red = yr + PF_RPC * R;                                  // [256][R]
    const int64_t b = blockIdx.x >> 1;
    const int2 sf = __ldg(slots + b);
    const int64_t i = sf.x, chunk = b - pre[i];
    const DFront f = fr[sf.y];
    const int64_t J0 = S * WS, J1 = min(J0 + WS, f.k);
    const int wb = (int)(J1 - J0);
    const int64_t r0 = J1 + chunk * PR + (blockIdx.x & 1) * PF_RPC;
    const int nr = (int)max((int64_t)0, min((int64_t)PF_RPC, f.m - r0));
    if (nr > 0) cp_async_tile<T>(Lt, pitch, panel + f.poff + r0 * f.ldp + J0, f.ldp, nr, wb, nr, cols, 256);
    cp_async_commit();
    pdl_wait();
    for (int idx = threadIdx.x; idx < PF_RPC * R; idx += 256) {
        const int rr = idx / R, j = idx - rr * R;
        double v = 0.0;
        if (rr < nr) {
            const int64_t r = r0 + rr;
            const int64_t q = r < f.k ? f.start + r : rows[f.rows_off + r - f.k];
            v = __ldcg(Y + q * R + j);
        }
        yr[idx] = v;
    }
    cp_async_wait<0>();
    __syncthreads();
    const int G = 256 / cols, g = threadIdx.x / cols, p = threadIdx.x - g * cols;
    if (g < G) {
        double acc[R][2];
#pragma unroll
        for (int j = 0; j < R; j++) acc[j][0] = acc[j][1] = 0.0;
        int rr = g;
        for (; rr + G < nr; rr += 2 * G) {
            const double l0 = Lt[rr * pitch + p], l1 = Lt[(rr + G) * pitch + p];
#pragma unroll
            for (int j = 0; j < R; j++) {
                acc[j][0] = fma(l0, yr[rr * R + j], acc[j][0]);
                acc[j][1] = fma(l1, yr[(rr + G) * R + j], acc[j][1]);
            }
        }
        if (rr < nr) {
            const double l0 = Lt[rr * pitch + p];
#pragma unroll
            for (int j = 0; j < R; j++) acc[j][0] = fma(l0, yr[rr * R + j], acc[j][0]);
        }
        if (G == 1) {
            if (p < wb) {
                double* out = partial + (2 * (pre_part[i] + chunk * wb) + (blockIdx.x & 1) * wb + p) * R;
#pragma unroll
                for (int j = 0; j < R; j++) out[j] = acc[j][0] + acc[j][1];
            }
            return;
        }
#pragma unroll
        for (int j = 0; j < R; j++) red[(g * cols + p) * R + j] = acc[j][0] + acc[j][1];
    }
    if (G == 1) return;
    __syncthreads();
    double* out = partial + (2 * (pre_part[i] + chunk * wb) + (blockIdx.x & 1) * wb) * R;
    for (int o = threadIdx.x; o < wb * R; o += 256) {
        double v = 0.0;
        for (int gg = 0; gg < G; gg++) v += red[gg * cols * R + o];
        out[o] = v;
    }
}

// z_B = y_B/D − Σ partial blocks (nc of them from block offset off), zero beyond the block.
template <int R>
__device__ __forceinline__ void wbwd_sum_partials(double* z, const double* Y, const double* __restrict__ d,
                                                  const double* partial, const DFront& f,
                                                  int64_t J0, int wb, int nbw, int64_t nc, int64_t off) {
    const int nout = wb * R;
    const double* pbase = partial + off * R;
    for (int o = threadIdx.x; o < nbw * NB * R; o += 256) {
        double v = 0.0;
        if (o < nout) {
            // blocks added in order; loaded 32 at a time so the loads overlap (the
            // top-of-tree steps have up to two hundred blocks)
            int64_t c = 0;
            for (; c + 32 <= nc; c += 32) {
                double t[32];
#pragma unroll
                for (int u = 0; u < 32; u++) t[u] = __ldcg(&pbase[(c + u) * nout + o]);
#pragma unroll
                for (int u = 0; u < 32; u++) v += t[u];
            }
            for (; c + 8 <= nc; c += 8) {
                double t[8];
#pragma unroll
                for (int u = 0; u < 8; u++) t[u] = __ldcg(&pbase[(c + u) * nout + o]);
#pragma unroll
                for (int u = 0; u < 8; u++) v += t[u];
            }
            for (; c < nc; c++) v += __ldcg(&pbase[c * nout + o]);
            v = __ldcg(Y + (f.start + J0) * R + o) / d[f.start + J0 + o / R] - v;
        }
        z[o] = v;
    }
}

// Backward diagonal block: one CTA (256 threads) per active front. z_B = y_B − Σ partials
// (chunks in order), then for sub-blocks bb from the last: y_bb = L_bb⁻ᵀ·z_bb and
// z_b2 −= L[bb, b2]ᵀ·y_bb for b2 < bb. Pieces in row-block order (1,0) (2,0) (2,1) (3,0)
// (3,1) (3,2); with four sub-blocks inverse blocks 1..3 are prefetched and block 0 is
// copied into the space of row block 3 once stage 3 is done.
template <int R>
__global__ void __launch_bounds__(256) k_wbwd_diag_pf(double* __restrict__ Y, const float* __restrict__ panel,
                                                      const double* __restrict__ linv, const DFront* __restrict__ fr,
                                                      const int64_t* __restrict__ order, int64_t fr_off,
                                                      const int64_t* __restrict__ pre,
                                                      const int64_t* __restrict__ pre_part, int64_t S,
                                                      const double* partial, int nbw_max,
                                                      const double* __restrict__ d) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    double* Li = sm;                                                       // [nli][NB][NB]
    float* Pr = reinterpret_cast<float*>(sm + pf_nli(nbw_max) * NB * NB);  // [npc][NB][NB]
    double* z = sm + pf_nli(nbw_max) * NB * NB + pf_npc(nbw_max) * NB * NB / 2;  // [WS][R]
    double* yb = z + WS * R;                                                     // [NB][R]
    double* red = yb + NB * R;                                                   // [4][NB][R]
    const int64_t i = blockIdx.x;
    const DFront f = fr[order[fr_off + i]];
    const int64_t J0 = S * WS;
    const int wb = (int)min((int64_t)WS, f.k - J0), nbw = (wb + NB - 1) / NB;
    const double* lsrc = linv + (f.blk_off + S * 4) * (int64_t)(NB * NB);
    // inverse block bb in slot bb − shift: with four sub-blocks, blocks 1..3 in slots 0..2
    // and block 0 later in the pieces of row block 3
    const int shift = nbw == 4 ? 1 : 0;
    cp_async_flat(Li, lsrc + shift * NB * NB, (nbw - shift) * NB * NB / 2, 256);
    for (int bb = 1; bb < nbw; bb++)
        for (int b2 = 0; b2 < bb; b2++) {
            const int pi = bb * (bb - 1) / 2 + b2;
            cp_async_tile<float>(Pr + pi * NB * NB, NB, panel + f.poff + (J0 + bb * NB) * f.ldp + J0 + b2 * NB, f.ldp,
                                 min(NB, wb - bb * NB), NB, NB, NB, 256);
        }
    cp_async_commit();
    pdl_wait();
    wbwd_sum_partials<R>(z, Y, d, partial, f, J0, wb, nbw, 2 * (pre[i + 1] - pre[i]), 2 * pre_part[i]);
    cp_async_wait<0>();
    for (int bb = nbw - 1; bb >= 0; bb--) {
        const int jbb = min(NB, wb - bb * NB);
        if (bb == 0 && nbw == 4) cp_async_wait<0>();
        __syncthreads();
        // y_bb = L_bb⁻ᵀ·z_bb: thread (p, g) sums rows q ∈ [16g, 16g+16) of column p
        const double* L = (nbw == 4 && bb == 0) ? reinterpret_cast<const double*>(Pr + 3 * NB * NB)
                                                : Li + (bb - shift) * NB * NB;
        {
            const int p = threadIdx.x & 63, g = threadIdx.x >> 6;
            double acc[R][2];
#pragma unroll
            for (int j = 0; j < R; j++) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll
            for (int q = 16 * g; q < 16 * g + 16; q += 2) {
                const double l0 = L[q * NB + p], l1 = L[(q + 1) * NB + p];
#pragma unroll
                for (int j = 0; j < R; j++) {
                    acc[j][0] = fma(l0, z[(bb * NB + q) * R + j], acc[j][0]);
                    acc[j][1] = fma(l1, z[(bb * NB + q + 1) * R + j], acc[j][1]);
                }
            }
#pragma unroll
            for (int j = 0; j < R; j++) red[(g * NB + p) * R + j] = acc[j][0] + acc[j][1];
        }
        __syncthreads();
        for (int o = threadIdx.x; o < NB * R; o += 256) {
            const double v = red[o] + red[NB * R + o] + red[2 * NB * R + o] + red[3 * NB * R + o];
            yb[o] = v;
            if (o < jbb * R) Y[(f.start + J0 + bb * NB) * R + o] = v;
        }
        if (bb == 0) break;
        __syncthreads();
        // z_b2 −= L[bb, b2]ᵀ·y_bb, one thread per column of row block bb
        if (threadIdx.x < bb * NB) {
            const int b2 = threadIdx.x >> 6, c = threadIdx.x & 63;
            const float* T = Pr + (bb * (bb - 1) / 2 + b2) * NB * NB;
            double acc[R][4];
#pragma unroll
            for (int j = 0; j < R; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0;
#pragma unroll 4
            for (int q = 0; q < NB; q += 4) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const double l = T[(q + u) * NB + c];
#pragma unroll
                    for (int j = 0; j < R; j++) acc[j][u] = fma(l, yb[(q + u) * R + j], acc[j][u]);
                }
            }
#pragma unroll
            for (int j = 0; j < R; j++) z[(b2 * NB + c) * R + j] -= (acc[j][0] + acc[j][1]) + (acc[j][2] + acc[j][3]);
        }
        if (bb == 3) {
            __syncthreads();  // row block 3's pieces are read: inverse block 0 goes there
            cp_async_flat(Pr + 3 * NB * NB, lsrc, NB * NB / 2, 256);
            cp_async_commit();
        }
    }
}

// The diagonal kernels of an FP64 factor: inverse blocks and pieces are 32 KB tiles, taken in
// the order of use (forward: inverse b, then the pieces (b2, b) below it; backward: inverse
// bb, then the pieces (bb, b2) left of it) through PD_SLOTS slots. A block of up to three
// sub-blocks is prefetched whole before the wait for the vectors; of a full block the first
// six tiles are, and the last four take the first slots when stage 0 is done with them.
// A step is bound by the latency of its chain of launches and barriers, not by the factor's
// bytes: with these kernels (launched as programmatic dependents) and the solve chains instead
// of the plain step kernels, a refined-solve call with the FP64 factor of the 33³ cube went
// from 3.72 to 1.79 ms (now 1.55), of the 45³ cube from 6.25 to 3.26 ms, of a 410-equation plate
// from 0.224 to 0.181 ms (now 0.10).
template <bool FWD>
__device__ __forceinline__ void pd_issue(double* sm, int tile, const double* panel, const DFront& f,
                                         const double* lsrc, int64_t J0, int wb, int nbw) {
    double* dst = sm + (tile % PD_SLOTS) * NB * NB;
    int st = 0, i = tile;  // stage st, the i-th tile of it
    while (i > nbw - 1 - st) {
        i -= nbw - st;
        st++;
    }
    const int b = FWD ? st : nbw - 1 - st;
    if (i == 0) {
        cp_async_flat(dst, lsrc + b * NB * NB, NB * NB / 2, 256);
    } else {
        const int rb = FWD ? b + i : b, cb = FWD ? b : i - 1;
        cp_async_tile<double>(dst, NB, panel + f.poff + (J0 + rb * NB) * f.ldp + J0 + cb * NB, f.ldp,
                              min(NB, wb - rb * NB), NB, NB, NB, 256);
    }
}

template <int R>
__global__ void __launch_bounds__(256) k_wfwd_diag_pd(const double* X, double* __restrict__ Y,
                                                      const double* __restrict__ panel, const double* __restrict__ linv,
                                                      const DFront* __restrict__ fr, const int64_t* __restrict__ order,
                                                      int64_t fr_off, int64_t S, int nbw_max,
                                                      const double* V, const int32_t* __restrict__ imap) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    double* xB = sm + pd_slots(nbw_max) * NB * NB;  // [WS][R]
    double* yb = xB + WS * R;                       // [NB][R]
    const DFront f = fr[order[fr_off + blockIdx.x]];
    const int64_t J0 = S * WS;
    const int wb = (int)min((int64_t)WS, f.k - J0), nbw = (wb + NB - 1) / NB;
    const double* lsrc = linv + (f.blk_off + S * 4) * (int64_t)(NB * NB);
    const int ntile = nbw + pf_npc(nbw);
    for (int i = 0; i < min(ntile, PD_SLOTS); i++) pd_issue<true>(sm, i, panel, f, lsrc, J0, wb, nbw);
    cp_async_commit();
    pdl_wait();
    const double* xs = X + (f.start + J0) * R;
    if (threadIdx.x < nbw * NB) {
        const int p = threadIdx.x;
#pragma unroll
        for (int r = 0; r < R; r++) {
            double x = p < wb ? __ldcg(xs + p * R + r) : 0.0;
            if (S == 0 && p < wb) x = kids_add(x, V, imap, f, p, R, r);
            xB[p * R + r] = x;
        }
    }
    cp_async_wait<0>();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sel = (lane >> 2) & 7;
    int t0 = 0;  // the stage's first tile
    for (int b = 0; b < nbw; b++) {
        const int jbb = min(NB, wb - b * NB);
        __syncthreads();
        {
            const double* L = sm + (t0 % PD_SLOTS) * NB * NB;
            double x0[R], x1[R], v[8][R], out[R];
#pragma unroll
            for (int j = 0; j < R; j++) {
                x0[j] = xB[(b * NB + lane) * R + j];
                x1[j] = xB[(b * NB + lane + 32) * R + j];
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const double l0 = L[(8 * warp + i) * NB + lane], l1 = L[(8 * warp + i) * NB + lane + 32];
#pragma unroll
                for (int j = 0; j < R; j++) v[i][j] = fma(l0, x0[j], l1 * x1[j]);
            }
            warp_sum8<R>(v, out);
            if ((lane & 3) == 0) {
                const int p = 8 * warp + sel;
#pragma unroll
                for (int j = 0; j < R; j++) {
                    yb[p * R + j] = out[j];
                    if (p < jbb) Y[(f.start + J0 + b * NB + p) * R + j] = out[j];
                }
            }
        }
        if (b == 1 && nbw == 4) cp_async_wait<0>();  // the last four tiles
        __syncthreads();
        if (b + 1 < nbw) {
            double y0[R], y1[R];
#pragma unroll
            for (int j = 0; j < R; j++) {
                y0[j] = yb[lane * R + j];
                y1[j] = yb[(lane + 32) * R + j];
            }
            const int ngrp = (nbw - 1 - b) * NB / 8;
            for (int g = warp; g < ngrp; g += 8) {
                const double* Lp = sm + ((t0 + 1 + g / 8) % PD_SLOTS) * NB * NB;
                double v[8][R], out[R];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const double* row = Lp + (8 * (g & 7) + i) * NB;
                    const double l0 = row[lane], l1 = row[lane + 32];
#pragma unroll
                    for (int j = 0; j < R; j++) v[i][j] = fma(l0, y0[j], l1 * y1[j]);
                }
                warp_sum8<R>(v, out);
                if ((lane & 3) == 0) {
#pragma unroll
                    for (int j = 0; j < R; j++) xB[((b + 1) * NB + 8 * g + sel) * R + j] -= out[j];
                }
            }
            if (b == 0 && nbw == 4) {
                __syncthreads();  // stage 0's four tiles are read
                for (int i = PD_SLOTS; i < ntile; i++) pd_issue<true>(sm, i, panel, f, lsrc, J0, wb, nbw);
                cp_async_commit();
            }
        }
        t0 += nbw - b;
    }
}

template <int R>
__global__ void __launch_bounds__(256) k_wbwd_diag_pd(double* __restrict__ Y, const double* __restrict__ panel,
                                                      const double* __restrict__ linv, const DFront* __restrict__ fr,
                                                      const int64_t* __restrict__ order, int64_t fr_off,
                                                      const int64_t* __restrict__ pre,
                                                      const int64_t* __restrict__ pre_part, int64_t S,
                                                      const double* partial, int nbw_max,
                                                      const double* __restrict__ d) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    double* z = sm + pd_slots(nbw_max) * NB * NB;  // [WS][R]
    double* yb = z + WS * R;                       // [NB][R]
    double* red = yb + NB * R;                     // [4][NB][R]
    const int64_t i = blockIdx.x;
    const DFront f = fr[order[fr_off + i]];
    const int64_t J0 = S * WS;
    const int wb = (int)min((int64_t)WS, f.k - J0), nbw = (wb + NB - 1) / NB;
    const double* lsrc = linv + (f.blk_off + S * 4) * (int64_t)(NB * NB);
    const int ntile = nbw + pf_npc(nbw);
    for (int t = 0; t < min(ntile, PD_SLOTS); t++) pd_issue<false>(sm, t, panel, f, lsrc, J0, wb, nbw);
    cp_async_commit();
    pdl_wait();
    wbwd_sum_partials<R>(z, Y, d, partial, f, J0, wb, nbw, 2 * (pre[i + 1] - pre[i]), 2 * pre_part[i]);
    cp_async_wait<0>();
    int t0 = 0;  // the stage's first tile
    for (int bb = nbw - 1; bb >= 0; bb--) {
        const int jbb = min(NB, wb - bb * NB);
        __syncthreads();
        // y_bb = L_bb⁻ᵀ·z_bb: thread (p, g) sums rows q ∈ [16g, 16g+16) of column p
        const double* L = sm + (t0 % PD_SLOTS) * NB * NB;
        {
            const int p = threadIdx.x & 63, g = threadIdx.x >> 6;
            double acc[R][2];
#pragma unroll
            for (int j = 0; j < R; j++) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll
            for (int q = 16 * g; q < 16 * g + 16; q += 2) {
                const double l0 = L[q * NB + p], l1 = L[(q + 1) * NB + p];
#pragma unroll
                for (int j = 0; j < R; j++) {
                    acc[j][0] = fma(l0, z[(bb * NB + q) * R + j], acc[j][0]);
                    acc[j][1] = fma(l1, z[(bb * NB + q + 1) * R + j], acc[j][1]);
                }
            }
#pragma unroll
            for (int j = 0; j < R; j++) red[(g * NB + p) * R + j] = acc[j][0] + acc[j][1];
        }
        __syncthreads();
        for (int o = threadIdx.x; o < NB * R; o += 256) {
            const double v = red[o] + red[NB * R + o] + red[2 * NB * R + o] + red[3 * NB * R + o];
            yb[o] = v;
            if (o < jbb * R) Y[(f.start + J0 + bb * NB) * R + o] = v;
        }
        if (bb == 0) break;
        if (bb == 2 && nbw == 4) cp_async_wait<0>();  // the last four tiles
        __syncthreads();
        // z_b2 −= L[bb, b2]ᵀ·y_bb, one thread per column of row block bb
        if (threadIdx.x < bb * NB) {
            const int b2 = threadIdx.x >> 6, c = threadIdx.x & 63;
            const double* T = sm + ((t0 + 1 + b2) % PD_SLOTS) * NB * NB;
            double acc[R][4];
#pragma unroll
            for (int j = 0; j < R; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0;
#pragma unroll 4
            for (int q = 0; q < NB; q += 4) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const double l = T[(q + u) * NB + c];
#pragma unroll
                    for (int j = 0; j < R; j++) acc[j][u] = fma(l, yb[(q + u) * R + j], acc[j][u]);
                }
            }
#pragma unroll
            for (int j = 0; j < R; j++) z[(b2 * NB + c) * R + j] -= (acc[j][0] + acc[j][1]) + (acc[j][2] + acc[j][3]);
        }
        if (bb == 3) {
            __syncthreads();  // stage 0's four tiles are read
            for (int t = PD_SLOTS; t < ntile; t++) pd_issue<false>(sm, t, panel, f, lsrc, J0, wb, nbw);
            cp_async_commit();
        }
        t0 += bb + 1;
    }
}

// ---------------------------------------------------------------------------
// Step kernels for 5 to 32 right-hand sides (a block of load cases, the subspace iteration of
// an eigen solver) on the FP64 tensor-core path (m8n8k4). The diagonal kernels take one front
// and eight right-hand sides per CTA: warp w owns rows (columns backward) 8w ... of each
// sub-block, the inverse blocks and panel pieces stream through MM_SLOTS slots in the order of
// use with one barrier per tile. The rows and partial kernels take all right-hand sides of a
// block (NT groups of eight), so that the factor is read once. Vectors stand in rows of
// 8·NT + 4 doubles: a fragment load (four rows, eight columns) meets every bank once per
// half-warp. They are bound by the latency of a step's launches and tiles (the hex20 20³ cube
// with 32 right-hand sides: 0.5 GB of factor and 16 GFLOP per sweep); with CUDA-core products,
// a warp per 256 rows for the children's vectors and one CTA per 256 pivots a refined solve of
// it (four sweeps) took 47.3 ms, now 11.7 ms; the FP64 solve of 160 batched plates with 8
// right-hand sides went from 3.25 to 1.16 ms.
// ---------------------------------------------------------------------------
constexpr int MM_SLOTS = 5;
constexpr int MM_P = NB + 4;       // tile pitch (elements): conflict-free row fragments
constexpr int MM_TILE = NB * MM_P; // doubles per slot
constexpr int MM_V = 12;           // pitch of a group's vector rows
constexpr int MM_ROWS = 64;        // rows of a rows CTA
// rows of a stage of the partial-sum kernel (two stages, PR rows per CTA), and its tile pitch
template <typename T>
constexpr int MM_PST = 256 / (int)sizeof(T);
template <typename T>
__host__ __device__ inline int mm_part_pitch(int cols) { return cols + (sizeof(T) == 4 ? 8 : 4); }
__host__ __device__ inline int mm_slots(int nbw) { return nbw + pf_npc(nbw) < MM_SLOTS ? nbw + pf_npc(nbw) : MM_SLOTS; }
inline size_t mm_diag_smem(int nbw) {
    return ((size_t)mm_slots(nbw) * MM_TILE + (size_t)(nbw * NB + NB) * MM_V) * sizeof(double);
}
template <typename T>
size_t mm_rows_smem(int cols, int nt) {
    return (size_t)MM_ROWS * (cols + 4) * sizeof(T) + (size_t)cols * (8 * nt + 4) * sizeof(double);
}
template <typename T>
size_t mm_part_smem(int cols, int nt) {
    return (size_t)2 * MM_PST<T> * mm_part_pitch<T>(cols) * sizeof(T) + (size_t)PR * (8 * nt + 4) * sizeof(double);
}

// The tile-th tile of a diagonal block into its slot (nothing past the last): the used part of
// inverse block b (its first jb rows and columns, rounded up to eight) or of panel piece
// (rb, cb), rows padded with zeros to eight. A tile counts as one commit group either way.
template <typename T, bool FWD>
__device__ __forceinline__ void mm_issue(double* sm, int tile, int ntile, const T* panel, const DFront& f,
                                         const double* lsrc, int64_t J0, int wb, int nbw) {
    if (tile < ntile) {
        double* dst = sm + (tile % MM_SLOTS) * MM_TILE;
        int st = 0, i = tile;  // stage st, the i-th tile of it
        while (i > nbw - 1 - st) {
            i -= nbw - st;
            st++;
        }
        const int b = FWD ? st : nbw - 1 - st;
        if (i == 0) {
            const int jr = (min(NB, wb - b * NB) + 7) & ~7;
            cp_async_tile<double>(dst, MM_P, lsrc + b * NB * NB, NB, jr, jr, jr, jr, 256);
        } else {
            const int rb = FWD ? b + i : b, cb = FWD ? b : i - 1, nr = min(NB, wb - rb * NB);
            cp_async_tile<T>(reinterpret_cast<T*>(dst), MM_P, panel + f.poff + (J0 + rb * NB) * f.ldp + J0 + cb * NB,
                             f.ldp, nr, NB, (nr + 7) & ~7, NB, 256);
        }
    }
    cp_async_commit();
}

template <typename T>
__global__ void __launch_bounds__(256) k_mm_fwd_diag(const double* X, double* __restrict__ Y,
                                                     const double* V, const T* __restrict__ panel,
                                                     const double* __restrict__ linv, const DFront* __restrict__ fr,
                                                     const int64_t* __restrict__ order, int64_t fr_off, int64_t S,
                                                     int nrhs, int nbw_max, const int32_t* __restrict__ imap) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    double* xB = sm + mm_slots(nbw_max) * MM_TILE;  // [nbw·NB][MM_V]
    double* yb = xB + nbw_max * NB * MM_V;          // [NB][MM_V]
    const DFront f = fr[order[fr_off + blockIdx.x]];
    const int j0 = blockIdx.y * 8, rc = min(8, nrhs - j0);
    const int64_t J0 = S * WS;
    const int wb = (int)min((int64_t)WS, f.k - J0), nbw = (wb + NB - 1) / NB;
    const double* lsrc = linv + (f.blk_off + S * 4) * (int64_t)(NB * NB);
    const int ntile = nbw + pf_npc(nbw);
    for (int i = 0; i < MM_SLOTS - 1; i++) mm_issue<T, true>(sm, i, ntile, panel, f, lsrc, J0, wb, nbw);
    pdl_wait();
    for (int e = threadIdx.x; e < nbw * NB * 8; e += 256) {
        const int p = e >> 3, n = e & 7;
        double x = 0.0;
        if (p < wb && n < rc) {
            x = __ldcg(X + (f.start + J0 + p) * nrhs + j0 + n);
            if (S == 0) x = kids_add(x, V, imap, f, p, nrhs, j0 + n);
        }
        xB[p * MM_V + n] = x;
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    int i = 0;
    for (int b = 0; b < nbw; b++) {
        const int jb = min(NB, wb - b * NB), jr = (jb + 7) & ~7;
        for (int b2 = b; b2 < nbw; b2++, i++) {
            cp_async_wait<MM_SLOTS - 2>();
            __syncthreads();  // tile i and the last stage's vectors visible; tile i − 1 is read
            mm_issue<T, true>(sm, i + MM_SLOTS - 1, ntile, panel, f, lsrc, J0, wb, nbw);
            const double* tile = sm + (i % MM_SLOTS) * MM_TILE;
            double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};
            if (b2 == b) {
                // y_b = L_bb⁻¹·x_b: rows 8w ... of the lower triangle
                if (8 * w >= jr) continue;
                const double* A = tile + (8 * w + g) * MM_P + q;
                const double* B = xB + (b * NB + q) * MM_V + g;
                for (int k = 0; k < 8 * w + 8; k += 8) {
                    dmma_884(a0[0], a0[1], A[k], B[k * MM_V]);
                    dmma_884(a1[0], a1[1], A[k + 4], B[(k + 4) * MM_V]);
                }
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int p = 8 * w + g, n = 2 * q + e;
                    const double y = p < jb ? a0[e] + a1[e] : 0.0;
                    yb[p * MM_V + n] = y;
                    if (p < jb && n < rc) Y[(f.start + J0 + b * NB + p) * nrhs + j0 + n] = y;
                }
            } else {
                // x_b2 −= L[b2, b]·y_b (b is a full sub-block)
                if (8 * w >= min(NB, wb - b2 * NB)) continue;
                const T* A = reinterpret_cast<const T*>(tile) + (8 * w + g) * MM_P + q;
                const double* B = yb + q * MM_V + g;
#pragma unroll
                for (int k = 0; k < NB; k += 8) {
                    dmma_884(a0[0], a0[1], (double)A[k], B[k * MM_V]);
                    dmma_884(a1[0], a1[1], (double)A[k + 4], B[(k + 4) * MM_V]);
                }
                double* x = xB + (b2 * NB + 8 * w + g) * MM_V + 2 * q;
                x[0] -= a0[0] + a1[0];
                x[1] -= a0[1] + a1[1];
            }
        }
    }
}

// Rows below a wide block: X (pivot rows) or V (later rows) −= L[r, J0:J1]·Y_B, MM_ROWS rows per
// CTA (two CTAs per PR-row chunk), warp w rows 8w ....
template <typename T, int NT>
__global__ void __launch_bounds__(256) k_mm_fwd_rows(double* __restrict__ X, double* __restrict__ V,
                                                     const double* Y, const T* __restrict__ panel,
                                                     const DFront* __restrict__ fr, const int2* __restrict__ slots,
                                                     const int64_t* __restrict__ pre,
                                                     int64_t S, int nrhs, int cols, const int32_t* __restrict__ imap) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    constexpr int VP = 8 * NT + 4;
    const int pitch = cols + 4;
    double* yB = sm;                                 // [cols][VP]
    T* Lt = reinterpret_cast<T*>(sm + cols * VP);    // [MM_ROWS][pitch]
    const int64_t b = blockIdx.x >> 1;
    const int2 sf = __ldg(slots + b);
    const int64_t i = sf.x, chunk = b - pre[i];
    const DFront f = fr[sf.y];
    const int64_t J0 = S * WS, J1 = min(J0 + WS, f.k);
    const int wb = (int)(J1 - J0);
    const int64_t r0 = J1 + chunk * PR + (blockIdx.x & 1) * MM_ROWS;
    const int nr = (int)max((int64_t)0, min((int64_t)MM_ROWS, f.m - r0));
    if (nr > 0) cp_async_tile<T>(Lt, pitch, panel + f.poff + r0 * f.ldp + J0, f.ldp, nr, wb, (nr + 7) & ~7, cols, 256);
    cp_async_commit();
    pdl_wait();
    if (nr == 0) return;
    const double* ys = Y + (f.start + J0) * nrhs;
    for (int e = threadIdx.x; e < cols * 8 * NT; e += 256) {
        const int p = e / (8 * NT), n = e % (8 * NT);
        yB[p * VP + n] = (p < wb && n < nrhs) ? __ldcg(ys + p * nrhs + n) : 0.0;
    }
    cp_async_wait<0>();
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    if (8 * w >= nr) return;
    double acc[2][NT][2] = {};
    const T* A = Lt + (8 * w + g) * pitch + q;
    const double* B = yB + q * VP + g;
    const int kend = (wb + 7) & ~7;
#pragma unroll 2
    for (int k = 0; k < kend; k += 8) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const double a = (double)A[k + 4 * h];
#pragma unroll
            for (int n = 0; n < NT; n++) dmma_884(acc[h][n][0], acc[h][n][1], a, B[(k + 4 * h) * VP + 8 * n]);
        }
    }
    const int rr = 8 * w + g;
    if (rr >= nr) return;
    const int64_t r = r0 + rr;
    double* tgt = r < f.k ? X + (f.start + r) * nrhs : V + (f.vuoff + r - f.k) * nrhs;
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int j = 8 * n + 2 * q + e;
            if (j >= nrhs) continue;
            double x = (S > 0 || r < f.k) ? __ldcg(tgt + j) : 0.0;
            if (S == 0) x = kids_add(x, V, imap, f, r, nrhs, j);
            tgt[j] = x - (acc[0][n][e] + acc[1][n][e]);
        }
}

// Backward partial sums: out[p][j] = Σ_rr L[r0+rr][J0+p]·y(r0+rr)[j] over a chunk's PR rows, one
// block of partials per chunk; warp w takes the columns 8w + 64i ....
template <typename T, int NT>
__global__ void __launch_bounds__(256) k_mm_bwd_part(const double* Y, const T* __restrict__ panel,
                                                     const DFront* __restrict__ fr, const int2* __restrict__ slots,
                                                     const int64_t* __restrict__ pre,
                                                     const int64_t* __restrict__ pre_part,
                                                     const int64_t* __restrict__ rows, int64_t S, int nrhs,
                                                     double* __restrict__ partial, int cols) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    constexpr int VP = 8 * NT + 4, ST = MM_PST<T>;
    const int pitch = mm_part_pitch<T>(cols);
    double* yr = sm;                            // [PR][VP]
    T* ring = reinterpret_cast<T*>(sm + PR * VP);  // [2][ST][pitch]
    const int2 sf = __ldg(slots + blockIdx.x);
    const int64_t i = sf.x, chunk = blockIdx.x - pre[i];
    const DFront f = fr[sf.y];
    const int64_t J0 = S * WS, J1 = min(J0 + WS, f.k);
    const int wb = (int)(J1 - J0);
    const int64_t r0 = J1 + chunk * PR;
    const int nr = (int)max((int64_t)0, min((int64_t)PR, f.m - r0)), nst = (nr + ST - 1) / ST;
    auto issue = [&](int h) {
        if (h < nst)
            cp_async_tile<T>(ring + (h & 1) * ST * pitch, pitch, panel + f.poff + (r0 + h * ST) * f.ldp + J0, f.ldp,
                             nr - h * ST, wb, min(ST, (nr - h * ST + 7) & ~7), cols, 256);
        cp_async_commit();
    };
    issue(0);
    issue(1);
    pdl_wait();
    for (int e = threadIdx.x; e < ((nr + 7) & ~7) * 8 * NT; e += 256) {
        const int rr = e / (8 * NT), n = e % (8 * NT);
        double v = 0.0;
        if (rr < nr && n < nrhs) {
            const int64_t r = r0 + rr;
            v = __ldcg(Y + (r < f.k ? f.start + r : rows[f.rows_off + r - f.k]) * nrhs + n);
        }
        yr[rr * VP + n] = v;
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    double acc[4][NT][2] = {};
    for (int h = 0; h < nst; h++) {
        cp_async_wait<1>();
        __syncthreads();
        const T* A = ring + (h & 1) * ST * pitch + q * pitch + 8 * w + g;
        const double* B = yr + (h * ST + q) * VP + g;
        const int kend = min(ST, (nr - h * ST + 7) & ~7);
#pragma unroll 2
        for (int k = 0; k < kend; k += 4) {
            double fb[NT];
#pragma unroll
            for (int n = 0; n < NT; n++) fb[n] = B[k * VP + 8 * n];
#pragma unroll
            for (int m = 0; m < 4; m++)
                if (64 * m + 8 * w < wb) {
                    const double a = (double)A[k * pitch + 64 * m];
#pragma unroll
                    for (int n = 0; n < NT; n++) dmma_884(acc[m][n][0], acc[m][n][1], a, fb[n]);
                }
        }
        if (h + 2 < nst) __syncthreads();  // stage h is read
        issue(h + 2);
    }
    double* out = partial + (pre_part[i] + chunk * wb) * nrhs;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const int p = 64 * m + 8 * w + g;
        if (p >= wb) continue;
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int j = 8 * n + 2 * q + e;
                if (j < nrhs) out[p * nrhs + j] = acc[m][n][e];
            }
    }
}

// Backward diagonal block: z_B = y_B/D − Σ partial blocks (chunks in order), then for sub-blocks
// bb from the last: y_bb = L_bb⁻ᵀ·z_bb and z_b2 −= L[bb, b2]ᵀ·y_bb for b2 < bb.
template <typename T>
__global__ void __launch_bounds__(256) k_mm_bwd_diag(double* __restrict__ Y, const T* __restrict__ panel,
                                                     const double* __restrict__ linv, const double* __restrict__ d,
                                                     const DFront* __restrict__ fr, const int64_t* __restrict__ order,
                                                     int64_t fr_off, const int64_t* __restrict__ pre,
                                                     const int64_t* __restrict__ pre_part, int64_t S, int nrhs,
                                                     int nbw_max, const double* partial) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) double sm[];
    double* z = sm + mm_slots(nbw_max) * MM_TILE;  // [nbw·NB][MM_V]
    double* yb = z + nbw_max * NB * MM_V;          // [NB][MM_V]
    const int64_t fi = blockIdx.x;
    const DFront f = fr[order[fr_off + fi]];
    const int j0 = blockIdx.y * 8, rc = min(8, nrhs - j0);
    const int64_t J0 = S * WS;
    const int wb = (int)min((int64_t)WS, f.k - J0), nbw = (wb + NB - 1) / NB;
    const double* lsrc = linv + (f.blk_off + S * 4) * (int64_t)(NB * NB);
    const int ntile = nbw + pf_npc(nbw);
    for (int i = 0; i < MM_SLOTS - 1; i++) mm_issue<T, false>(sm, i, ntile, panel, f, lsrc, J0, wb, nbw);
    pdl_wait();
    {
        const int64_t nc = pre[fi + 1] - pre[fi], bs = (int64_t)wb * nrhs;
        const double* pb = partial + pre_part[fi] * nrhs + j0;
        for (int e = threadIdx.x; e < nbw * NB * 8; e += 256) {
            const int p = e >> 3, n = e & 7;
            double v = 0.0;
            if (p < wb && n < rc) {
                const double* pe = pb + (int64_t)p * nrhs + n;
                int64_t c = 0;
                for (; c + 8 <= nc; c += 8) {
                    double t[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) t[u] = __ldcg(pe + (c + u) * bs);
#pragma unroll
                    for (int u = 0; u < 8; u++) v += t[u];
                }
                for (; c < nc; c++) v += __ldcg(pe + c * bs);
                v = __ldcg(Y + (f.start + J0 + p) * nrhs + j0 + n) / d[f.start + J0 + p] - v;
            }
            z[p * MM_V + n] = v;
        }
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    int i = 0;
    for (int bb = nbw - 1; bb >= 0; bb--) {
        const int jb = min(NB, wb - bb * NB), jr = (jb + 7) & ~7;
        for (int b2 = -1; b2 < bb; b2++, i++) {
            cp_async_wait<MM_SLOTS - 2>();
            __syncthreads();  // tile i and the last stage's vectors visible; tile i − 1 is read
            mm_issue<T, false>(sm, i + MM_SLOTS - 1, ntile, panel, f, lsrc, J0, wb, nbw);
            const double* tile = sm + (i % MM_SLOTS) * MM_TILE;
            double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};
            if (b2 < 0) {
                // y_bb = L_bb⁻ᵀ·z_bb: columns 8w ..., rows from 8w on
                if (8 * w >= jr) continue;
                const double* A = tile + q * MM_P + 8 * w + g;
                const double* B = z + (bb * NB + q) * MM_V + g;
                for (int k = 8 * w; k < jr; k += 8) {
                    dmma_884(a0[0], a0[1], A[k * MM_P], B[k * MM_V]);
                    dmma_884(a1[0], a1[1], A[(k + 4) * MM_P], B[(k + 4) * MM_V]);
                }
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int p = 8 * w + g, n = 2 * q + e;
                    const double y = p < jb ? a0[e] + a1[e] : 0.0;
                    yb[p * MM_V + n] = y;
                    if (p < jb && n < rc) Y[(f.start + J0 + bb * NB + p) * nrhs + j0 + n] = y;
                }
            } else {
                const T* A = reinterpret_cast<const T*>(tile) + q * MM_P + 8 * w + g;
                const double* B = yb + q * MM_V + g;
                for (int k = 0; k < jr; k += 8) {
                    dmma_884(a0[0], a0[1], (double)A[k * MM_P], B[k * MM_V]);
                    dmma_884(a1[0], a1[1], (double)A[(k + 4) * MM_P], B[(k + 4) * MM_V]);
                }
                double* zz = z + (b2 * NB + 8 * w + g) * MM_V + 2 * q;
                zz[0] -= a0[0] + a1[0];
                zz[1] -= a0[1] + a1[1];
            }
        }
    }
}

// caller column-major b (ncaller × nrhs) -> internal X (nsym × nrhs, row-major)
__global__ void k_gather_rhs(const double* __restrict__ b, double* __restrict__ X, const int64_t* __restrict__ eq,
                             int64_t ncaller, int nrhs) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ncaller * nrhs; e += (int64_t)gridDim.x * blockDim.x) {
        int64_t i = e % ncaller;
        int j = (int)(e / ncaller);
        int64_t q = eq[i];
        if (q >= 0) X[q * nrhs + j] = b[e];
    }
}

__global__ void k_scatter_rhs(double* __restrict__ b, const double* __restrict__ X, const int64_t* __restrict__ eq,
                              int64_t ncaller, int nrhs) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ncaller * nrhs; e += (int64_t)gridDim.x * blockDim.x) {
        int64_t i = e % ncaller;
        int j = (int)(e / ncaller);
        int64_t q = eq[i];
        if (q >= 0) b[e] = X[q * nrhs + j];
    }
}

__global__ void k_iso_divide(double* __restrict__ b, const int64_t* __restrict__ idx, const double* __restrict__ dv,
                             int64_t niso, int64_t ncaller, int nrhs) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < niso * nrhs; e += (int64_t)gridDim.x * blockDim.x) {
        int64_t i = e % niso;
        int j = (int)(e / niso);
        b[idx[i] + j * ncaller] /= dv[i];
    }
}

// ---------------------------------------------------------------------------
// refinement: the factored matrix as a full CSR, y = A x, residual norms
// ---------------------------------------------------------------------------
// both triangles of every assembled entry: entry 2i = (row, col) of segment i, entry
// 2i+1 its mirror (or a sentinel row n on the diagonal); value = (col << 32) | segment
__global__ void k_seg_entries(const DFront* __restrict__ fr, const int64_t* __restrict__ order,
                              const int64_t* __restrict__ front_seg, const int64_t* __restrict__ seg_dst,
                              const int64_t* __restrict__ rows, int64_t n, int32_t* __restrict__ key,
                              uint64_t* __restrict__ val) {
    const DFront f = fr[order[blockIdx.x]];
    for (int64_t i = front_seg[blockIdx.x] + threadIdx.x; i < front_seg[blockIdx.x + 1]; i += blockDim.x) {
        int64_t off = seg_dst[i] - f.poff;
        int64_t lr = off / f.ldp, lc = off - lr * f.ldp;
        int64_t qc = f.start + lc;
        int64_t qr = lr < f.k ? f.start + lr : rows[f.rows_off + lr - f.k];
        key[2 * i] = (int32_t)qr;
        val[2 * i] = ((uint64_t)qc << 32) | (uint64_t)i;
        key[2 * i + 1] = (int32_t)(qr != qc ? qc : n);
        val[2 * i + 1] = ((uint64_t)qr << 32) | (uint64_t)i;
    }
}

// counting sort of the entries by row (rows n are the discarded diagonal mirrors): the
// count per row, then (after the prefix sum of the counts) each entry at its row's
// offset plus a ticket; the order inside a row is fixed afterwards by sorting the row
__global__ void k_count_rows(const int32_t* __restrict__ key, int64_t cnt, unsigned long long* __restrict__ rc) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < cnt; e += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(rc + key[e], 1ull);
}

__global__ void k_place_rows(const int32_t* __restrict__ key, const uint64_t* __restrict__ val, int64_t cnt,
                             const int64_t* __restrict__ rp, int32_t* __restrict__ ticket,
                             uint64_t* __restrict__ out) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < cnt; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t r = key[e];
        out[rp[r] + atomicAdd(ticket + r, 1)] = val[e];
    }
}

// Columns and sources of the sorted entries in 32 bits. With direct_src the source is the index
// of the entry's only source value, otherwise its segment.
__global__ void k_split_entries(const uint64_t* __restrict__ val, int64_t cnt, int32_t* __restrict__ col,
                                uint32_t* __restrict__ from, const int64_t* __restrict__ direct_src) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < cnt; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t seg = (int64_t)(val[e] & 0xffffffffull);
        col[e] = (int32_t)(val[e] >> 32);
        from[e] = (uint32_t)(direct_src ? direct_src[seg] : seg);
    }
}

// Values of the CSR entries of a factorization (the sum of each entry's source values) and the
// rows' sums of |a|, one warp per row. Runs once per numeric phase.
__global__ void k_gather_rows(const int64_t* __restrict__ rp, const uint32_t* __restrict__ from,
                              const double* __restrict__ src, const int64_t* __restrict__ seg_ptr,
                              const int64_t* __restrict__ seg_src, bool direct, int64_t n, double* __restrict__ val,
                              double* __restrict__ rowsum) {
    const int lane = threadIdx.x & 31;
    for (int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; row < n;
         row += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t e1 = rp[row + 1];
        double a = 0.0;
        for (int64_t e = rp[row] + lane; e < e1; e += 32) {
            double s = 0.0;
            if (direct) {
                s = src[from[e]];
            } else if (seg_ptr) {
                const int64_t i = from[e];
                for (int64_t j = seg_ptr[i]; j < seg_ptr[i + 1]; j++) s += src[seg_src[j]];
            } else {
                s = src[seg_src[from[e]]];
            }
            val[e] = s;
            a += fabs(s);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0) rowsum[row] = a;
    }
}

// Y = A·X for one right-hand side, one warp per row: bound by the entries (12 bytes each)
__global__ void k_spmv(const int64_t* __restrict__ rp, const int32_t* __restrict__ col, const double* __restrict__ val,
                       const double* __restrict__ X, double* __restrict__ Y, int64_t n) {
    const int lane = threadIdx.x & 31;
    for (int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; row < n;
         row += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t e1 = rp[row + 1];
        double acc = 0.0;
        for (int64_t e = rp[row] + lane; e < e1; e += 32) acc = fma(val[e], X[col[e]], acc);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) Y[row] = acc;
    }
}

// Y = A·X for two or more right-hand sides (X, Y row-major, n × nrhs): groups of L lanes
// (L a power of two, the smallest >= min(nrhs, 32)) take one row each and lane j of a
// group right-hand side j (chunks of L for more), so an X row is read as L consecutive
// doubles and the group's lanes read each matrix entry at the same address (one access).
__global__ void k_spmm(const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                       const double* __restrict__ val, const double* __restrict__ X, double* __restrict__ Y,
                       int64_t n, int nrhs, int L) {
    const int sub = (int)(threadIdx.x & (L - 1));
    const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) / L;
    for (int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / L; row < n; row += ngroups) {
        const int64_t e0 = rp[row], e1 = rp[row + 1];
        for (int j = sub; j < nrhs; j += L) {
            const double* xj = X + j;
            double a0 = 0.0, a1 = 0.0;
            int64_t e = e0;
            for (; e + 1 < e1; e += 2) {
                a0 = fma(val[e], xj[(int64_t)col[e] * nrhs], a0);
                a1 = fma(val[e + 1], xj[(int64_t)col[e + 1] * nrhs], a1);
            }
            if (e < e1) a0 = fma(val[e], xj[(int64_t)col[e] * nrhs], a0);
            Y[row * nrhs + j] = a0 + a1;
        }
    }
}

// maxima of nonnegative doubles by their bits (a NaN stays the largest)
__device__ __forceinline__ double max_nonneg(double a, double b) {
    return __longlong_as_double(max(__double_as_longlong(a), __double_as_longlong(b)));
}
__device__ __forceinline__ void atomic_max_nonneg(double* a, double v) {
    atomicMax((unsigned long long*)a, (unsigned long long)__double_as_longlong(v));
}

// Per-system reductions of the refinement residual. The internal rows are split into
// segments (one per independent model of a batched factorization, else one), each
// reduced by blocks of SEG_ROWS rows: R = B − AX, and red[(g·nrhs + j)·5 + {0..4}] =
// {max|r|, max|x|, max|b|, Σr², Σb²} of segment g, right-hand side j. The block takes whole
// rows of right-hand sides at a time, so a thread keeps one right-hand side and its five
// values in registers; the threads of a right-hand side are then combined in halves.
// (Shared-memory atomics per entry, and 2048 rows per block, took 93 µs on the 33³ cube
// with one right-hand side and 338 µs on the hex20 20³ cube with 32; now 6 and 40 µs.)
constexpr int64_t SEG_ROWS = 512;

__global__ void __launch_bounds__(256) k_residual_seg(double* __restrict__ R, const double* __restrict__ AX,
                                                      const double* __restrict__ B, const double* __restrict__ X,
                                                      const int64_t* __restrict__ seg_off,
                                                      const int64_t* __restrict__ blk_pre, int64_t nseg, int nrhs,
                                                      double* __restrict__ red) {
    __shared__ double s[5][256];
    const int64_t g = find_slot2(blk_pre, nseg, blockIdx.x);
    const int64_t r0 = seg_off[g] + (blockIdx.x - blk_pre[g]) * SEG_ROWS;
    const int64_t r1 = min(seg_off[g + 1], r0 + SEG_ROWS);
    const int G = 256 / nrhs, T = G * nrhs, t = threadIdx.x;  // G rows at a time
    double mr = 0.0, mx = 0.0, mb = 0.0, sr = 0.0, sb = 0.0;
    if (t < T) {
#pragma unroll 4
        for (int64_t e = r0 * nrhs + t; e < r1 * nrhs; e += T) {
            const double b = B[e], x = X[e], r = b - AX[e];
            R[e] = r;
            mr = max_nonneg(mr, fabs(r));
            mx = max_nonneg(mx, fabs(x));
            mb = max_nonneg(mb, fabs(b));
            sr = fma(r, r, sr);
            sb = fma(b, b, sb);
        }
    }
    s[0][t] = mr;
    s[1][t] = mx;
    s[2][t] = mb;
    s[3][t] = sr;
    s[4][t] = sb;
    const int row = t / nrhs;
    for (int h = 128; h > 0; h >>= 1) {
        __syncthreads();
        if (row < h && row + h < G) {
            const int o = t + h * nrhs;
#pragma unroll
            for (int w = 0; w < 3; w++) s[w][t] = max_nonneg(s[w][t], s[w][o]);
            s[3][t] += s[3][o];
            s[4][t] += s[4][o];
        }
    }
    if (t < nrhs) {
        double* dst = &red[(g * nrhs + t) * 5];
#pragma unroll
        for (int w = 0; w < 3; w++) atomic_max_nonneg(dst + w, s[w][t]);
        atomicAdd(dst + 3, s[3][t]);
        atomicAdd(dst + 4, s[4][t]);
    }
}

// anorm[g] = max row sum of |A| over the rows of segment g
__global__ void k_seg_max(const double* __restrict__ rowsum, const int64_t* __restrict__ seg_off,
                          const int64_t* __restrict__ blk_pre, int64_t nseg, double* __restrict__ anorm) {
    int64_t g = find_slot2(blk_pre, nseg, blockIdx.x);
    int64_t r0 = seg_off[g] + (blockIdx.x - blk_pre[g]) * SEG_ROWS;
    int64_t r1 = min(seg_off[g + 1], r0 + SEG_ROWS);
    double m = 0.0;
    for (int64_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) m = fmax(m, rowsum[r]);
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomic_max_nonneg(&anorm[g], m);
}

// out = {max over (g, j) of the normwise backward error ‖r‖∞ / (‖A_g‖∞‖x‖∞ + ‖b‖∞),
//        max over (g, j) of ‖r‖₂ / ‖b‖₂}; one block of 256 threads
__global__ void k_seg_eta(const double* __restrict__ red, const double* __restrict__ anorm, int64_t nseg, int nrhs,
                          double* __restrict__ out) {
    __shared__ double se[8], sq[8];
    double e = 0.0, q = 0.0;
    for (int64_t i = threadIdx.x; i < nseg * nrhs; i += blockDim.x) {
        const double* v = red + i * 5;
        double den = anorm[i / nrhs] * v[1] + v[2];
        if (den > 0) e = fmax(e, v[0] / den);
        if (v[4] > 0) q = fmax(q, sqrt(v[3] / v[4]));
    }
    for (int o = 16; o > 0; o >>= 1) {
        e = fmax(e, __shfl_xor_sync(0xffffffffu, e, o));
        q = fmax(q, __shfl_xor_sync(0xffffffffu, q, o));
    }
    if ((threadIdx.x & 31) == 0) {
        se[threadIdx.x >> 5] = e;
        sq[threadIdx.x >> 5] = q;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
            e = fmax(e, se[w]);
            q = fmax(q, sq[w]);
        }
        out[0] = e;
        out[1] = q;
    }
}

__global__ void k_axpy(double* __restrict__ X, const double* __restrict__ D, int64_t cnt) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < cnt; e += (int64_t)gridDim.x * blockDim.x)
        X[e] += D[e];
}

__global__ void k_max_reduce(const double* __restrict__ v, int64_t n, double* __restrict__ out) {
    double m = 0.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        m = fmax(m, v[e]);
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomic_max_nonneg(out, m);
}

unsigned grid_for(int64_t work, int64_t per = 256) {
    int64_t g = (work + per - 1) / per;
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(g, 148 * 32));
}

// a kernel of a sweep, as a programmatic dependent of the previous one when pdl is set
template <typename... KArgs, typename... Args>
void launch_chained(bool pdl, void (*kern)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                    Args... args) {
    launch_pdl(pdl, kern, dim3(grid), dim3(block), smem, st, args...);
}

template <typename T, int R>
void wfwd_pf(const WStep& w, int nbw_max, int cols, double* X, double* Y, double* V, const T* panel,
             const double* linv, const DevPlan& dp, cudaStream_t st) {
    const int32_t* imap = dp.imap;
    if constexpr (sizeof(T) == 4)
        launch_chained(true, k_wfwd_diag_pf<R>, (unsigned)w.nact, 256, pf_diag_smem(nbw_max, R), st, X, Y, panel, linv,
                       dp.fronts, dp.level_order, w.fr_off, w.S, nbw_max, V, imap);
    else
        launch_chained(true, k_wfwd_diag_pd<R>, (unsigned)w.nact, 256, pd_diag_smem(nbw_max, R), st, X, Y, panel, linv,
                       dp.fronts, dp.level_order, w.fr_off, w.S, nbw_max, V, imap);
    launch_chained(true, k_wfwd_rows_pf<T, R>, (unsigned)(PR / PF_ROWS<T> * w.n_rows), PR, pf_rows_smem<T>(cols, R), st,
                   X, V, Y, panel, dp.fronts, dp.wrow_slot + w.row_off, dp.pre_wrows + w.pre_off, w.S, cols, imap);
}
template <typename T, int R>
void wbwd_pf(const WStep& w, int nbw_max, int cols, double* Y, const T* panel, const double* linv,
             const double* d, const DevPlan& dp, double* partial, cudaStream_t st) {
    launch_chained(true, k_wbwd_part_pf<T, R>, (unsigned)(2 * w.n_rows), 256, pf_part_smem<T>(cols, R), st, Y, panel,
                   dp.fronts, dp.wrow_slot + w.row_off, dp.pre_wrows + w.pre_off, dp.pre_wpart + w.pre_off, dp.rows, w.S,
                   partial, cols);
    if constexpr (sizeof(T) == 4)
        launch_chained(true, k_wbwd_diag_pf<R>, (unsigned)w.nact, 256, pf_diag_smem(nbw_max, R), st, Y, panel, linv,
                       dp.fronts, dp.level_order, w.fr_off, dp.pre_wrows + w.pre_off, dp.pre_wpart + w.pre_off, w.S,
                       partial, nbw_max, d);
    else
        launch_chained(true, k_wbwd_diag_pd<R>, (unsigned)w.nact, 256, pd_diag_smem(nbw_max, R), st, Y, panel, linv,
                       dp.fronts, dp.level_order, w.fr_off, dp.pre_wrows + w.pre_off, dp.pre_wpart + w.pre_off, w.S,
                       partial, nbw_max, d);
}


// five to 32 right-hand sides, NT groups of eight
template <typename T, int NT>
void wfwd_mm(const WStep& w, int nbw_max, int cols, double* X, double* Y, double* V, const T* panel,
             const double* linv, const DevPlan& dp, int nrhs, cudaStream_t st) {
    launch_pdl(true, k_mm_fwd_diag<T>, dim3((unsigned)w.nact, NT), dim3(256), mm_diag_smem(nbw_max), st,
               (const double*)X, Y, (const double*)V, panel, linv, (const DFront*)dp.fronts,
               (const int64_t*)dp.level_order, w.fr_off, w.S, nrhs, nbw_max, (const int32_t*)dp.imap);
    launch_pdl(true, k_mm_fwd_rows<T, NT>, dim3((unsigned)(2 * w.n_rows)), dim3(256), mm_rows_smem<T>(cols, NT), st, X,
               V, (const double*)Y, panel, (const DFront*)dp.fronts, (const int2*)(dp.wrow_slot + w.row_off),
               (const int64_t*)(dp.pre_wrows + w.pre_off), w.S, nrhs, cols, (const int32_t*)dp.imap);
}
template <typename T, int NT>
void wbwd_mm(const WStep& w, int nbw_max, int cols, double* Y, const T* panel, const double* linv, const double* d,
             const DevPlan& dp, double* partial, int nrhs, cudaStream_t st) {
    launch_pdl(true, k_mm_bwd_part<T, NT>, dim3((unsigned)w.n_rows), dim3(256), mm_part_smem<T>(cols, NT), st,
               (const double*)Y, panel, (const DFront*)dp.fronts, (const int2*)(dp.wrow_slot + w.row_off),
               (const int64_t*)(dp.pre_wrows + w.pre_off), (const int64_t*)(dp.pre_wpart + w.pre_off),
               (const int64_t*)dp.rows, w.S, nrhs, partial, cols);
    launch_pdl(true, k_mm_bwd_diag<T>, dim3((unsigned)w.nact, NT), dim3(256), mm_diag_smem(nbw_max), st, Y, panel, linv,
               d, (const DFront*)dp.fronts, (const int64_t*)dp.level_order, w.fr_off,
               (const int64_t*)(dp.pre_wrows + w.pre_off), (const int64_t*)(dp.pre_wpart + w.pre_off), w.S, nrhs,
               nbw_max, (const double*)partial);
}

// fn(std::integral_constant<int, n>) for n = 1 .. 4
template <typename F>
void by_count(int n, F&& fn) {
    if (n <= 1)
        fn(std::integral_constant<int, 1>());
    else if (n == 2)
        fn(std::integral_constant<int, 2>());
    else if (n == 3)
        fn(std::integral_constant<int, 3>());
    else
        fn(std::integral_constant<int, 4>());
}

}  // namespace

void launch_gather_rhs(const double* b, double* X, const int64_t* eq, int64_t ncaller, int64_t nsym, int64_t nrhs,
                       cudaStream_t st) {
    RFG_CUDA(cudaMemsetAsync(X, 0, std::max<int64_t>(nsym * nrhs, 1) * sizeof(double), st));
    if (ncaller * nrhs > 0) k_gather_rhs<<<grid_for(ncaller * nrhs), 256, 0, st>>>(b, X, eq, ncaller, (int)nrhs);
}

void launch_scatter_rhs(double* b, const double* X, const int64_t* eq, const int64_t* iso_idx, const double* iso_d,
                        int64_t niso, int64_t ncaller, int64_t nsym, int64_t nrhs, cudaStream_t st) {
    (void)nsym;
    if (X && ncaller * nrhs > 0) k_scatter_rhs<<<grid_for(ncaller * nrhs), 256, 0, st>>>(b, X, eq, ncaller, (int)nrhs);
    if (niso * nrhs > 0) k_iso_divide<<<grid_for(niso * nrhs), 256, 0, st>>>(b, iso_idx, iso_d, niso, ncaller, (int)nrhs);
}

ChainArgs Engine::chain_args() const {
    return ChainArgs{dp_.fronts, dp_.rows, dp_.imap, dp_.chain_blk, dp_.chain_colbase, linv_, chain_inv_, d_,
                     plan_.chain_blocks, chain_err_};
}

template <typename T>
int64_t Engine::forward_steps(int64_t l, double* X, double* Y, double* V, int nrhs, int* chain) {
    const Plan& P = plan_;
    const T* panel = (const T*)panel_;
    if (chain && P.level_chain[l]) {
        const int64_t i0 = P.chain_fwd_off[l], r0 = P.chain_rows_off[l], nr = P.chain_rows_off[l + 1] - r0;
        launch_chain_fwd(nrhs, P.chain_fwd_off[l + 1] - i0, (const double*)X, Y, (const double*)V, panel, chain_args(),
                         dp_.chain_fwd + 2 * i0, chain, chain + 8 * P.chain_blocks + 2 * l, stream_);
        launch_chain_rows(nrhs, nr, (const double*)Y, V, panel, chain_args(), dp_.chain_rows + 2 * r0, stream_);
        return nr > 0 ? 2 : 1;
    }
    int64_t launches = 0;
    for (int64_t wi = P.wstep_off[l]; wi < P.wstep_off[l + 1]; wi++) {
        const WStep& w = P.wsteps[wi];
        const int64_t wb_max = std::max<int64_t>(1, std::min<int64_t>(WS, P.level_maxk[l] - w.S * WS));
        const int nbw_max = (int)((wb_max + NB - 1) / NB), cols = pf_cols(wb_max);
        if (nrhs <= PF_MAXR)
            by_count(nrhs, [&](auto r) {
                wfwd_pf<T, decltype(r)::value>(w, nbw_max, cols, X, Y, V, panel, linv_, dp_, stream_);
            });
        else
            by_count((nrhs + 7) / 8, [&](auto nt) {
                wfwd_mm<T, decltype(nt)::value>(w, nbw_max, cols, X, Y, V, panel, linv_, dp_, nrhs, stream_);
            });
        launches += 2;
    }
    return launches;
}

template <typename T>
int64_t Engine::backward_steps(int64_t l, double* Y, double* V, int nrhs, double* partial, int* chain) {
    const Plan& P = plan_;
    const T* panel = (const T*)panel_;
    if (chain && P.level_chain[l]) {
        const int64_t i0 = P.chain_bwd_off[l], r0 = P.chain_rows_off[l], c0 = P.chain_cols_off[l];
        const int64_t nr = P.chain_rows_off[l + 1] - r0, nc = P.chain_cols_off[l + 1] - c0;
        launch_chain_cols(nrhs, nr, dp_.chain_rows + 2 * r0, nc, dp_.chain_cols + 2 * c0, (const double*)Y, V, partial,
                          panel, chain_args(), stream_);
        launch_chain_bwd(nrhs, P.chain_bwd_off[l + 1] - i0, Y, (const double*)partial, panel, chain_args(),
                         dp_.chain_bwd + 2 * i0, chain + 4 * P.chain_blocks, chain + 8 * P.chain_blocks + 2 * l + 1,
                         stream_);
        return nc > 0 ? 3 : 1;
    }
    int64_t launches = 0;
    for (int64_t wi = P.wstep_off[l + 1] - 1; wi >= P.wstep_off[l]; wi--) {
        const WStep& w = P.wsteps[wi];
        const int64_t wb_max = std::max<int64_t>(1, std::min<int64_t>(WS, P.level_maxk[l] - w.S * WS));
        const int nbw_max = (int)((wb_max + NB - 1) / NB), cols = pf_cols(wb_max);
        if (nrhs <= PF_MAXR)
            by_count(nrhs, [&](auto r) {
                wbwd_pf<T, decltype(r)::value>(w, nbw_max, cols, Y, panel, linv_, d_, dp_, partial, stream_);
            });
        else
            by_count((nrhs + 7) / 8, [&](auto nt) {
                wbwd_mm<T, decltype(nt)::value>(w, nbw_max, cols, Y, panel, linv_, d_, dp_, partial, nrhs, stream_);
            });
        launches += 2;
    }
    return launches;
}

template <typename T>
void Engine::solve_impl(double* X, int64_t nrhs_total) {
    const Plan& P = plan_;
    int64_t launches = 0;
    // X is row-major n × nrhs_total; sweeps of at most MAXR right-hand sides work on a
    // contiguous copy when nrhs_total > MAXR
    if (nrhs_total > MAXR) {
        double* tmp = (double*)nullptr;
        tmp = (decltype(tmp))dev_alloc(P.n * MAXR * sizeof(double), stream_);
        for (int64_t j0 = 0; j0 < nrhs_total; j0 += MAXR) {
            int64_t nr = std::min<int64_t>(MAXR, nrhs_total - j0);
            RFG_CUDA(cudaMemcpy2DAsync(tmp, nr * sizeof(double), X + j0, nrhs_total * sizeof(double), nr * sizeof(double),
                                       P.n, cudaMemcpyDeviceToDevice, stream_));
            solve_impl<T>(tmp, nr);
            RFG_CUDA(cudaMemcpy2DAsync(X + j0, nrhs_total * sizeof(double), tmp, nr * sizeof(double), nr * sizeof(double),
                                       P.n, cudaMemcpyDeviceToDevice, stream_));
        }
        dev_free(tmp, stream_);
        return;
    }
    int nrhs = (int)nrhs_total;
    int* chain = has_chain() ? counters_ : nullptr;
    if (chain) RFG_CUDA(cudaMemsetAsync(chain, 0, chain_flag_words(P) * sizeof(int), stream_));
    for (int64_t l = 0; l < P.nlevels; l++) launches += forward_steps<T>(l, X, ybuf_, vupd_, nrhs, chain);
    for (int64_t l = P.nlevels - 1; l >= 0; l--)
        launches += backward_steps<T>(l, ybuf_, vupd_, nrhs, partial_, chain);
    RFG_CUDA(cudaMemcpyAsync(X, ybuf_, P.n * nrhs * sizeof(double), cudaMemcpyDeviceToDevice, stream_));
    RFG_CUDA(cudaGetLastError());
    solve_launches += launches;
}

// Large dynamic shared-memory limits of the sweep kernels. Function attributes belong
// to the current device's context, so they are set once per device (a handle on a
// second device in the same process needs its own), under a lock because handles may
// be used from several host threads.
static void solve_set_attributes_current_device();

void solve_set_attributes() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    RFG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) throw CudaError("solve_set_attributes: device ordinal out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev]) return;
    solve_set_attributes_current_device();
    done[dev] = true;
}

static void solve_set_attributes_current_device() {
    auto attr = [](auto kern, size_t bytes) {
        RFG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    };
    auto pf_attrs = [&](auto r) {
        constexpr int R = decltype(r)::value;
        attr(k_wfwd_diag_pf<R>, pf_diag_smem(4, R));
        attr(k_wbwd_diag_pf<R>, pf_diag_smem(4, R));
        attr(k_wfwd_diag_pd<R>, pd_diag_smem(4, R));
        attr(k_wbwd_diag_pd<R>, pd_diag_smem(4, R));
        attr(k_wfwd_rows_pf<float, R>, pf_rows_smem<float>(WS, R));
        attr(k_wfwd_rows_pf<double, R>, pf_rows_smem<double>(WS, R));
        attr(k_wbwd_part_pf<float, R>, pf_part_smem<float>(WS, R));
        attr(k_wbwd_part_pf<double, R>, pf_part_smem<double>(WS, R));
        attr(k_mm_fwd_rows<float, R>, mm_rows_smem<float>(WS, R));
        attr(k_mm_fwd_rows<double, R>, mm_rows_smem<double>(WS, R));
        attr(k_mm_bwd_part<float, R>, mm_part_smem<float>(WS, R));
        attr(k_mm_bwd_part<double, R>, mm_part_smem<double>(WS, R));
    };
    attr(k_mm_fwd_diag<float>, mm_diag_smem(4));
    attr(k_mm_fwd_diag<double>, mm_diag_smem(4));
    attr(k_mm_bwd_diag<float>, mm_diag_smem(4));
    attr(k_mm_bwd_diag<double>, mm_diag_smem(4));
    for (int n = 1; n <= 4; n++) by_count(n, pf_attrs);
}

void Engine::solve_device(double* X, int64_t nrhs, bool allow_graph) {
    if (nrhs <= 0 || plan_.n == 0) return;
    solve_set_attributes();
    // the sweep's workspace must exist before a capture. It is sized for up to four
    // right-hand sides, or for MAXR once a wider solve comes: a handle solved with one
    // right-hand side does not take (and grow the memory pool by) 32 columns of it
    if (ws_nrhs_ < std::min<int64_t>(nrhs, MAXR)) {
        const int64_t w = nrhs <= 4 ? 4 : MAXR;
        if (ws_nrhs_ > 0) {
            // the captured sweeps refer to the narrower buffers
            RFG_CUDA(cudaStreamSynchronize(stream_));
            for (auto& g : solve_graphs_) RFG_CUDA(cudaGraphExecDestroy(g.exec));
            solve_graphs_.clear();
            solve_seen_.clear();
            for (void* q : {(void*)vupd_, (void*)partial_, (void*)ybuf_, (void*)counters_}) {
                allocs_.erase(std::find(allocs_.begin(), allocs_.end(), q));
                dev_free(q, stream_);
            }
        }
        vupd_ = (double*)dalloc(std::max<int64_t>(plan_.vu_rows * w, 1) * sizeof(double));
        partial_ = (double*)dalloc(std::max<int64_t>(partial_rows(has_chain()) * w, 1) * sizeof(double));
        ybuf_ = (double*)dalloc(std::max<int64_t>(plan_.n * w, 1) * sizeof(double));
        counters_ = (int*)dalloc(flag_words(has_chain()) * sizeof(int));
        ws_nrhs_ = w;
    }
    ensure_chain_inverse();
    if (use_graphs_ && nrhs <= MAXR) {
        cudaGraphExec_t ex = nullptr;
        for (auto& g : solve_graphs_)
            if (g.X == X && g.nrhs == nrhs) ex = g.exec;
        if (!ex) {
            // a sweep is captured the second time it runs on the same buffer and width; the
            // first run goes directly (a one-off solve does not pay for the capture)
            int64_t* uses = nullptr;
            for (auto& k : solve_seen_)
                if (k.first.first == X && k.first.second == nrhs) uses = &k.second;
            if (!uses) {
                solve_seen_.push_back({{X, nrhs}, 0});
                uses = &solve_seen_.back().second;
            }
            if (++*uses < 2 || !allow_graph) {
                if (prec_ == PREC_FP64)
                    solve_impl<double>(X, nrhs);
                else
                    solve_impl<float>(X, nrhs);
                return;
            }
        }
        if (!ex) {
            cudaGraph_t g;
            int64_t before = solve_launches;
            RFG_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
            if (prec_ == PREC_FP64)
                solve_impl<double>(X, nrhs);
            else
                solve_impl<float>(X, nrhs);
            RFG_CUDA(cudaStreamEndCapture(stream_, &g));
            RFG_CUDA(cudaGraphInstantiate(&ex, g, 0));
            RFG_CUDA(cudaGraphDestroy(g));
            solve_graphs_.push_back({X, nrhs, ex});
            solve_graph_launches_ = solve_launches - before;
            solve_launches = before;
        }
        RFG_CUDA(cudaGraphLaunch(ex, stream_));
        solve_launches += solve_graph_launches_;
        return;
    }
    if (prec_ == PREC_FP64)
        solve_impl<double>(X, nrhs);
    else
        solve_impl<float>(X, nrhs);
}

namespace {
int64_t round256(int64_t b) { return (b + 255) / 256 * 256; }
}  // namespace

int64_t Engine::partial_rows(bool chain) const {
    return std::max<int64_t>(2 * plan_.max_wpart, chain ? plan_.chain_colpart : 0);
}

int64_t Engine::flag_words(bool chain) const {
    return std::max<int64_t>(1, chain ? chain_flag_words(plan_) : 0);
}

// The chain blocks' inverses for the current FP32 factor: formed by the first sweep after each
// numeric phase (on the engine's stream, before that sweep's launches or graph).
void Engine::ensure_chain_inverse() {
    if (!chain_inv_ || chain_inv_at_ == factor_calls_) return;
    launch_chain_inverse(chain_inv_, (const float*)panel_, linv_, dp_.fronts, dp_.chain_blk, dp_.chain_bfront,
                         plan_.chain_blocks, stream_);
    solve_launches++;
    chain_inv_at_ = factor_calls_;
}

void Engine::chain_check() {
    if (!chain_err_) return;
    int v = 0;
    RFG_CUDA(cudaMemcpyAsync(&v, chain_err_, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    RFG_CUDA(cudaStreamSynchronize(stream_));
    if (v != 0) {
        RFG_CUDA(cudaMemsetAsync(chain_err_, 0, sizeof(int), stream_));
        throw CudaError("solve chain: a bounded wait gave up; the solutions since the last check are invalid");
    }
}

int64_t Engine::sweep_workspace_bytes(int64_t nrhs, bool chain) const {
    const Plan& P = plan_;
    return round256(std::max<int64_t>(P.n * nrhs, 1) * 8) + round256(std::max<int64_t>(P.vu_rows * nrhs, 1) * 8) +
           round256(std::max<int64_t>(partial_rows(chain) * nrhs, 1) * 8) + sweep_flag_bytes(chain);
}

int64_t Engine::sweep_flag_bytes(bool chain) const { return round256(flag_words(chain) * 4); }

Engine::SweepWorkspace Engine::carve_sweep_workspace(void* base, int64_t nrhs, bool chain) const {
    const Plan& P = plan_;
    char* p = (char*)base;
    SweepWorkspace ws;
    ws.y = (double*)p;
    p += round256(std::max<int64_t>(P.n * nrhs, 1) * 8);
    ws.v = (double*)p;
    p += round256(std::max<int64_t>(P.vu_rows * nrhs, 1) * 8);
    ws.partial = (double*)p;  // two blocks of partials per chunk on the prefetching path
    p += round256(std::max<int64_t>(partial_rows(chain) * nrhs, 1) * 8);
    ws.flags = (int*)p;
    ws.chain = chain;
    return ws;
}

// The launches of solve_impl, on the workspace ws instead of the engine's own buffers.
template <typename T>
void Engine::solve_sweep_impl(double* X, int64_t nrhs_total, const SweepWorkspace& ws) {
    const Plan& P = plan_;
    int nrhs = (int)nrhs_total;
    int* chain = ws.chain ? ws.flags : nullptr;
    if (chain) RFG_CUDA(cudaMemsetAsync(chain, 0, chain_flag_words(P) * sizeof(int), stream_));
    for (int64_t l = 0; l < P.nlevels; l++) forward_steps<T>(l, X, ws.y, ws.v, nrhs, chain);
    for (int64_t l = P.nlevels - 1; l >= 0; l--) backward_steps<T>(l, ws.y, ws.v, nrhs, ws.partial, chain);
    RFG_CUDA(cudaMemcpyAsync(X, ws.y, P.n * nrhs * sizeof(double), cudaMemcpyDeviceToDevice, stream_));
    RFG_CUDA(cudaGetLastError());
}

void Engine::solve_sweep_on(double* X, int64_t nrhs, const SweepWorkspace& ws) {
    if (nrhs <= 0 || plan_.n == 0) return;
    if (nrhs > MAXR) throw CudaError("solve_sweep_on: at most 32 right-hand sides per sweep");
    solve_set_attributes();
    if (ws.chain) ensure_chain_inverse();
    if (prec_ == PREC_FP64)
        solve_sweep_impl<double>(X, nrhs, ws);
    else
        solve_sweep_impl<float>(X, nrhs, ws);
}

void* noalloc_scratch() {
    static std::mutex mu;
    static void* addr[64] = {};
    int dev = 0;
    RFG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) throw CudaError("noalloc_scratch: device ordinal out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void* ptr = nullptr;
        cudaError_t rc = cudaGetSymbolAddress((void**)&ptr, g_noalloc_scratch);
        if (rc != cudaSuccess || !ptr)
            throw CudaError(std::string("cudaGetSymbolAddress of the static solve scratch failed: ") +
                            cudaGetErrorString(rc));
        addr[dev] = ptr;
    }
    return addr[dev];
}

void Engine::set_segments(const std::vector<int64_t>& off) {
    if (off.size() < 2 || off.front() != 0 || off.back() != plan_.n) throw CudaError("set_segments: bad offsets");
    // the norms kept from solve to solve, and the buffers, belong to the systems
    if (!seg_off_.empty()) throw CudaError("set_segments: the systems of a handle are set once, before its first refined solve");
    int64_t nseg = (int64_t)off.size() - 1;
    std::vector<int64_t> pre(nseg + 1, 0);
    for (int64_t g = 0; g < nseg; g++) {
        if (off[g + 1] < off[g]) throw CudaError("set_segments: offsets must not decrease");
        pre[g + 1] = pre[g] + (off[g + 1] - off[g] + SEG_ROWS - 1) / SEG_ROWS;
    }
    seg_off_ = off;
    seg_blocks_ = pre[nseg];
    d_seg_off_ = (int64_t*)dalloc((nseg + 1) * sizeof(int64_t));
    d_seg_blk_ = (int64_t*)dalloc((nseg + 1) * sizeof(int64_t));
    RFG_CUDA(cudaMemcpyAsync(d_seg_off_, off.data(), (nseg + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, stream_));
    RFG_CUDA(cudaMemcpyAsync(d_seg_blk_, pre.data(), (nseg + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, stream_));
    RFG_CUDA(cudaStreamSynchronize(stream_));
}

void Engine::build_matrix() {
    int64_t n = plan_.n, nseg = nseg_;
    if (nseg >= ((int64_t)1 << 32) || n >= ((int64_t)1 << 31)) throw CudaError("build_matrix: matrix too large");
    int64_t cnt = 2 * nseg;
    // the work buffers: the update arena when it is large enough (its update blocks are
    // dead once the numeric phase has run, and the next numeric phase rewrites them), so a
    // new handle's first solve allocates nothing of this size
    auto r256 = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t c1 = (size_t)std::max<int64_t>(cnt, 1);
    const size_t nr = (size_t)n + 2;  // rows 0..n (n: diagonal mirrors) and the total
    const size_t need = r256(c1 * 4) + 2 * r256(c1 * 8) + r256(nr * 8) + r256(nr * 4) +
                        r256((size_t)scan_tmp_elems((int64_t)nr) * 8);
    const size_t es = prec_ == PREC_FP64 ? sizeof(double) : sizeof(float);
    char* base = nullptr;
    const bool in_arena = (size_t)plan_.upd_elems * es >= need;
    base = in_arena ? (char*)upd_ : (char*)dev_alloc(need, stream_);
    char* p = base;
    int32_t* k0 = (int32_t*)p;
    p += r256(c1 * 4);
    uint64_t* v0 = (uint64_t*)p;
    p += r256(c1 * 8);
    uint64_t* v1 = (uint64_t*)p;
    p += r256(c1 * 8);
    int64_t* rp = (int64_t*)p;
    p += r256(nr * 8);
    int32_t* ticket = (int32_t*)p;
    p += r256(nr * 4);
    int64_t* stmp = (int64_t*)p;
    if (plan_.nfronts > 0)
        k_seg_entries<<<(unsigned)plan_.nfronts, 256, 0, stream_>>>(dp_.fronts, dp_.level_order, dp_.front_seg,
                                                                    dp_.seg_dst, dp_.rows, n, k0, v0);
    RFG_CUDA(cudaMemsetAsync(rp, 0, nr * 8, stream_));
    RFG_CUDA(cudaMemsetAsync(ticket, 0, nr * 4, stream_));
    if (cnt > 0) k_count_rows<<<grid_for(cnt), 256, 0, stream_>>>(k0, cnt, (unsigned long long*)rp);
    exclusive_scan_i64(rp, (int64_t)nr, stmp, stream_);
    if (cnt > 0) k_place_rows<<<grid_for(cnt), 256, 0, stream_>>>(k0, v0, cnt, rp, ticket, v1);
    // (column << 32 | segment) is distinct within a row: sorted rows do not depend on
    // the order in which the tickets were drawn
    sort_rows_u64(v1, rp, n, stream_);
    RFG_CUDA(cudaMemcpyAsync(a_rowptr_, rp, (n + 1) * sizeof(int64_t), cudaMemcpyDeviceToDevice, stream_));
    int64_t nnz = 0;
    RFG_CUDA(cudaMemcpyAsync(&nnz, rp + n, sizeof(int64_t), cudaMemcpyDeviceToHost, stream_));
    RFG_CUDA(cudaStreamSynchronize(stream_));
    a_nnz_ = nnz;
    // one source per entry and 32-bit indices: the values are gathered without the segments
    a_direct_ = !dp_.seg_ptr && nsrc_ <= ((int64_t)1 << 32);
    if (nnz > 0)
        k_split_entries<<<grid_for(nnz), 256, 0, stream_>>>(v1, nnz, a_col_, a_src_,
                                                            a_direct_ ? (const int64_t*)dp_.seg_src : nullptr);
    if (!in_arena) dev_free(base, stream_);
    RFG_CUDA(cudaStreamSynchronize(stream_));
    matrix_built_ = true;
}

void Engine::matvec(const double* X, double* Y, int64_t nrhs) {
    const int64_t n = plan_.n;
    if (nrhs <= 1) {
        k_spmv<<<grid_for(n * 32, 256), 256, 0, stream_>>>(a_rowptr_, a_col_, a_val_, X, Y, n);
        return;
    }
    int L = 1;
    while (L < nrhs && L < 32) L *= 2;
    k_spmm<<<grid_for(n * L, 256), 256, 0, stream_>>>(a_rowptr_, a_col_, a_val_, X, Y, n, (int)nrhs, L);
}

SolveStats Engine::solve_refined(double* X, const double* B, int64_t nrhs, double tol, int max_iter) {
    SolveStats st;
    int64_t n = plan_.n;
    if (n == 0 || nrhs == 0) return st;
    if (nrhs > MAXR) throw CudaError("solve_refined: at most 32 right-hand sides per call");
    HostTimer timer("solve_refined");
    // with RFG_HOST_TIMING set, each lap waits for the stream so that it times the device work
    auto lap = [&](const char* what) {
        if (!timer.on) return;
        RFG_CUDA(cudaStreamSynchronize(stream_));
        timer.lap(what);
    };
    if (!matrix_built_) build_matrix();
    lap("matrix");
    // the first refined solve of an engine runs its sweeps without capturing graphs
    const bool graphs = refined_calls_++ > 0;
    int64_t l0 = solve_launches;
    if (seg_off_.empty()) set_segments({0, n});
    const int64_t nseg = (int64_t)seg_off_.size() - 1;
    // red: 5 values per (segment, right-hand side), then anorm per segment, then ‖A‖∞
    // and the two maxima of k_seg_eta
    const int64_t nred = 5 * nseg * MAXR + nseg + 3;
    if (ref_nrhs_ < nrhs) {
        if (ref_r_) dev_free(ref_r_, stream_);
        if (ref_dx_) dev_free(ref_dx_, stream_);
        if (ref_red_) dev_free(ref_red_, stream_);
        ref_r_ = (double*)dev_alloc(n * MAXR * sizeof(double), stream_);
        ref_dx_ = (double*)dev_alloc(n * MAXR * sizeof(double), stream_);
        ref_red_ = (double*)dev_alloc(nred * sizeof(double), stream_);
        ref_nrhs_ = MAXR;
        a_val_at_ = -1;
    }
    double* seg_anorm = ref_red_ + 5 * nseg * MAXR;
    double* eta_out = seg_anorm + nseg + 1;
    if (a_val_at_ != factor_calls_) {
        // the matrix values of the current factorization and its norms: formed by the first
        // refined solve after each numeric phase
        RFG_CUDA(cudaMemsetAsync(seg_anorm, 0, (nseg + 3) * sizeof(double), stream_));
        k_gather_rows<<<grid_for(n * 32, 256), 256, 0, stream_>>>(a_rowptr_, a_src_, src_, dp_.seg_ptr, dp_.seg_src,
                                                                 a_direct_, n, a_val_, ref_dx_);
        k_max_reduce<<<grid_for(n), 256, 0, stream_>>>(ref_dx_, n, seg_anorm + nseg);
        if (seg_blocks_ > 0)
            k_seg_max<<<(unsigned)seg_blocks_, 256, 0, stream_>>>(ref_dx_, d_seg_off_, d_seg_blk_, nseg, seg_anorm);
        RFG_CUDA(cudaMemcpyAsync(&anorm_, seg_anorm + nseg, sizeof(double), cudaMemcpyDeviceToHost, stream_));
        a_val_at_ = factor_calls_;
    }
    if (X != B) RFG_CUDA(cudaMemcpyAsync(X, B, n * nrhs * sizeof(double), cudaMemcpyDeviceToDevice, stream_));
    lap("values, norms");
    solve_device(X, nrhs, graphs);
    lap("sweep");
    double eo[2] = {0.0, 0.0};
    for (int it = 0;; it++) {
        RFG_CUDA(cudaMemsetAsync(ref_red_, 0, 5 * nseg * nrhs * sizeof(double), stream_));
        matvec(X, ref_dx_, nrhs);
        if (seg_blocks_ > 0)
            k_residual_seg<<<(unsigned)seg_blocks_, 256, 0, stream_>>>(ref_r_, ref_dx_, B, X, d_seg_off_, d_seg_blk_,
                                                                      nseg, (int)nrhs, ref_red_);
        k_seg_eta<<<1, 256, 0, stream_>>>(ref_red_, seg_anorm, nseg, (int)nrhs, eta_out);
        solve_launches += 3;
        RFG_CUDA(cudaMemcpyAsync(eo, eta_out, 2 * sizeof(double), cudaMemcpyDeviceToHost, stream_));
        RFG_CUDA(cudaStreamSynchronize(stream_));
        st.backward_error = eo[0];
        st.rel_residual = eo[1];
        st.iterations = it;
        lap("residual");
        if (eo[0] <= tol || it >= max_iter) break;
        solve_device(ref_r_, nrhs, graphs);
        k_axpy<<<grid_for(n * nrhs), 256, 0, stream_>>>(X, ref_r_, n * nrhs);
        solve_launches += 1;
        lap("sweep");
    }
    chain_check();
    st.launches = solve_launches - l0;
    return st;
}

}  // namespace rfg
