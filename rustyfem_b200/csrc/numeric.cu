// Numeric phase of the multifrontal LDLᵀ on the GPU (sm_100a).
//
// Level by level (see plan.h), each level of the elimination tree is
//   1. assembled: the children's update matrices gathered into its fronts in child
//      order (k_assemble); before the first level the panels of all levels are
//      zeroed, the original entries stored (k_scatter) and the original diagonal
//      captured for the pivot test (k_capture_diag),
//   2. factored in steps of NB pivots over all fronts of the level at once:
//        k_pivot_block  one CTA per front: blocked LDLᵀ of the NB×NB diagonal
//                       block in shared memory (FP64), with the reference's
//                       positive definite rule (src/sparse.rs:528-531); the
//                       blocks' inverses, for the solves, all at the end
//                       (k_block_inverse);
//        k_panel        PNR rows below the block per CTA (FP64 tensor-core path):
//                       W = F·L⁻ᵀ, L = W·D⁻¹, plus the W and L operands of the Schur
//                       update in a scratch of NB-wide rows;
//        k_schur*       lower-triangular tiles of the trailing matrix,
//                       F −= W·Lᵀ (src/sparse.rs:559-573), written to the panel
//                       (pivot columns) or the update block (F22): in FP64 on the
//                       FP64 tensor-core path (mma.sync f64; k_schur_dmma64 for
//                       64-tiles, k_schur_dmma for the 128-tiles of large fronts),
//                       in the mixed path on tcgen05 (kernels_tc.cu) or, without
//                       tensor cores, on the CUDA cores (k_schur, k_schur_big).
// Storage T is double (FP64 path) or float (mixed path); pivot blocks are
// always factored in FP64 and the pivots D are kept in FP64.

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>

#include "engine.h"
#include "tc.cuh"
#include "tiles.cuh"

namespace rfg {

namespace {

template <typename T>
__global__ void k_scatter(T* __restrict__ panel, const double* __restrict__ src, const int64_t* __restrict__ dst,
                          const int64_t* __restrict__ seg_ptr, const int64_t* __restrict__ seg_src, int64_t lo,
                          int64_t hi) {
    pdl_wait();  // wait first: a dependent launched early may then read our inputs
    pdl_launch_dependents();
    for (int64_t i = lo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < hi; i += (int64_t)gridDim.x * blockDim.x) {
        double s;
        if (seg_ptr) {
            s = 0.0;
            for (int64_t j = seg_ptr[i]; j < seg_ptr[i + 1]; j++) s += src[seg_src[j]];
        } else {
            s = src[seg_src[i]];
        }
        panel[dst[i]] = (T)s;
    }
}

template <typename T>
__global__ void k_capture_diag(const T* panel, double* __restrict__ adiag, const DFront* __restrict__ fr,
                               const int64_t* __restrict__ order, int64_t lo) {
    pdl_wait();  // wait first: a dependent launched early may then read our inputs
    pdl_launch_dependents();
    const DFront f = fr[order[lo + blockIdx.x]];
    for (int64_t i = threadIdx.x; i < f.k; i += blockDim.x) adiag[f.start + i] = (double)__ldcg(panel + f.poff + i * f.ldp + i);
}

// Children's update matrices into the fronts of a level, by gathering: the lower triangle of a
// front is cut into XT × XT tiles (the update block's triangle alone for a front without
// children), one warp per tile and eight tiles per CTA, lane l takes column C0 + l of the
// tile's rows. imap gives the child row (or none) of each front row; the maps grow with the
// row, so a child's entry (x, y), y <= x, lies in the front's lower triangle too. An update-block
// entry is written once (child 0 + child 1, zeros where there is neither), a panel entry gets
// both children on top of the original entry, and only where one of them has something. The
// least traffic is each child entry read once and each update entry written once; what bounds
// the kernel is the latency of the rows' loads, so every lane first asks for one row's part of
// the children (the whole tile on its way into L2), six CTAs fit on an SM, a lane without a
// child column reads a zero at stride 0 instead of a predicate, and a tile that only one child
// reaches leaves the other out. (Zeroing, then one read-modify-write pass per child, took, with
// the original entries stored level by level, 14.5 ms of a 60³ mixed factorization, 8.7 ms of a
// 45³ FP64 one, 1.17 ms of 160 batched plates and 0.44 ms of a 9³ one; now 11.4, 5.8, 0.66 and
// 0.19 ms. Two columns per lane with four CTAs per SM were as fast at 60³ and slower below.)
static __device__ double g_zero = 0.0;

template <typename T, bool PANEL, bool K0, bool K1>
__device__ __forceinline__ void asm_rows(T* col, const T* p0, const T* p1, int s0, int s1, bool put, int cr, int ld,
                                         int nr, int32_t r0, int32_t r1) {
    constexpr int U = 4;
    for (int x0 = 0; x0 < nr; x0 += U) {
        T v0[U], v1[U], old[U];
        bool some[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            // rows past the tile have no child row (r0 = r1 = -1)
            const int32_t a0 = K0 ? __shfl_sync(0xffffffffu, r0, (x0 + u) & (XT - 1)) : -1;
            const int32_t a1 = K1 ? __shfl_sync(0xffffffffu, r1, (x0 + u) & (XT - 1)) : -1;
            some[u] = a0 >= 0 || a1 >= 0;
            v0[u] = K0 && a0 >= 0 ? p0[(int64_t)a0 * s0] : T(0);
            v1[u] = K1 && a1 >= 0 ? p1[(int64_t)a1 * s1] : T(0);
            if (PANEL) old[u] = put && some[u] ? col[(int64_t)(x0 + u) * ld] : T(0);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (put && (!PANEL || some[u]) && x0 + u >= cr && x0 + u < nr)
                col[(int64_t)(x0 + u) * ld] = PANEL ? (old[u] + v0[u]) + v1[u] : v0[u] + v1[u];
    }
}

// The part [lo, hi] of a child's row of this lane into L2, lo and hi over the warp's columns.
template <typename T>
__device__ __forceinline__ void asm_prefetch(const T* base, int64_t ldu, int32_t row, int32_t c) {
    const int lo = (int)__reduce_min_sync(0xffffffffu, (uint32_t)c), hi = __reduce_max_sync(0xffffffffu, c);
    if (row < 0) return;
    const char* p = reinterpret_cast<const char*>(base + row * ldu + lo);
    const char* e = reinterpret_cast<const char*>(base + row * ldu + hi);
    for (; p <= e; p += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

template <typename T>
__global__ void __launch_bounds__(256, 6) k_assemble(T* __restrict__ panel, T* __restrict__ upd,
                                                     const DFront* __restrict__ fr, const int64_t* __restrict__ order,
                                                     const int64_t* __restrict__ pre, int64_t nfronts,
                                                     const int32_t* __restrict__ imap, int64_t* __restrict__ status) {
    const int64_t i = find_slot_warp(pre, nfronts, blockIdx.x);
    const int64_t t = order[i], chunk = blockIdx.x - pre[i];
    const DFront f = fr[t];
    const bool kids = f.imap_off >= 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t base = kids ? 0 : f.k;  // first row and column of the tile grid
    const int64_t nt = (f.m - base + XT - 1) / XT, lt = chunk * 8 + warp;
    int64_t ti = (int64_t)((sqrt(8.0 * (double)lt + 1.0) - 1.0) * 0.5);
    while (ti * (ti + 1) / 2 > lt) ti--;
    while ((ti + 1) * (ti + 2) / 2 <= lt) ti++;
    const int64_t tj = lt - ti * (ti + 1) / 2;
    const int64_t R0 = base + ti * XT, R1 = min(f.m, R0 + XT), c = base + tj * XT + lane;
    const bool in = lt < nt * (nt + 1) / 2;
    // the children's rows of this lane's column and of the tile's rows (one per lane, handed
    // out by shuffles)
    int32_t c0 = -1, c1 = -1, r0 = -1, r1 = -1;
    DFront k0{}, k1{};
    if (kids && f.kid0 >= 0) k0 = fr[f.kid0];
    if (kids && f.kid1 >= 0) k1 = fr[f.kid1];
    if (kids && in && c < f.m) {
        c0 = imap[f.imap_off + c];
        c1 = imap[f.imap_off + f.m + c];
    }
    if (kids && in && R0 + lane < R1) {
        r0 = imap[f.imap_off + R0 + lane];
        r1 = imap[f.imap_off + f.m + R0 + lane];
    }
    pdl_wait();
    pdl_launch_dependents();
    if (kids && ((f.kid0 >= 0 && status[f.kid0] != -1) || (f.kid1 >= 0 && status[f.kid1] != -1))) {
        if (chunk == 0 && threadIdx.x == 0) status[t] = -2;  // an ancestor of a failed front
        return;
    }
    if (!in) return;
    const int nr = (int)(R1 - R0), cr = (int)min(c - R0, (int64_t)XT);  // this lane's rows start at cr
    const bool any0 = __any_sync(0xffffffffu, c0 >= 0) && __any_sync(0xffffffffu, r0 >= 0);
    const bool any1 = __any_sync(0xffffffffu, c1 >= 0) && __any_sync(0xffffffffu, r1 >= 0);
    if (any0) asm_prefetch(upd + k0.uoff, k0.ldu, r0, c0);
    if (any1) asm_prefetch(upd + k1.uoff, k1.ldu, r1, c1);
    const T* const zero = reinterpret_cast<const T*>(&g_zero);
    const T* const p0 = c0 >= 0 ? upd + k0.uoff + c0 : zero;
    const T* const p1 = c1 >= 0 ? upd + k1.uoff + c1 : zero;
    const int s0 = c0 >= 0 ? (int)k0.ldu : 0, s1 = c1 >= 0 ? (int)k1.ldu : 0;
    // the tile's columns in the panel, then those in the update block (a tile on the border
    // takes both passes)
    if (c - lane < f.k && (any0 || any1))
        asm_rows<T, true, true, true>(panel + f.poff + R0 * f.ldp + c, p0, p1, s0, s1,
                                      c < f.k && (c0 >= 0 || c1 >= 0), cr, (int)f.ldp, nr, r0, r1);
    if (c - lane + XT > f.k && R1 > f.k) {
        T* const col = upd + f.uoff + (R0 - f.k) * f.ldu + (c - f.k);
        const bool put = c >= f.k;
        if (any0 && any1)
            asm_rows<T, false, true, true>(col, p0, p1, s0, s1, put, cr, (int)f.ldu, nr, r0, r1);
        else if (any0)
            asm_rows<T, false, true, false>(col, p0, p1, s0, s1, put, cr, (int)f.ldu, nr, r0, r1);
        else if (any1)
            asm_rows<T, false, false, true>(col, p0, p1, s0, s1, put, cr, (int)f.ldu, nr, r0, r1);
        else
            asm_rows<T, false, false, false>(col, p0, p1, s0, s1, put, cr, (int)f.ldu, nr, r0, r1);
    }
}

// LDLᵀ of the NB×NB diagonal block [j0, j1) of each active front in FP64, one CTA of PBT
// threads per front. A launch is a chain of 64 dependent pivots, so the kernel is built around
// the length of that chain. The block is factored in sub-panels of PB = 8 pivots. Warps 0 and 1
// hold one row below the sub-panel's diagonal 8×8 block per lane, and every lane also holds the
// whole diagonal block and eliminates it for itself: from pivot to pivot there is no exchange,
// only the reciprocal and one multiply-add on registers. (One barrier of the two warps stands
// between their loads of the block and the store of its factor in its place.) The sub-panel's rank-8 update of the
// trailing block runs on the FP64 tensor-core path (two m8n8k4 products per 8×8 tile), first for
// the next sub-panel's columns, then, while the next sub-panel is eliminated, for the rest
// (warps 2 to 6); warp 7 tests the pivots and inverts the finished 16×16 diagonal blocks. The block's slot of `linv`
// receives L in FP64 strictly below the diagonal (unit rows beyond jb) and the inverse of each
// 16×16 diagonal block, transposed, above it: what the panels need. The inverse of the whole
// block, which only the solves read, is formed for all blocks at once at the end of the numeric
// phase (k_block_inverse). This is the factorization of the reference's diagonal block (row by
// row there, src/sparse.rs:516-537) with the same sums taken in another order; the pivot test
// (src/sparse.rs:528-531) runs on every pivot in order and stops the front at the first
// failure, recording that equation. (With 16-pivot sub-panels whose pivot columns went through
// shared memory, the block's inverse inside and uncoalesced block loads and stores, the pivot
// launches of a factorization took 4.1 ms on the 33³ cube, 174 of them, 1.47 ms on the 22³ cube
// and 10.2 ms on the 60³ cube; now 3.0, 1.07 and 8.2 ms with k_block_inverse. A single launch is
// about 21,000 cycles: 2,800 to load, 1,750 per sub-panel, of which the elimination takes 1,100
// and the two barriers with the look-ahead between them the rest, 2,800 for the last inverse and
// the stores.)
constexpr int PBT = 256;       // threads
constexpr int PB = 8;          // pivots per sub-panel
constexpr int SB = 16;         // diagonal blocks inverted for the panels
constexpr int PBP = NB + 2;    // pitch of the block (doubles)
constexpr int PBW = 12;        // pitch of the sub-panel operands: conflict-free fragments
constexpr size_t PB_SMEM = (size_t)(NB * (PBP + 4 * PBW) + SB * PBW) * sizeof(double);

// Rank-8 update of the 8×8 tile (ti, tj) of the block: A −= W[ti]·L[tj]ᵀ. All lanes of a warp.
__device__ __forceinline__ void pb_tile(double* A, const double* W, const double* L, int ti, int tj) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    double2* c = reinterpret_cast<double2*>(A + (8 * ti + g) * PBP + 8 * tj + 2 * q);
    double2 v = *c;
    const double* w = W + (8 * ti + g) * PBW + q;
    const double* l = L + (8 * tj + g) * PBW + q;
    dmma_884(v.x, v.y, -w[0], l[0]);
    dmma_884(v.x, v.y, -w[4], l[4]);
    *c = v;
}

// The same for the tiles (t0 + i, t0 + j), j <= i < n, numbered along the rows: warp x of PBR
// takes the tiles x, x + PBR, ..., all operands loaded before any store.
constexpr int PBR = 5;
__device__ __noinline__ void pb_rest(double* A, const double* W, const double* L, int t0, int n, int x) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, cnt = n * (n + 1) / 2;
    constexpr int M = 5;  // 21 tiles at most: n <= 6
    double2 v[M];
    double w0[M], w1[M], l0[M], l1[M];
    int off[M];
#pragma unroll
    for (int u = 0; u < M; u++) {
        const int e = x + PBR * u;
        if (e >= cnt) continue;
        const int i = (e >= 1) + (e >= 3) + (e >= 6) + (e >= 10) + (e >= 15), j = e - i * (i + 1) / 2;
        off[u] = (8 * (t0 + i) + g) * PBP + 8 * (t0 + j) + 2 * q;
        v[u] = *reinterpret_cast<const double2*>(A + off[u]);
        const double* w = W + (8 * (t0 + i) + g) * PBW + q;
        const double* l = L + (8 * (t0 + j) + g) * PBW + q;
        w0[u] = -w[0];
        w1[u] = -w[4];
        l0[u] = l[0];
        l1[u] = l[4];
    }
#pragma unroll
    for (int u = 0; u < M; u++)
        if (x + PBR * u < cnt) dmma_884(v[u].x, v[u].y, w0[u], l0[u]);
#pragma unroll
    for (int u = 0; u < M; u++)
        if (x + PBR * u < cnt) {
            dmma_884(v[u].x, v[u].y, w1[u], l1[u]);
            *reinterpret_cast<double2*>(A + off[u]) = v[u];
        }
}

// Inverse of the unit lower SB×SB diagonal block at cp into the upper half of the slot,
// transposed (out[cp + c][cp + r] = X[r][c]), by one warp: the two 8×8 diagonal inverses a column
// per lane (lanes 0 .. 15), then X21 = −X22·(L21·X11) as two tensor-core products. S: a work tile
// of SB rows of PBW doubles.
__device__ __noinline__ void pb_diag_inverse(const double* A, double* S, double* out, int cp) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    if (lane < SB) {
        const int c = lane & 7, b8 = cp + (lane & 8);
        double x[PB];
#pragma unroll
        for (int r = 0; r < PB; r++) {
            double v = r == c ? 1.0 : 0.0;
#pragma unroll
            for (int k = 0; k < r; k++) v -= A[(b8 + r) * PBP + b8 + k] * x[k];
            x[r] = v;  // zero above the diagonal: x[k] = 0 for k < c
        }
#pragma unroll
        for (int r = 0; r < PB; r++) {
            S[((lane & 8) + r) * PBW + c] = x[r];
            if (r > c) out[(b8 + c) * NB + b8 + r] = x[r];
        }
    }
    __syncwarp();
    const double* l = A + (cp + PB + g) * PBP + cp + q;
    double y0 = 0.0, y1 = 0.0;
    dmma_884(y0, y1, l[0], S[q * PBW + g]);
    dmma_884(y0, y1, l[4], S[(q + 4) * PBW + g]);
    // Y as the right operand: Y[k][n] is in lane 4k + n/2, element n & 1
    double b[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int src = 4 * (q + 4 * h) + (g >> 1);
        const double v0 = __shfl_sync(0xffffffffu, y0, src), v1 = __shfl_sync(0xffffffffu, y1, src);
        b[h] = g & 1 ? v1 : v0;
    }
    double x0 = 0.0, x1 = 0.0;
    dmma_884(x0, x1, -S[(PB + g) * PBW + q], b[0]);
    dmma_884(x0, x1, -S[(PB + g) * PBW + q + 4], b[1]);
    out[(cp + 2 * q) * NB + cp + PB + g] = x0;
    out[(cp + 2 * q + 1) * NB + cp + PB + g] = x1;
    __syncwarp();  // S is read
}

template <typename T>
__global__ void __launch_bounds__(PBT, 2) k_pivot_block(T* __restrict__ panel, double* __restrict__ d,
                                                        const double* adiag,
                                                        const DFront* __restrict__ fr, const int64_t* __restrict__ order,
                                                        int64_t fr_off, int64_t s, int64_t* __restrict__ status,
                                                        double* __restrict__ linv) {
    extern __shared__ __align__(16) double pb_smem[];
    double* A = pb_smem;                // [NB][PBP]
    double* Wq = pb_smem + NB * PBP;    // [2][NB][PBW]: the sub-panel's W = L·D and L rows, by parity
    double* Lq = Wq + 2 * NB * PBW;     // [2][NB][PBW]
    double* Sv = Lq + 2 * NB * PBW;     // [SB][PBW]: work tile of the inverses
    __shared__ double orig[NB];
    __shared__ int bad;                 // first pivot of the block that breaks the rule, or NB
    const int64_t t = order[fr_off + blockIdx.x];
    const DFront f = fr[t];
    pdl_wait();
    pdl_launch_dependents();
    if (status[t] != -1) return;
    const int64_t j0 = s * NB;
    const int jb = (int)min((int64_t)NB, f.k - j0), nsp = (jb + PB - 1) / PB;
    T* blk = panel + f.poff + j0 * f.ldp + j0;
    double* out = linv + (f.blk_off + s) * (int64_t)(NB * NB);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    using VT = typename std::conditional<sizeof(T) == 4, float2, double2>::type;
    {
        // warp w: rows w, w + 8, ... (two columns per lane, all loads issued before any store).
        // Rows and columns beyond jb get a unit diagonal so the sub-panels need no bounds
        VT v[NB / 8];
#pragma unroll
        for (int i = 0; i < NB / 8; i++) {
            const int r = warp + 8 * i;
            v[i] = VT{};
            if (r < jb && 2 * lane <= r) v[i] = *reinterpret_cast<const VT*>(blk + (int64_t)r * f.ldp + 2 * lane);
        }
        for (int p = tid; p < NB; p += PBT) orig[p] = p < jb ? __ldcg(adiag + f.start + j0 + p) : 1.0;
        if (tid == 0) bad = NB;
#pragma unroll
        for (int i = 0; i < NB / 8; i++) {
            const int r = warp + 8 * i, c = 2 * lane;
            double2 w = make_double2((double)v[i].x, (double)v[i].y);
            if (r >= jb && c == r) w.x = 1.0;
            if (r >= jb && c + 1 == r) w.y = 1.0;
            *reinterpret_cast<double2*>(A + r * PBP + c) = w;
        }
    }
    __syncthreads();
    for (int b = 0; b < nsp; b++) {
        const int c0 = b * PB;
        double* const W = Wq + (b & 1) * NB * PBW;
        double* const L = Lq + (b & 1) * NB * PBW;
        if (warp < 2) {
            // lane: row c0 + 8 + tid below the diagonal block (rows past the block idle along)
            const int r = c0 + PB + tid;
            const bool live = r < NB;
            double D[PB][PB], a[PB];
            double* const wr = W + (live ? r : c0) * PBW;  // an idle lane's entries are read by nobody
#pragma unroll
            for (int i = 0; i < PB; i++)
#pragma unroll
                for (int k = 0; k <= i; k += 2) {
                    const double2 v = *reinterpret_cast<const double2*>(A + (c0 + i) * PBP + c0 + k);
                    D[i][k] = v.x;
                    if (k + 1 <= i) D[i][k + 1] = v.y;
                }
            const double* row = A + (live ? r : c0) * PBP + c0;
#pragma unroll
            for (int k = 0; k < PB; k += 2) {
                const double2 v = *reinterpret_cast<const double2*>(row + k);
                a[k] = v.x;
                a[k + 1] = v.y;
            }
            // Both warps hold the diagonal block before thread 32 stores its factor over it. (A
            // named barrier of the 64 threads: the six other warps are in the previous
            // sub-panel's update.)
            asm volatile("bar.sync 1, 64;" ::: "memory");
            // the eight pivots without a branch: the rule is checked on all of them afterwards (a
            // bad pivot spoils only values that nobody reads, the front stops here)
#pragma unroll
            for (int j = 0; j < PB; j++) {
                const double rinv = recip_chebyshev(D[j][j]);
                double l[PB];
#pragma unroll
                for (int i = j + 1; i < PB; i++) {
                    l[i] = D[i][j] * rinv;
#pragma unroll
                    for (int k = j + 1; k <= i; k++) D[i][k] -= l[i] * D[k][j];
                }
                wr[j] = a[j];
                a[j] *= rinv;
#pragma unroll
                for (int k = j + 1; k < PB; k++) a[k] -= a[j] * D[k][j];
#pragma unroll
                for (int i = j + 1; i < PB; i++) D[i][j] = l[i];
            }
            if (live) {
                double* const ar = A + r * PBP + c0;
                double* const lr = L + r * PBW;
#pragma unroll
                for (int k = 0; k < PB; k += 2) {
                    const double2 v = make_double2(a[k], a[k + 1]);
                    *reinterpret_cast<double2*>(ar + k) = v;
                    *reinterpret_cast<double2*>(lr + k) = v;
                }
            }
            if (tid == 32) {
#pragma unroll
                for (int i = 0; i < PB; i++)
#pragma unroll
                    for (int k = 0; k <= i; k += 2) {
                        if (k + 1 <= i)
                            *reinterpret_cast<double2*>(A + (c0 + i) * PBP + c0 + k) = make_double2(D[i][k], D[i][k + 1]);
                        else
                            A[(c0 + i) * PBP + c0 + k] = D[i][k];
                    }
            }
        } else if (b > 0) {
            // the previous sub-panel's update right of this one, and the finished inverses
            const double* Wp = Wq + ((b - 1) & 1) * NB * PBW;
            const double* Lp = Lq + ((b - 1) & 1) * NB * PBW;
            if (warp == 7) {
                if ((b & 1) == 0) pb_diag_inverse(A, Sv, out, (b - 2) * PB);
            } else {
                pb_rest(A, Wp, Lp, b + 1, nsp - b - 1, warp - 2);
            }
        }
        __syncthreads();
        // look-ahead: this sub-panel's update of the next one's columns; warp 7, which has none of it,
        // tests the sub-panel's pivots
        if (warp < 7) {
            if (b + 1 + warp < nsp) pb_tile(A, W, L, b + 1 + warp, b + 1);
        } else {
            const int p = c0 + lane;
            const bool mine = lane < PB && p < jb;
            const double pv = mine ? A[p * PBP + p] : 1.0, o = mine ? orig[p] : 1.0;
            const unsigned fail = __ballot_sync(0xffffffffu, !(o > 0.0) || !(pv > 1e-12 * o));
            const int first = fail ? c0 + __ffs(fail) - 1 : NB;
            if (mine && p < first) d[f.start + j0 + p] = pv;
            if (fail && lane == 0) {
                bad = first;
                status[t] = f.start + j0 + first;
            }
        }
        __syncthreads();
        if (bad < NB) return;
    }
    // the last 16×16 block's inverse beside the stores of L: the slot's rows and columns of whole
    // 16×16 blocks (beyond them the slot is the identity since the engine was set up)
    const int nd = (jb + SB - 1) / SB * SB;
    if (warp == 0) {
        pb_diag_inverse(A, Sv, out, nd - SB);
    } else {
        const int c = 2 * lane;
#pragma unroll
        for (int i = 0; i < (NB + 6) / 7; i++) {
            const int r = warp - 1 + 7 * i;
            if (r >= nd || c > r) continue;
            const double2 w = *reinterpret_cast<const double2*>(A + r * PBP + c);
            if (r < jb) {
                T* const o = blk + (int64_t)r * f.ldp + c;
                if (c + 1 <= r) {
                    VT v;
                    v.x = (T)w.x;
                    v.y = (T)w.y;
                    *reinterpret_cast<VT*>(o) = v;
                } else {
                    o[0] = (T)w.x;
                }
            }
            if (c + 1 < r) {
                *reinterpret_cast<double2*>(out + r * NB + c) = w;
            } else if (c < r) {
                out[r * NB + c] = w.x;
            }
        }
    }
}

// Unit lower slots (the identity): rows and columns that no block fills stay so.
__global__ void k_slot_identity(double* __restrict__ linv) {
    double* slot = linv + blockIdx.x * (int64_t)(NB * NB);
    for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) slot[e] = e / NB == e % NB ? 1.0 : 0.0;
}

// The slots of linv from L and the transposed 16×16 inverses (k_pivot_block) to the inverses of
// the whole blocks (lower triangular, zeros above), which the solves read: by block rows,
// X_pp given, X[p, :p] = −X_pp·(L[p, :p]·X[:p, :p]). One CTA of four warps per slot, products on the
// FP64 tensor-core path, only the 16×16 blocks that hold pivots (width[slot] pivots); bound by the
// bytes a slot reads and writes.
constexpr int BIP = NB + 4;
constexpr size_t BI_SMEM = (size_t)(2 * NB + SB) * BIP * sizeof(double);
__global__ void __launch_bounds__(128) k_block_inverse(double* __restrict__ linv, const uint8_t* __restrict__ width) {
    extern __shared__ __align__(16) double bi_smem[];
    double* L = bi_smem;             // [NB][BIP]
    double* X = bi_smem + NB * BIP;  // [NB][BIP]
    double* Y = X + NB * BIP;        // [SB][BIP]
    double* slot = linv + blockIdx.x * (int64_t)(NB * NB);
    const int nb = (width[blockIdx.x] + SB - 1) / SB, nd = nb * SB;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    pdl_wait();
    pdl_launch_dependents();
    for (int r = w; r < nd; r += 4) {
        const int c = 2 * lane;
        if (c >= nd) continue;
        const double2 v = *reinterpret_cast<const double2*>(slot + r * NB + c);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const double x = u ? v.y : v.x;
            const int cc = c + u;
            L[r * BIP + cc] = cc < r ? x : 0.0;
            // a diagonal 16×16 block holds its inverse transposed above the diagonal
            if ((cc ^ r) < SB)
                X[cc * BIP + r] = cc > r ? x : (cc == r ? 1.0 : 0.0);
            else if (cc > r)
                X[r * BIP + cc] = 0.0;
        }
    }
    __syncthreads();
    for (int p = 1; p < nb; p++) {
        const int cp = p * SB;
        // 8×8 tiles: two tile rows, 2p tile columns, of which warp w takes w and w + 4
        for (int ct = w; ct < 2 * p; ct += 4) {
            double acc[2][2] = {};
            for (int k = (ct & ~1) * 8; k < cp; k += 4) {  // X is zero above its diagonal blocks
                const double b = X[(k + q) * BIP + 8 * ct + g];
#pragma unroll
                for (int m = 0; m < 2; m++) dmma_884(acc[m][0], acc[m][1], L[(cp + 8 * m + g) * BIP + k + q], b);
            }
#pragma unroll
            for (int m = 0; m < 2; m++) {
                Y[(8 * m + g) * BIP + 8 * ct + 2 * q] = acc[m][0];
                Y[(8 * m + g) * BIP + 8 * ct + 2 * q + 1] = acc[m][1];
            }
        }
        __syncwarp();  // a warp's columns of Y are its own
        for (int ct = w; ct < 2 * p; ct += 4) {
            double acc[2][2] = {};
#pragma unroll
            for (int k = 0; k < SB; k += 4) {
                const double b = Y[(k + q) * BIP + 8 * ct + g];
#pragma unroll
                for (int m = 0; m < 2; m++) dmma_884(acc[m][0], acc[m][1], X[(cp + 8 * m + g) * BIP + cp + k + q], b);
            }
#pragma unroll
            for (int m = 0; m < 2; m++) {
                X[(cp + 8 * m + g) * BIP + 8 * ct + 2 * q] = -acc[m][0];
                X[(cp + 8 * m + g) * BIP + 8 * ct + 2 * q + 1] = -acc[m][1];
            }
        }
        __syncthreads();
    }
    for (int r = w; r < nd; r += 4) {
        const int c = 2 * lane;
        if (c < nd) *reinterpret_cast<double2*>(slot + r * NB + c) = *reinterpret_cast<const double2*>(X + r * BIP + c);
    }
}

// FP16 split of the tensor-core update: the power-of-two scale of a row of U = L·D^(1/2)
// from the row's diagonal a_rr in the original matrix. Every Schur complement of a
// positive definite matrix has its diagonal below the original one and U[r, p]² is at
// most the diagonal of row r in the Schur complement that eliminates p, so
// |U[r, p]| ≤ a_rr^(1/2) and the scaled row stays below 2^12, far inside the FP16 range
// (65504). 0 for a diagonal that is not positive and finite.
__device__ __forceinline__ float u16_row_scale(double arr) {
    if (!(arr > 0.0) || !(arr < INFINITY)) return 0.f;
    int e;
    frexp(sqrt(arr), &e);  // sqrt(a_rr) < 2^e
    return (float)ldexp(1.0, 12 - e);
}

// Panel of one step: for the PNR rows r in [j1, m) of a CTA, W[r, :] = F[r, j0:j1]·L_bb⁻ᵀ and
// L[r, :] = W[r, :]·D⁻¹ (the forward substitution w ← w·L⁻ᵀ of src/sparse.rs:547-558), on the
// FP64 tensor-core path (m8n8k4) in both precisions. A warp keeps 16 rows in registers from
// the load to the store: lane (g, q) holds the columns 16G + 4q ... + 3 of the rows g and 8 + g.
// The two n-tiles of a 16-column group take the columns 4q + {0, 1} and 4q + {2, 3}, so that
// a result fragment is an operand fragment of the next product as it stands (the k index runs
// over q), and loads and stores are four consecutive columns a lane. The other operand
// stands in shared memory in rows of PNP doubles: the 16-byte fragment
// loads (two rows, four lanes each 32 bytes apart) meet every bank once.
// The substitution goes by 16-column groups, T = F_b − Σ_{a<b} W_a·L_baᵀ, W_b = T·L_bb⁻ᵀ with the
// inverse of the 16 × 16 diagonal block, and for an FP64 factor one refinement step against that
// block (R = T − W_b·L_bbᵀ, W_b += R·L_bb⁻ᵀ).
// L goes to the panel, and as the plan's mode says, W and L rows to the outer block's scratch in
// the storage precision (PANEL_SCR; front row r is scratch row pre_scr[i] + r − J0, columns
// j0 − J0 ...) and the split operands of the tensor cores (PANEL_SPLIT): the TF32 heads and
// tails of W and L (whi non-null) or the FP16 head and tail of U·s_r = L·D^(1/2)·s_r (uhi
// non-null). U is formed in FP32 from L as stored (one FP64 → FP32 conversion per entry for L
// and U together). A scaled U entry outside the FP16 range sets *err = 21.
// Near the top of the tree a launch has a few rows per SM and its time is one CTA's: with 128
// rows per CTA through shared memory and (FP64) three full 64-column products the panel launches
// of a factorization took 6.2 ms on the 33³ cube (FP64, 173 launches; now 3.5 ms), 2.8 ms for 160
// batched plates (0.8 ms) and 17.4 ms on the 60³ cube (mixed, 415 launches; 11.8 ms). At the
// leaves it is bound by the stores.
constexpr int PNP = NB + 2;   // pitch of L_bb (doubles)
constexpr int PNI = 18;       // pitch of the 16-column diagonal inverses
constexpr int PNT = 128;      // threads
constexpr size_t PANEL_SMEM = NB * (PNP + PNI) * sizeof(double);

// acc (two n-tiles of two row tiles) += ±A·Bᵀ over one 16-column group: A the lane's four values
// per row tile, B rows at b0 (n-tile 0) and b0 + 2 rows (n-tile 1).
template <bool NEG, int P>
__device__ __forceinline__ void panel_group(double (&acc)[2][4], const double (&a)[2][4], const double* b0) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const double2 u = *reinterpret_cast<const double2*>(b0 + 2 * h * P);
        const double2 v = *reinterpret_cast<const double2*>(b0 + 2 * h * P + 2);
        const double b[4] = {u.x, u.y, v.x, v.y};
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int m = 0; m < 2; m++)
                dmma_884(acc[m][2 * h], acc[m][2 * h + 1], NEG ? -a[m][k] : a[m][k], b[k]);
    }
}

template <typename T>
__global__ void __launch_bounds__(PNT) k_panel(T* __restrict__ panel, const double* d,
                                               const double* linv, const DFront* __restrict__ fr,
                                               const int64_t* __restrict__ order, int64_t fr_off, int64_t nact,
                                               const int64_t* __restrict__ pre_panel, const int64_t* __restrict__ pre_scr,
                                               int64_t s, T* __restrict__ scr_w, T* __restrict__ scr_l,
                                               const int64_t* status, float* __restrict__ whi,
                                               float* __restrict__ wlo, float* __restrict__ lhi, float* __restrict__ llo,
                                               const uint8_t* __restrict__ mode, const int64_t* __restrict__ rows,
                                               const double* adiag0, __half* __restrict__ uhi,
                                               __half* __restrict__ ulo, float* __restrict__ uscale,
                                               int* __restrict__ err) {
    extern __shared__ __align__(16) double pnl_smem[];
    double* Lb = pnl_smem;             // [NB][PNP]: L_bb
    double* Iv = pnl_smem + NB * PNP;  // [NB][PNI]: the inverses of its 16 × 16 diagonal blocks
    __shared__ double dinv[NB];
    __shared__ float usq[NB];
    const int64_t i = find_slot_warp(pre_panel, nact, blockIdx.x);
    const int64_t chunk = blockIdx.x - pre_panel[i];
    const int64_t t = order[fr_off + i];
    const DFront f = fr[t];
    const int64_t j0 = s * NB;
    const int jb = (int)min((int64_t)NB, f.k - j0);
    const int64_t j1 = j0 + jb;
    const int64_t J0 = (s / KO) * NBO;
    const int64_t r0 = j1 + chunk * PNR;
    const int nr = (int)min((int64_t)PNR, f.m - r0);
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    // the chunk's rows of the step's columns are final once the update kernel before the
    // pivot kernel has completed, which the pivot kernel waited for before it let this
    // kernel start (programmatic launch): they are loaded, from L2, while the pivot block is factored.
    // A group of four columns that starts below jb ends inside the row's padding (zeros).
    double F[4][2][4];
#pragma unroll
    for (int G = 0; G < 4; G++)
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int rr = 16 * w + 8 * m + g, c = 16 * G + 4 * q;
            const bool ok = rr < nr && c < jb;
            const T* p = panel + f.poff + (r0 + rr) * f.ldp + j0 + c;
            if constexpr (sizeof(T) == 4) {
                const float4 v = ok ? __ldcg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
                F[G][m][0] = v.x;
                F[G][m][1] = v.y;
                F[G][m][2] = v.z;
                F[G][m][3] = v.w;
            } else {
                const double2 z = make_double2(0.0, 0.0);
                const double2 u = ok ? __ldcg(reinterpret_cast<const double2*>(p)) : z;
                const double2 v = ok ? __ldcg(reinterpret_cast<const double2*>(p + 2)) : z;
                F[G][m][0] = u.x;
                F[G][m][1] = u.y;
                F[G][m][2] = v.x;
                F[G][m][3] = v.y;
            }
        }
    // the scratch rows and the split operands only where an update reads them
    const uint8_t md = mode[i];
    if (!(md & PANEL_SPLIT)) {
        whi = nullptr;
        uhi = nullptr;
    }
    const bool scr = (md & PANEL_SCR) != 0;
    const int64_t sr0 = pre_scr[i] + (r0 - J0);  // scratch row of the chunk's first row
    float rsc = 0.f;  // the scale of the warp's row `lane` (lanes 0 .. 15)
    if (sizeof(T) == sizeof(float) && uhi && lane < 16 && 16 * w + lane < nr) {
        // the rows' scales from their original diagonal (known since the assembly), also
        // kept per scratch row for the tensor-core epilogue: while the pivot block runs
        const int64_t r = r0 + 16 * w + lane;
        rsc = u16_row_scale(__ldcg(adiag0 + (r < f.k ? f.start + r : rows[f.rows_off + r - f.k])));
        if (rsc == 0.f) atomicExch(err, 21);
        uscale[sr0 + 16 * w + lane] = rsc;
    }
    pdl_wait();
    pdl_launch_dependents();
    if (status[t] != -1) return;
    {
        // the block's slot: L strictly below the diagonal, the 16 × 16 inverses transposed above
        const double* li = linv + (f.blk_off + s) * (int64_t)(NB * NB);
        constexpr int PER = NB * NB / 2 / PNT;  // 16-byte loads per thread, all issued before any store
        double2 v[PER];
#pragma unroll
        for (int u = 0; u < PER; u++) v[u] = __ldcg(reinterpret_cast<const double2*>(li) + u * PNT + tid);
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int e = 2 * (u * PNT + tid), r = e / NB, c = e % NB;
            double2 l = v[u];
            if (c >= r) l.x = c == r ? 1.0 : 0.0;
            if (c + 1 >= r) l.y = c + 1 == r ? 1.0 : 0.0;
            *reinterpret_cast<double2*>(Lb + r * PNP + c) = l;
            if ((c ^ r) < 16) {
                Iv[c * PNI + (r & 15)] = c > r ? v[u].x : (c == r ? 1.0 : 0.0);
                Iv[(c + 1) * PNI + (r & 15)] = c + 1 > r ? v[u].y : (c + 1 == r ? 1.0 : 0.0);
            }
        }
    }
    if (tid < NB) {
        const double dv = tid < jb ? __ldcg(d + f.start + j0 + tid) : 0.0;
        dinv[tid] = tid < jb ? 1.0 / dv : 0.0;
        if (sizeof(T) == sizeof(float)) usq[tid] = tid < jb ? (float)sqrt(dv) : 0.f;
    }
    __syncthreads();
    if (16 * w >= nr) return;
    const int orow = 4 * (g >> 1) + (g & 1);  // n-tile 0: output column 16G + orow, n-tile 1: + 2
#pragma unroll
    for (int b = 0; b < 4; b++) {
        if (16 * b >= jb) break;
        const double* Lr = Lb + (16 * b + orow) * PNP + 4 * q;
        const double* Ir = Iv + (16 * b + orow) * PNI + 4 * q;
#pragma unroll
        for (int a = 0; a < b; a++) panel_group<true, PNP>(F[b], F[a], Lr + 16 * a);
        double x[2][4] = {};
        panel_group<false, PNI>(x, F[b], Ir);
        if constexpr (sizeof(T) == 8) {
            panel_group<true, PNP>(F[b], x, Lr + 16 * b);
            panel_group<false, PNI>(x, F[b], Ir);
        }
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int e = 0; e < 4; e++) F[b][m][e] = x[m][e];
    }
#pragma unroll
    for (int m = 0; m < 2; m++) {
        const int rr = 16 * w + 8 * m + g;
        const float rs = __shfl_sync(0xffffffffu, rsc, 8 * m + g);
        if (rr >= nr) continue;
        T* prow = panel + f.poff + (r0 + rr) * f.ldp + j0;
        const int64_t so = (sr0 + rr) * NBO + (j0 - J0);
#pragma unroll
        for (int G = 0; G < 4; G++) {
            const int c = 16 * G + 4 * q;
            const double(&wv)[4] = F[G][m];
            double l[4];
#pragma unroll
            for (int e = 0; e < 4; e++) l[e] = wv[e] * dinv[c + e];
            if constexpr (sizeof(T) == 4) {
                const float4 lf = make_float4((float)l[0], (float)l[1], (float)l[2], (float)l[3]);
                if (c < jb) *reinterpret_cast<float4*>(prow + c) = lf;
                if (scr) {
                    *reinterpret_cast<float4*>(scr_l + so + c) = lf;
                    *reinterpret_cast<float4*>(scr_w + so + c) =
                        make_float4((float)wv[0], (float)wv[1], (float)wv[2], (float)wv[3]);
                }
                const float la[4] = {lf.x, lf.y, lf.z, lf.w};
                if (whi) {
                    float wh[4], wl[4], lh[4], ll[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float wf = (float)wv[e];
                        wh[e] = tc::to_tf32(wf);
                        wl[e] = tc::to_tf32(wf - wh[e]);
                        lh[e] = tc::to_tf32(la[e]);
                        ll[e] = tc::to_tf32(la[e] - lh[e]);
                    }
                    *reinterpret_cast<float4*>(whi + so + c) = make_float4(wh[0], wh[1], wh[2], wh[3]);
                    *reinterpret_cast<float4*>(wlo + so + c) = make_float4(wl[0], wl[1], wl[2], wl[3]);
                    *reinterpret_cast<float4*>(lhi + so + c) = make_float4(lh[0], lh[1], lh[2], lh[3]);
                    *reinterpret_cast<float4*>(llo + so + c) = make_float4(ll[0], ll[1], ll[2], ll[3]);
                }
                if (uhi) {
                    __half2 hi[2], lo[2];
#pragma unroll
                    for (int e = 0; e < 4; e += 2) {
                        const float u0 = la[e] * usq[c + e] * rs, u1 = la[e + 1] * usq[c + e + 1] * rs;
                        const __half h0 = __float2half_rn(u0), h1 = __float2half_rn(u1);
                        hi[e / 2] = __halves2half2(h0, h1);
                        lo[e / 2] = __halves2half2(__float2half_rn(u0 - __half2float(h0)),
                                                   __float2half_rn(u1 - __half2float(h1)));
                        if (!(fabsf(u0) < 65504.f) || !(fabsf(u1) < 65504.f)) atomicExch(err, 21);
                    }
                    *reinterpret_cast<uint2*>(uhi + so + c) = *reinterpret_cast<const uint2*>(hi);
                    *reinterpret_cast<uint2*>(ulo + so + c) = *reinterpret_cast<const uint2*>(lo);
                }
            } else {
                const double2 l0 = make_double2(l[0], l[1]), l1 = make_double2(l[2], l[3]);
                if (c < jb) {
                    *reinterpret_cast<double2*>(prow + c) = l0;
                    *reinterpret_cast<double2*>(prow + c + 2) = l1;
                }
                if (scr) {
                    *reinterpret_cast<double2*>(scr_l + so + c) = l0;
                    *reinterpret_cast<double2*>(scr_l + so + c + 2) = l1;
                    *reinterpret_cast<double2*>(scr_w + so + c) = make_double2(wv[0], wv[1]);
                    *reinterpret_cast<double2*>(scr_w + so + c + 2) = make_double2(wv[2], wv[3]);
                }
            }
        }
    }
}

// Tile lt of a step's update on the UT×UT grid, with the pivots it applies (kofs, klen:
// offset and count in the outer block's scratch rows):
//   inner (OUTER = false): rows [j1, m), columns [j1, J1e), the step's pivots [j0, j1);
//   outer (OUTER = true):  rows [J1e, m), columns [J1e, k) (panel) and [k, m) (update
//                          block), the outer block's pivots [J0, J1e).
// The panel part's lower-triangular tiles come first (column by column, rows from the
// diagonal tile down), then the lower triangle of the update block.
struct SmallTile {
    int64_t row0, col0, col_end, kofs, klen;
    bool in_panel;
};
template <bool OUTER>
__device__ __forceinline__ SmallTile small_tile(const DFront& f, int64_t s, int64_t lt) {
    const int64_t j0 = s * NB;
    const int64_t j1 = min(j0 + NB, f.k);
    const int64_t J0 = (s / KO) * NBO;
    const int64_t J1e = min(J0 + NBO, f.k);
    const int64_t rbase = OUTER ? J1e : j1;
    const int64_t pcol_end = OUTER ? f.k : J1e;
    SmallTile b;
    b.kofs = OUTER ? 0 : j0 - J0;
    b.klen = OUTER ? J1e - J0 : j1 - j0;
    const int64_t R = f.m - rbase;
    const int64_t nrt = (R + UT - 1) / UT, ncp = (pcol_end - rbase + UT - 1) / UT;
    const int64_t cntP = ncp * nrt - ncp * (ncp - 1) / 2;
    if (lt < cntP) {
        int64_t tj = 0, cnt = nrt;
        while (lt >= cnt) {
            lt -= cnt;
            tj++;
            cnt = nrt - tj;
        }
        b.row0 = rbase + (tj + lt) * UT;
        b.col0 = rbase + tj * UT;
        b.col_end = pcol_end;
        b.in_panel = true;
    } else {
        const int64_t idx = lt - cntP;
        int64_t ti = (int64_t)((sqrt(8.0 * (double)idx + 1.0) - 1.0) * 0.5);
        while (ti * (ti + 1) / 2 > idx) ti--;
        while ((ti + 1) * (ti + 2) / 2 <= idx) ti++;
        const int64_t tj = idx - ti * (ti + 1) / 2;
        b.row0 = f.k + ti * UT;
        b.col0 = f.k + tj * UT;
        b.col_end = f.m;
        b.in_panel = false;
    }
    return b;
}

// Schur update F[r, c] −= Σ_p W[r, p]·L[c, p] for c <= r on the tiles of small_tile, tile
// UT×UT, 256 threads with 4×4 outputs each, K in chunks of NB through shared memory.
template <typename T, typename S, bool OUTER>
__global__ void __launch_bounds__(256) k_schur(T* __restrict__ panel, T* __restrict__ upd, const DFront* __restrict__ fr,
                                               const int64_t* __restrict__ order, int64_t fr_off, int64_t nact,
                                               const int64_t* __restrict__ pre_tiles, const int64_t* __restrict__ pre_scr,
                                               int64_t s, const S* scr_w, const S* scr_l,
                                               const int64_t* status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S* As = reinterpret_cast<S*>(smem_raw);  // [NB][UT + 1]
    S* Bs = As + NB * (UT + 1);
    int64_t b = blockIdx.x;
    int64_t i = find_slot_warp(pre_tiles, nact, b);
    int64_t lt = b - pre_tiles[i];
    int64_t t = order[fr_off + i];
    const DFront f = fr[t];
    pdl_wait();  // before this only plan data is read, which no kernel writes
    pdl_launch_dependents();
    if (status[t] != -1) return;
    const int64_t J0 = (s / KO) * NBO;
    const SmallTile st = small_tile<OUTER>(f, s, lt);
    const int64_t row0 = st.row0, col0 = st.col0, col_end = st.col_end, kofs = st.kofs, klen = st.klen;
    const bool in_panel = st.in_panel;
    // scratch row of front row r: pre_scr[i] + r − J0
    const S* wbase = scr_w + (pre_scr[i] - J0) * NBO + kofs;
    const S* lbase = scr_l + (pre_scr[i] - J0) * NBO + kofs;
    int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    S acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[a][c] = (S)0;
    for (int64_t k0 = 0; k0 < klen; k0 += NB) {
        int kc = (int)min((int64_t)NB, klen - k0);
        if (k0 > 0) __syncthreads();
        for (int idx = threadIdx.x; idx < UT * NB; idx += blockDim.x) {
            int rr = idx / NB, kk = idx - rr * NB;
            int64_t r = row0 + rr, c = col0 + rr;
            bool kin = kk < kc;
            As[kk * (UT + 1) + rr] = (kin && r < f.m) ? __ldcg(wbase + r * NBO + k0 + kk) : (S)0;
            Bs[kk * (UT + 1) + rr] = (kin && c < col_end) ? __ldcg(lbase + c * NBO + k0 + kk) : (S)0;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < NB; kk++) {
            S av[4], bv[4];
#pragma unroll
            for (int a = 0; a < 4; a++) av[a] = As[kk * (UT + 1) + ty + 16 * a];
#pragma unroll
            for (int c = 0; c < 4; c++) bv[c] = Bs[kk * (UT + 1) + tx + 16 * c];
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[a][c] = fma(av[a], bv[c], acc[a][c]);
        }
    }
#pragma unroll
    for (int a = 0; a < 4; a++) {
        int64_t r = row0 + ty + 16 * a;
        if (r >= f.m) continue;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            int64_t cc = col0 + tx + 16 * c;
            if (cc >= col_end || cc > r) continue;
            if (in_panel)
                panel[f.poff + r * f.ldp + cc] -= (T)acc[a][c];
            else
                upd[f.uoff + (r - f.k) * f.ldu + (cc - f.k)] -= (T)acc[a][c];
        }
    }
}

// Outer update of large fronts on the CUDA cores: 128×128 tiles (the tile grid of the
// tensor-core kernel), 256 threads with 8×8 outputs each, K in chunks of 16 through
// a two-stage shared-memory ring.
constexpr int BT = 128, BK = 16;
template <typename S>
constexpr size_t big_smem() {
    return 2 * 2 * BK * (BT + 1) * sizeof(S);
}

// Tile lt of an outer update on the 128×128 grid: first the lower-triangular tiles of the
// panel columns [J1e, k) (column by column, rows from the diagonal tile down), then the
// lower triangle of the update block [k, m)².
struct BigTile {
    int64_t row0, col0, col_end;
    bool in_panel;
};
__device__ __forceinline__ BigTile big_tile(const DFront& f, int64_t J1e, int64_t lt) {
    const int64_t R = f.m - J1e;
    const int64_t nrt = (R + BT - 1) / BT, ncp = (f.k - J1e + BT - 1) / BT;
    const int64_t cntP = ncp * nrt - ncp * (ncp - 1) / 2;
    BigTile b;
    if (lt < cntP) {
        int64_t tj = 0, cnt = nrt;
        while (lt >= cnt) {
            lt -= cnt;
            tj++;
            cnt = nrt - tj;
        }
        b.row0 = J1e + (tj + lt) * BT;
        b.col0 = J1e + tj * BT;
        b.col_end = f.k;
        b.in_panel = true;
    } else {
        const int64_t idx = lt - cntP;
        int64_t ti = (int64_t)((sqrt(8.0 * (double)idx + 1.0) - 1.0) * 0.5);
        while (ti * (ti + 1) / 2 > idx) ti--;
        while ((ti + 1) * (ti + 2) / 2 <= idx) ti++;
        const int64_t tj = idx - ti * (ti + 1) / 2;
        b.row0 = f.k + ti * BT;
        b.col0 = f.k + tj * BT;
        b.col_end = f.m;
        b.in_panel = false;
    }
    return b;
}

template <typename T, typename S>
__global__ void __launch_bounds__(256) k_schur_big(T* __restrict__ panel, T* __restrict__ upd, const DFront* __restrict__ fr,
                                                   const int64_t* __restrict__ order, int64_t fr_off, int64_t nact,
                                                   const int64_t* __restrict__ pre_tiles,
                                                   const int64_t* __restrict__ pre_scr, int64_t s,
                                                   const S* scr_w, const S* scr_l,
                                                   const int64_t* status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S* sbuf = reinterpret_cast<S*>(smem_raw);  // [2 stages][A|B][BK][BT + 1]
    int64_t b = blockIdx.x;
    int64_t i = find_slot_warp(pre_tiles, nact, b);
    int64_t lt = b - pre_tiles[i];
    int64_t t = order[fr_off + i];
    const DFront f = fr[t];
    pdl_wait();  // before this only plan data is read, which no kernel writes
    pdl_launch_dependents();
    if (status[t] != -1) return;
    int64_t J0 = (s / KO) * NBO;
    int64_t J1e = min(J0 + NBO, f.k);
    int64_t klen = J1e - J0;
    const BigTile bt = big_tile(f, J1e, lt);
    const int64_t row0 = bt.row0, col0 = bt.col0, col_end = bt.col_end;
    const bool in_panel = bt.in_panel;
    const S* wbase = scr_w + (pre_scr[i] - J0) * NBO;
    const S* lbase = scr_l + (pre_scr[i] - J0) * NBO;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    // loader: asynchronous copies (cp.async, zero-filled outside the tile) of 128 rows ×
    // BK pivots of W and of L into one stage; consecutive threads take consecutive pivots
    auto load = [&](int stage, int64_t k0) {
        S* As = sbuf + stage * 2 * BK * (BT + 1);
        S* Bs = As + BK * (BT + 1);
        for (int idx = threadIdx.x; idx < BT * BK; idx += 256) {
            int rr = idx / BK, kk = idx - rr * BK;
            int64_t r = row0 + rr, c = col0 + rr;
            bool kin = k0 + kk < klen;
            bool ra = kin && r < f.m, rb = kin && c < col_end;
            const S* ga = ra ? wbase + r * NBO + k0 + kk : wbase;
            const S* gb = rb ? lbase + c * NBO + k0 + kk : lbase;
            uint32_t sa = (uint32_t)__cvta_generic_to_shared(As + kk * (BT + 1) + rr);
            uint32_t sb = (uint32_t)__cvta_generic_to_shared(Bs + kk * (BT + 1) + rr);
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(sa), "l"(ga), "n"(sizeof(S)),
                         "r"(ra ? (int)sizeof(S) : 0)
                         : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(sb), "l"(gb), "n"(sizeof(S)),
                         "r"(rb ? (int)sizeof(S) : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    S acc[8][8];
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
        for (int c = 0; c < 8; c++) acc[a][c] = (S)0;
    int nk = (int)((klen + BK - 1) / BK);
    load(0, 0);
    for (int kc = 0; kc < nk; kc++) {
        if (kc + 1 < nk) {
            load((kc + 1) & 1, (int64_t)(kc + 1) * BK);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const S* As = sbuf + (kc & 1) * 2 * BK * (BT + 1);
        const S* Bs = As + BK * (BT + 1);
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            S av[8], bv[8];
#pragma unroll
            for (int a = 0; a < 8; a++) av[a] = As[kk * (BT + 1) + ty + 16 * a];
#pragma unroll
            for (int c = 0; c < 8; c++) bv[c] = Bs[kk * (BT + 1) + tx + 16 * c];
#pragma unroll
            for (int a = 0; a < 8; a++)
#pragma unroll
                for (int c = 0; c < 8; c++) acc[a][c] = fma(av[a], bv[c], acc[a][c]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 8; a++) {
        int64_t r = row0 + ty + 16 * a;
        if (r >= f.m) continue;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            int64_t cc = col0 + tx + 16 * c;
            if (cc >= col_end || cc > r) continue;
            if (in_panel)
                panel[f.poff + r * f.ldp + cc] -= (T)acc[a][c];
            else
                upd[f.uoff + (r - f.k) * f.ldu + (cc - f.k)] -= (T)acc[a][c];
        }
    }
}

// Outer update of large fronts in FP64 on the tensor cores' FP64 path (mma.sync m8n8k4
// f64, one instruction per 8×8×4 block). Two CTAs per 128×128 tile of k_schur_big's grid,
// one per 64-column half, and two CTAs per SM, so that one CTA's start (the front lookup)
// and read-modify-write epilogue overlap the other's MMAs. 4 warps of 64×32 outputs; K in
// chunks of 16 through a three-stage cp.async ring of padded rows (W and L copied
// row-major, pivots contiguous as in the scratch, pitch 20 doubles: the fragment loads,
// 8 rows × 4 pivots per warp, hit distinct banks in each half-warp). Each warp loads the
// fragments of the next 4-pivot step before it issues the MMAs of the current one.
constexpr int DM_BK = 16, DM_PITCH = 20, DM_STAGES = 3, DM_TN = 64, DM_THREADS = 128;
constexpr int DM_STAGE = (BT + DM_TN) * DM_PITCH;  // doubles per stage: W rows, then L rows
constexpr size_t DM_SMEM = (size_t)DM_STAGES * DM_STAGE * sizeof(double);

// Operand loads of the FP64 updates: ROWS scratch rows of W and then of L, DM_BK pivots each, 128
// threads. Thread (tid / 8, tid % 8) copies the 16 bytes of pivots 2·(tid % 8) of every 16th row, all
// from one pointer at constant offsets: with two warps per scheduler the instructions around the
// products are what keeps the tensor pipe waiting, so there are no bounds. Rows past the front's
// are another front's or the scratch's spare rows (DM_SPARE): they meet outputs that are not
// stored. Pivots past the block's are zeros that the panel stored. (With bounds and zero fill per
// copy there were 4.8 other instructions per product and the tensor pipe was 75 % active in a
// large launch of the 33³ cube; a factorization went from 76.2 to 71.1 ms at 45³, 17.6 to 16.9 ms at
// 33³, 3.63 to 3.49 ms at 22³.)
constexpr int DM_SPARE = 128;
__device__ __forceinline__ void cp_async16_full(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
struct DmLoader {
    const double *w, *l;
    uint32_t s;
    __device__ __forceinline__ DmLoader(const double* wrow, const double* lrow, double* sbuf) {
        const int r = threadIdx.x >> 3, c = (threadIdx.x & 7) * 2;
        w = wrow + r * NBO + c;
        l = lrow + r * NBO + c;
        s = (uint32_t)__cvta_generic_to_shared(sbuf + r * DM_PITCH + c);
    }
    // the next chunk of pivots into the stage at byte offset off
    template <int WR, int LR>
    __device__ __forceinline__ void next(uint32_t off) {
#pragma unroll
        for (int i = 0; i < WR / 16; i++) cp_async16_full(s + off + i * 16 * DM_PITCH * 8, w + i * 16 * NBO);
#pragma unroll
        for (int i = 0; i < LR / 16; i++) cp_async16_full(s + off + (WR + i * 16) * DM_PITCH * 8, l + i * 16 * NBO);
        w += DM_BK;
        l += DM_BK;
    }
};

// Start of front row r in the output of an outer-update tile, indexed by front column:
// the panel row (columns < k) or the update-block row (columns >= k).
__device__ __forceinline__ double* out_row(double* panel, double* upd, const DFront& f, bool in_panel, int64_t r) {
    return in_panel ? panel + f.poff + r * f.ldp : upd + f.uoff + (r - f.k) * f.ldu - f.k;
}

__global__ void __launch_bounds__(DM_THREADS, 2)
    k_schur_dmma(double* __restrict__ panel, double* __restrict__ upd, const DFront* __restrict__ fr,
                 const int64_t* __restrict__ order, int64_t fr_off, int64_t nact, const int64_t* __restrict__ pre_tiles,
                 const int64_t* __restrict__ pre_a, int part, const int64_t* __restrict__ pre_scr, int64_t s,
                 const double* scr_w, const double* scr_l,
                 const int64_t* status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sbuf = reinterpret_cast<double*>(smem_raw);  // [stage][BT W rows | DM_TN L rows][DM_PITCH]
    const int half = blockIdx.x & 1;
    int64_t lt;
    const int64_t i = find_tile_warp(pre_tiles, pre_a, part, nact, blockIdx.x >> 1, &lt);
    const int64_t t = order[fr_off + i];
    const DFront f = fr[t];
    pdl_wait();  // before this only plan data is read, which no kernel writes
    pdl_launch_dependents();
    if (status[t] != -1) return;
    const int64_t J0 = (s / KO) * NBO;
    const int64_t J1e = min(J0 + NBO, f.k);
    const int klen = (int)(J1e - J0);
    const BigTile bt = big_tile(f, J1e, lt);
    const int64_t col0 = bt.col0 + half * DM_TN;
    if (col0 >= bt.col_end) return;
    // scratch row of front row r: pre_scr[i] + r − J0
    const double* wrow = scr_w + (pre_scr[i] - J0 + bt.row0) * NBO;
    const double* lrow = scr_l + (pre_scr[i] - J0 + col0) * NBO;
    const int nk = (klen + DM_BK - 1) / DM_BK;
    {
        // L2 prefetch of this CTA's output rows (in range only), read back at the end
        const int64_t r = bt.row0 + threadIdx.x;
        const int64_t cend = r < f.m ? min(bt.col_end, min(col0 + DM_TN, r + 1)) : col0;
        if (cend > col0) {
            const double* rowp = out_row(panel, upd, f, bt.in_panel, r);
            for (int64_t c = col0; c < cend; c += 16) asm volatile("prefetch.global.L2 [%0];" ::"l"(rowp + c));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(rowp + cend - 1));
        }
    }
    DmLoader ld(wrow, lrow, sbuf);
    constexpr uint32_t STB = DM_STAGE * sizeof(double);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int wm = warp & 1, wn = warp >> 1;  // warp tile rows [64·wm, +64), columns [32·wn, +32)
    const int aoff = (wm * 64 + g) * DM_PITCH + q, boff = (BT + wn * 32 + g) * DM_PITCH + q;
    auto frag = [&](double* fa, double* fb, const double* st) {
#pragma unroll
        for (int a = 0; a < 8; a++) fa[a] = st[aoff + a * 8 * DM_PITCH];
#pragma unroll
        for (int c = 0; c < 4; c++) fb[c] = st[boff + c * 8 * DM_PITCH];
    };
    double acc[8][4][2];
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[a][c][0] = acc[a][c][1] = 0.0;
    double fa[2][8], fb[2][4];
    ld.next<BT, DM_TN>(0);
    cp_async_commit();
    if (nk > 1) ld.next<BT, DM_TN>(STB);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    if (nk > 2) ld.next<BT, DM_TN>(2 * STB);
    cp_async_commit();
    const double* st = sbuf;  // chunk kc's stage
    uint32_t soff = 0;        // its byte offset
    frag(fa[0], fb[0], st);
    for (int kc = 0; kc < nk; kc++) {
#pragma unroll
        for (int j = 0; j < DM_BK / 4; j++) {
            const int cur = j & 1, nxt = cur ^ 1;
            if (j + 1 < DM_BK / 4) {
                frag(fa[nxt], fb[nxt], st + (j + 1) * 4);
            } else if (kc + 1 < nk) {
                // chunk kc + 1 is in once at most one group is pending; after the barrier no
                // warp reads chunk kc's stage any more, so chunk kc + 3 may replace it
                cp_async_wait<1>();
                __syncthreads();
                if (kc + 3 < nk) ld.next<BT, DM_TN>(soff);
                cp_async_commit();
                soff = soff == 2 * STB ? 0 : soff + STB;
                st = sbuf + soff / sizeof(double);
                frag(fa[nxt], fb[nxt], st);
            }
#pragma unroll
            for (int a = 0; a < 8; a++)
#pragma unroll
                for (int c = 0; c < 4; c++) dmma_884(acc[a][c][0], acc[a][c][1], fa[cur][a], fb[cur][c]);
        }
    }
    cp_async_wait<0>();
    // accumulator (a, c, e): row 64·wm + 8a + g, column 32·wn + 8c + 2q + e; F −= W·Lᵀ on the
    // lower triangle, two columns per 16-byte access where the pair is aligned and in range.
    // Two batches of 16 pairs: all loads of a batch are in flight before its first store.
#pragma unroll
    for (int h = 0; h < 2; h++) {
        double2 v[4][4];
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const int64_t r = bt.row0 + wm * 64 + (h * 4 + a) * 8 + g;
            const int64_t cend = r < f.m ? min(bt.col_end, r + 1) : 0;
            const double* rowp = r < f.m ? out_row(panel, upd, f, bt.in_panel, r) : panel;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int64_t cc = col0 + wn * 32 + c * 8 + 2 * q;
                const double* p = rowp + cc;
                if (cc + 1 < cend && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
                    v[a][c] = *reinterpret_cast<const double2*>(p);
                } else {
                    v[a][c].x = cc < cend ? p[0] : 0.0;
                    v[a][c].y = cc + 1 < cend ? p[1] : 0.0;
                }
            }
        }
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const int64_t r = bt.row0 + wm * 64 + (h * 4 + a) * 8 + g;
            if (r >= f.m) continue;
            const int64_t cend = min(bt.col_end, r + 1);
            double* rowp = out_row(panel, upd, f, bt.in_panel, r);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int64_t cc = col0 + wn * 32 + c * 8 + 2 * q;
                double* p = rowp + cc;
                const double x = v[a][c].x - acc[h * 4 + a][c][0], y = v[a][c].y - acc[h * 4 + a][c][1];
                if (cc + 1 < cend && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
                    *reinterpret_cast<double2*>(p) = make_double2(x, y);
                } else {
                    if (cc < cend) p[0] = x;
                    if (cc + 1 < cend) p[1] = y;
                }
            }
        }
    }
}

// The FP64 updates on the UT×UT grid of k_schur (inner updates, and outer updates of small
// fronts) on the FP64 tensor-core path: 128 threads, 4 warps of 32×32 outputs, K in chunks
// of 16 through a three-stage cp.async ring (the ring, pitch and fragment pipelining of
// k_schur_dmma), two or more CTAs per SM.
constexpr int D64_STAGE = 2 * UT * DM_PITCH;  // doubles per stage: W rows, then L rows
constexpr size_t D64_SMEM = (size_t)DM_STAGES * D64_STAGE * sizeof(double);

template <bool OUTER>
__global__ void __launch_bounds__(128, 2) k_schur_dmma64(double* __restrict__ panel, double* __restrict__ upd,
                                                      const DFront* __restrict__ fr,
                                                      const int64_t* __restrict__ order, int64_t fr_off, int64_t nact,
                                                      const int64_t* __restrict__ pre_tiles,
                                                      const int64_t* __restrict__ pre_a, int part,
                                                      const int64_t* __restrict__ pre_scr, int64_t s,
                                                      const double* scr_w,
                                                      const double* scr_l,
                                                      const int64_t* status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sbuf = reinterpret_cast<double*>(smem_raw);  // [stage][UT W rows | UT L rows][DM_PITCH]
    int64_t lt;
    const int64_t i = find_tile_warp(pre_tiles, pre_a, part, nact, blockIdx.x, &lt);
    const int64_t t = order[fr_off + i];
    const DFront f = fr[t];
    pdl_wait();  // before this only plan data is read, which no kernel writes
    pdl_launch_dependents();
    if (status[t] != -1) return;
    const int64_t J0 = (s / KO) * NBO;
    const SmallTile tl = small_tile<OUTER>(f, s, lt);
    // scratch row of front row r: pre_scr[i] + r − J0; the tile's pivots start at kofs
    const double* wrow = scr_w + (pre_scr[i] - J0 + tl.row0) * NBO + tl.kofs;
    const double* lrow = scr_l + (pre_scr[i] - J0 + tl.col0) * NBO + tl.kofs;
    const int klen = (int)tl.klen;
    const int nk = (klen + DM_BK - 1) / DM_BK;
    DmLoader ld(wrow, lrow, sbuf);
    constexpr uint32_t STB = D64_STAGE * sizeof(double);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int wm = warp & 1, wn = warp >> 1;  // warp tile rows [32·wm, +32), columns [32·wn, +32)
    const int aoff = (wm * 32 + g) * DM_PITCH + q, boff = (UT + wn * 32 + g) * DM_PITCH + q;
    auto frag = [&](double* fa, double* fb, const double* st) {
#pragma unroll
        for (int a = 0; a < 4; a++) fa[a] = st[aoff + a * 8 * DM_PITCH];
#pragma unroll
        for (int c = 0; c < 4; c++) fb[c] = st[boff + c * 8 * DM_PITCH];
    };
    double acc[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[a][c][0] = acc[a][c][1] = 0.0;
    double fa[2][4], fb[2][4];
    ld.next<UT, UT>(0);
    cp_async_commit();
    if (nk > 1) ld.next<UT, UT>(STB);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    if (nk > 2) ld.next<UT, UT>(2 * STB);
    cp_async_commit();
    const double* st = sbuf;
    uint32_t soff = 0;
    frag(fa[0], fb[0], st);
    for (int kc = 0; kc < nk; kc++) {
#pragma unroll
        for (int j = 0; j < DM_BK / 4; j++) {
            const int cur = j & 1, nxt = cur ^ 1;
            if (j + 1 < DM_BK / 4) {
                frag(fa[nxt], fb[nxt], st + (j + 1) * 4);
            } else if (kc + 1 < nk) {
                cp_async_wait<1>();
                __syncthreads();
                if (kc + 3 < nk) ld.next<UT, UT>(soff);
                cp_async_commit();
                soff = soff == 2 * STB ? 0 : soff + STB;
                st = sbuf + soff / sizeof(double);
                frag(fa[nxt], fb[nxt], st);
            }
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int c = 0; c < 4; c++) dmma_884(acc[a][c][0], acc[a][c][1], fa[cur][a], fb[cur][c]);
        }
    }
    cp_async_wait<0>();
    // accumulator (a, c, e): row 32·wm + 8a + g, column 32·wn + 8c + 2q + e; all loads of
    // the tile's pairs are in flight before the first store
    double2 v[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++) {
        const int64_t r = tl.row0 + wm * 32 + a * 8 + g;
        const int64_t cend = r < f.m ? min(tl.col_end, r + 1) : 0;
        const double* rowp = r < f.m ? out_row(panel, upd, f, tl.in_panel, r) : panel;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int64_t cc = tl.col0 + wn * 32 + c * 8 + 2 * q;
            const double* p = rowp + cc;
            if (cc + 1 < cend && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
                v[a][c] = *reinterpret_cast<const double2*>(p);
            } else {
                v[a][c].x = cc < cend ? p[0] : 0.0;
                v[a][c].y = cc + 1 < cend ? p[1] : 0.0;
            }
        }
    }
#pragma unroll
    for (int a = 0; a < 4; a++) {
        const int64_t r = tl.row0 + wm * 32 + a * 8 + g;
        if (r >= f.m) continue;
        const int64_t cend = min(tl.col_end, r + 1);
        double* rowp = out_row(panel, upd, f, tl.in_panel, r);
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int64_t cc = tl.col0 + wn * 32 + c * 8 + 2 * q;
            double* p = rowp + cc;
            const double x = v[a][c].x - acc[a][c][0], y = v[a][c].y - acc[a][c][1];
            if (cc + 1 < cend && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
                *reinterpret_cast<double2*>(p) = make_double2(x, y);
            } else {
                if (cc < cend) p[0] = x;
                if (cc + 1 < cend) p[1] = y;
            }
        }
    }
}

// Scatter of the caller's entries built on the device, one warp per internal column,
// the columns in level order (lcol: the column, lfront: its front). Entry p of the
// caller's column c = owner[q] is an original entry of the factorization when its
// internal row eq[row] is at least q (the positive definite factorization reads the
// internal lower triangle, ffi/src/lib.rs:216-224). k_map_count counts them per column
// and flags (bit 0) a column whose rows are not strictly increasing; k_map_fill, given
// the prefix sums of the counts, writes each entry's panel offset and source index in
// the caller's order (the order of the host lists of scatter_from_caller). A row that
// the front does not hold sets bit 1 and is sent to the column's diagonal entry.
__global__ void k_map_count(const int64_t* __restrict__ indptr, const int64_t* __restrict__ indices,
                            const int64_t* __restrict__ eq, const int64_t* __restrict__ owner,
                            const int32_t* __restrict__ lcol, int64_t ncols, int64_t* __restrict__ cnt,
                            int* __restrict__ flag, int64_t* __restrict__ diag_src) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= ncols) return;
    const int64_t q = lcol[i], c = owner[q];
    const int64_t p0 = indptr[c], p1 = indptr[c + 1];
    int64_t z = 0;
    bool bad = false;
    for (int64_t p = p0 + lane; p < p1; p += 32) {
        const int64_t r = indices[p];
        z += eq[r] >= q ? 1 : 0;
        if (p > p0 && indices[p - 1] >= r) bad = true;
        if (r == c) diag_src[q] = p;  // rows are distinct when no column is flagged
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(flag, 1);
    if (lane == 0) cnt[i] = z;
}

__global__ void k_map_fill(const int64_t* __restrict__ indptr, const int64_t* __restrict__ indices,
                           const int64_t* __restrict__ eq, const int64_t* __restrict__ owner,
                           const int32_t* __restrict__ lcol, const int32_t* __restrict__ lfront,
                           const DFront* __restrict__ fr, const int64_t* __restrict__ rows, int64_t ncols,
                           const int64_t* __restrict__ off, int64_t* __restrict__ dst, int64_t* __restrict__ src,
                           int* __restrict__ flag) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= ncols) return;
    const int64_t q = lcol[i], c = owner[q];
    const DFront f = fr[lfront[i]];
    const int64_t p0 = indptr[c], p1 = indptr[c + 1];
    const int64_t colo = q - f.start;
    int64_t base = off[i];
    for (int64_t pb = p0; pb < p1; pb += 32) {
        const int64_t p = pb + lane;
        bool keep = false;
        int64_t lr = colo;
        if (p < p1) {
            const int64_t qr = eq[indices[p]];
            keep = qr >= q;
            if (keep) {
                if (qr < f.start + f.k) {
                    lr = qr - f.start;
                } else {
                    const int64_t* rw = rows + f.rows_off;
                    int64_t lo = 0, hi = f.u;
                    while (lo < hi) {
                        const int64_t mid = (lo + hi) >> 1;
                        if (rw[mid] < qr)
                            lo = mid + 1;
                        else
                            hi = mid;
                    }
                    if (lo < f.u && rw[lo] == qr) {
                        lr = f.k + lo;
                    } else {
                        atomicOr(flag, 2);
                        lr = colo;
                    }
                }
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const int64_t o = base + __popc(m & ((1u << lane) - 1u));
            dst[o] = f.poff + lr * f.ldp + colo;
            src[o] = p;
        }
        base += __popc(m);
    }
}

// the original diagonal of every equation (FP16 split scales): the value of the caller's
// diagonal entry of its column, or 0 where that entry is not known
__global__ void k_orig_diag(const double* __restrict__ src, const int64_t* __restrict__ diag_src, int64_t n,
                            double* __restrict__ out) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = diag_src[q];
        out[q] = p >= 0 ? src[p] : 0.0;
    }
}

// imap of a front's parent: the front's row x at the parent row emap[x]
__global__ void k_imap_fill(const DFront* __restrict__ fr, const int32_t* __restrict__ emap,
                            int32_t* __restrict__ imap) {
    const int64_t c = blockIdx.x;
    const DFront f = fr[c];
    if (f.parent < 0 || f.u == 0) return;
    const DFront p = fr[f.parent];
    int32_t* m = imap + p.imap_off + (p.kid0 == c ? 0 : p.m);
    for (int64_t x = threadIdx.x; x < f.u; x += blockDim.x) m[emap[f.emap_off + x]] = (int32_t)x;
}

__global__ void k_gather_i64(const int64_t* __restrict__ a, const int64_t* __restrict__ idx, int64_t n,
                             int64_t* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = a[idx[i]];
}

template <typename T>
struct ScrType {
    using type = T;
};

}  // namespace

// ---------------------------------------------------------------------------
// Engine
// ---------------------------------------------------------------------------
void* Engine::dalloc(size_t bytes) {
    void* p = dev_alloc(bytes, stream_);
    allocs_.push_back(p);
    return p;
}

template <typename V, typename A>
static V* upload(const std::vector<V, A>& v, cudaStream_t st, std::vector<void*>& allocs, int64_t& bytes_total) {
    V* p = nullptr;
    bytes_total += (int64_t)(v.size() * sizeof(V));
    size_t bytes = std::max<size_t>(v.size() * sizeof(V), 256);
    p = (V*)dev_alloc(bytes, st);
    allocs.push_back(p);
    if (!v.empty()) host_upload(p, v.data(), v.size() * sizeof(V), st);
    return p;
}

void Engine::upload_plan() {
    auto up = [&](const auto& v) { return upload(v, stream_, allocs_, plan_bytes_); };
    dp_.fronts = up(plan_.fronts);
    dp_.level_order = up(plan_.level_order);
    dp_.pre_panel = up(plan_.pre_panel);
    dp_.pre_inner = up(plan_.pre_inner);
    dp_.pre_inner_tc = up(plan_.pre_inner_tc);
    dp_.pre_wrows = up(plan_.pre_wrows);
    dp_.pre_wpart = up(plan_.pre_wpart);
    dp_.wrow_slot = (int2*)up(plan_.wrow_slot);
    dp_.pre_outer = up(plan_.pre_outer);
    dp_.pre_outer_tc = up(plan_.pre_outer_tc);
    dp_.pre_outer_tc2 = up(plan_.pre_outer_tc2);
    dp_.pre_outer_a = up(plan_.pre_outer_a);
    dp_.pre_outer_tc_a = up(plan_.pre_outer_tc_a);
    dp_.pre_scr = up(plan_.pre_scr);
    dp_.panel_mode = up(plan_.panel_mode);
    dp_.outer_mode = up(plan_.outer_mode);
    dp_.asm_pre = up(plan_.asm_pre);
    dp_.rows = up(plan_.rows);
    dp_.emap = up(plan_.emap);
    dp_.chain_blk = up(plan_.chain_blk);
    dp_.chain_bfront = up(plan_.chain_bfront);
    dp_.chain_fwd = up(plan_.chain_fwd);
    dp_.chain_bwd = up(plan_.chain_bwd);
    dp_.chain_rows = up(plan_.chain_rows);
    dp_.chain_cols = up(plan_.chain_cols);
    dp_.chain_colbase = up(plan_.chain_colbase);
    dp_.blk_width = up(plan_.blk_width);
}

// The host scatter lists on the device; the host copies of the per-entry lists are
// released (only the level and front offsets stay on the host).
void Engine::upload_scatter() {
    auto up = [&](const auto& v) { return upload(v, stream_, allocs_, plan_bytes_); };
    nseg_ = (int64_t)scatter_.dst.size();
    dp_.seg_dst = up(scatter_.dst);
    bool single = (int64_t)scatter_.src.size() == (int64_t)scatter_.dst.size();
    dp_.seg_ptr = single ? nullptr : up(scatter_.seg_ptr);
    dp_.seg_src = up(scatter_.src);
    dp_.front_seg = up(scatter_.front_seg);
    SegVec().swap(scatter_.dst);
    SegVec().swap(scatter_.src);
    std::vector<int64_t>().swap(scatter_.seg_ptr);
}

void Engine::build_scatter_device(const CallerPattern& cp) {
    const Plan& P = plan_;
    const std::vector<int64_t>& eq = *cp.eq;
    const int64_t N = cp.ncaller, nnz = N > 0 ? cp.indptr[N] : 0, n = P.n;
    // the internal columns in level order and their fronts; the position of each front's
    // first column
    std::vector<int32_t> lcol(std::max<int64_t>(n, 1)), lfront(std::max<int64_t>(n, 1));
    std::vector<int64_t> fpos(P.nfronts + 1, 0);
    {
        int64_t o = 0;
        for (int64_t j = 0; j < P.nfronts; j++) {
            const int64_t t = P.level_order[j];
            const DFront& d = P.fronts[t];
            fpos[j] = o;
            for (int64_t q = d.start; q < d.start + d.k; q++) {
                lcol[o] = (int32_t)q;
                lfront[o] = (int32_t)t;
                o++;
            }
        }
        fpos[P.nfronts] = o;
        if (o != n) throw CudaError("build_scatter_device: the fronts do not cover the equations");
    }
    std::vector<int64_t> owner(std::max<int64_t>(n, 1), 0);
    for (int64_t i = 0; i < N; i++)
        if (eq[i] >= 0) owner[eq[i]] = i;
    // work buffers: the update arena when it is large enough (unused before the first
    // numeric phase)
    auto r256 = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t nc1 = (size_t)n + 1;
    const size_t nind = cp.indices_dev ? 1 : (size_t)std::max<int64_t>(nnz, 1);
    const size_t need = r256(nind * 8) + r256(((size_t)N + 1) * 8) +
                        r256((size_t)std::max<int64_t>(N, 1) * 8) + r256(nc1 * 8) + 2 * r256(nc1 * 4) +
                        r256(nc1 * 8) + r256((size_t)scan_tmp_elems((int64_t)nc1) * 8) +
                        r256(((size_t)P.nfronts + 1) * 8) + r256(4) + 256;
    const size_t es = prec_ == PREC_FP64 ? sizeof(double) : sizeof(float);
    const bool in_arena = (size_t)P.upd_elems * es >= need;
    char* base = in_arena ? (char*)upd_ : (char*)dev_alloc(need, stream_);
    char* w = base;
    auto carve = [&](size_t bytes) {
        char* r = w;
        w += r256(bytes);
        return r;
    };
    int64_t* d_ind = (int64_t*)carve(nind * 8);
    int64_t* d_ptr = (int64_t*)carve(((size_t)N + 1) * 8);
    int64_t* d_eq = (int64_t*)carve((size_t)std::max<int64_t>(N, 1) * 8);
    int64_t* d_owner = (int64_t*)carve(nc1 * 8);
    int32_t* d_lcol = (int32_t*)carve(nc1 * 4);
    int32_t* d_lfront = (int32_t*)carve(nc1 * 4);
    int64_t* d_off = (int64_t*)carve(nc1 * 8);
    int64_t* d_stmp = (int64_t*)carve((size_t)scan_tmp_elems((int64_t)nc1) * 8);
    int64_t* d_fpos = (int64_t*)carve(((size_t)P.nfronts + 1) * 8);
    int* d_flag = (int*)carve(4);
    if ((size_t)(w - base) > need) throw CudaError("build_scatter_device: work buffer layout");
    const int64_t* ind = d_ind;
    if (cp.indices_dev) {
        ind = cp.indices_dev;
        if (cp.wait_indices) cp.wait_indices((void*)stream_);
    } else if (nnz > 0) {
        host_upload(d_ind, cp.indices, (size_t)nnz * 8, stream_);
    }
    host_upload(d_ptr, cp.indptr, ((size_t)N + 1) * 8, stream_);
    if (N > 0) host_upload(d_eq, eq.data(), (size_t)N * 8, stream_);
    host_upload(d_owner, owner.data(), (size_t)n * 8, stream_);
    host_upload(d_lcol, lcol.data(), (size_t)n * 4, stream_);
    host_upload(d_lfront, lfront.data(), (size_t)n * 4, stream_);
    host_upload(d_fpos, fpos.data(), ((size_t)P.nfronts + 1) * 8, stream_);
    RFG_CUDA(cudaMemsetAsync(d_flag, 0, 4, stream_));
    RFG_CUDA(cudaMemsetAsync(d_off + n, 0, 8, stream_));
    const unsigned wblocks = (unsigned)std::max<int64_t>(1, (n * 32 + 255) / 256);
    diag_src_ = (int64_t*)dalloc((size_t)std::max<int64_t>(n, 1) * 8);
    RFG_CUDA(cudaMemsetAsync(diag_src_, 0xff, (size_t)std::max<int64_t>(n, 1) * 8, stream_));
    if (n > 0)
        k_map_count<<<wblocks, 256, 0, stream_>>>(d_ptr, ind, d_eq, d_owner, d_lcol, n, d_off, d_flag, diag_src_);
    exclusive_scan_i64(d_off, (int64_t)nc1, d_stmp, stream_);
    int64_t total = 0;
    int flag = 0;
    RFG_CUDA(cudaMemcpyAsync(&total, d_off + n, 8, cudaMemcpyDeviceToHost, stream_));
    RFG_CUDA(cudaMemcpyAsync(&flag, d_flag, 4, cudaMemcpyDeviceToHost, stream_));
    RFG_CUDA(cudaStreamSynchronize(stream_));
    plan_bytes_ += (int64_t)((cp.indices_dev ? 0 : (size_t)nnz * 8) + ((size_t)N + 1) * 8 + (size_t)N * 8 +
                             (size_t)n * 16 + ((size_t)P.nfronts + 1) * 8);
    if (flag & 1) {
        // a column with unsorted or repeated rows: the host lists (duplicates summed); the
        // diagonal sources are not known, so the tensor cores keep the TF32 split
        diag_src_ = nullptr;
        if (!in_arena) dev_free(base, stream_);
        scatter_ = scatter_from_caller(P, *cp.sym, N, cp.indptr, cp.indices, eq);
        upload_scatter();
        return;
    }
    nseg_ = total;
    dp_.seg_dst = (int64_t*)dalloc((size_t)std::max<int64_t>(total, 1) * 8);
    dp_.seg_src = (int64_t*)dalloc((size_t)std::max<int64_t>(total, 1) * 8);
    dp_.seg_ptr = nullptr;
    dp_.front_seg = (int64_t*)dalloc(((size_t)P.nfronts + 1) * 8);
    if (n > 0)
        k_map_fill<<<wblocks, 256, 0, stream_>>>(d_ptr, ind, d_eq, d_owner, d_lcol, d_lfront, dp_.fronts, dp_.rows,
                                                 n, d_off, dp_.seg_dst, dp_.seg_src, d_flag);
    k_gather_i64<<<(unsigned)((P.nfronts + 256) / 256), 256, 0, stream_>>>(d_off, d_fpos, P.nfronts + 1,
                                                                           dp_.front_seg);
    RFG_CUDA(cudaGetLastError());
    scatter_.front_seg.assign(P.nfronts + 1, 0);
    RFG_CUDA(cudaMemcpyAsync(scatter_.front_seg.data(), dp_.front_seg, ((size_t)P.nfronts + 1) * 8,
                             cudaMemcpyDeviceToHost, stream_));
    RFG_CUDA(cudaMemcpyAsync(&flag, d_flag, 4, cudaMemcpyDeviceToHost, stream_));
    if (!in_arena) dev_free(base, stream_);
    RFG_CUDA(cudaStreamSynchronize(stream_));
    if (flag & 2) throw CudaError("build_scatter_device: an entry's row is not in its front (symbolic mismatch)");
}

Engine::Engine(Plan&& plan, Scatter&& scatter, int64_t nsrc, Precision prec, bool use_tc)
    : plan_(std::move(plan)), scatter_(std::move(scatter)), nsrc_(nsrc), prec_(prec),
      use_tc_(use_tc && prec == PREC_MIXED) {
    RFG_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    RFG_CUDA(cudaEventCreate(&ev0_));
    RFG_CUDA(cudaEventCreate(&ev1_));
    upload_plan();
    upload_scatter();
    init(use_tc);
}

Engine::Engine(Plan&& plan, const CallerPattern& pattern, int64_t nsrc, Precision prec, bool use_tc)
    : plan_(std::move(plan)), nsrc_(nsrc), prec_(prec), use_tc_(use_tc && prec == PREC_MIXED) {
    RFG_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    RFG_CUDA(cudaEventCreate(&ev0_));
    RFG_CUDA(cudaEventCreate(&ev1_));
    upload_plan();
    // the arenas first: the pattern is mapped in the (still unused) update arena
    size_t es = prec_ == PREC_FP64 ? sizeof(double) : sizeof(float);
    panel_ = dalloc(plan_.panel_elems * es);
    upd_ = dalloc(plan_.upd_elems * es);
    build_scatter_device(pattern);
    init(use_tc);
}

void Engine::init(bool) {
    set_attributes();
    size_t es = prec_ == PREC_FP64 ? sizeof(double) : sizeof(float);
    if (!panel_) panel_ = dalloc(plan_.panel_elems * es);
    if (!upd_) upd_ = dalloc(plan_.upd_elems * es);
    // FP64: two buffers, alternating with the parity of the outer block (a block's operands are
    // still read beside the next block's steps)
    const int64_t nscr = prec_ == PREC_FP64 ? 2 : 1;
    const int64_t scr_elems = (nscr * std::max<int64_t>(plan_.max_scr_rows, 1) + DM_SPARE) * NBO;
    scr_w_ = dalloc(scr_elems * es);
    scr_l_ = dalloc(scr_elems * es);
    if (prec_ == PREC_FP64) {
        int least = 0;
        RFG_CUDA(cudaDeviceGetStreamPriorityRange(&least, &high_prio_));
        RFG_CUDA(cudaStreamCreateWithFlags(&side_, cudaStreamNonBlocking));
        RFG_CUDA(cudaEventCreateWithFlags(&ev_fork_, cudaEventDisableTiming));
        RFG_CUDA(cudaEventCreateWithFlags(&ev_join_, cudaEventDisableTiming));
    }
    d_ = (double*)dalloc(std::max<int64_t>(plan_.n, 1) * sizeof(double));
    linv_ = (double*)dalloc(std::max<int64_t>(plan_.nblocks, 1) * NB * NB * sizeof(double));
    if (plan_.nblocks > 0) {
        k_slot_identity<<<(unsigned)plan_.nblocks, 256, 0, stream_>>>(linv_);
        RFG_CUDA(cudaGetLastError());
    }
    if (plan_.chain_blocks > 0) {
        if (prec_ == PREC_MIXED)
            chain_inv_ = (double*)dalloc(plan_.chain_blocks * (int64_t)WS * WS * sizeof(double));
        chain_err_ = (int*)dalloc(sizeof(int));
        RFG_CUDA(cudaMemsetAsync(chain_err_, 0, sizeof(int), stream_));
    }
    adiag_ = (double*)dalloc(std::max<int64_t>(plan_.n, 1) * sizeof(double));
    status_ = (int64_t*)dalloc(std::max<int64_t>(plan_.nfronts, 1) * sizeof(int64_t));
    src_ = (double*)dalloc(std::max<int64_t>(nsrc_, 1) * sizeof(double));
    {
        // the FP64 matrix of the refinement (CSR in the internal numbering, built by the
        // first refined solve), sized for every scattered entry and its mirror
        const int64_t cap = std::max<int64_t>(2 * nseg_, 1);
        a_rowptr_ = (int64_t*)dalloc((plan_.n + 1) * sizeof(int64_t));
        a_col_ = (int32_t*)dalloc(cap * sizeof(int32_t));
        a_src_ = (uint32_t*)dalloc(cap * sizeof(uint32_t));
        a_val_ = (double*)dalloc(cap * sizeof(double));
    }
    if (use_tc_) {
        // the split operands in two buffers, alternating with the parity of the outer block
        // (a block's operands stay readable while the next block's panels are written)
        size_t sz = 2 * std::max<int64_t>(plan_.max_scr_rows, 1) * NBO * sizeof(float);
        scr_whi_ = dalloc(sz);
        scr_wlo_ = dalloc(sz);
        scr_lhi_ = dalloc(sz);
        scr_llo_ = dalloc(sz);
        RFG_CUDA(cudaMemsetAsync(scr_whi_, 0, sz, stream_));
        RFG_CUDA(cudaMemsetAsync(scr_wlo_, 0, sz, stream_));
        RFG_CUDA(cudaMemsetAsync(scr_lhi_, 0, sz, stream_));
        RFG_CUDA(cudaMemsetAsync(scr_llo_, 0, sz, stream_));
        const size_t hz = 2 * std::max<int64_t>(plan_.max_scr_rows, 1) * NBO * 2;
        scr_uhi_ = dalloc(hz);
        scr_ulo_ = dalloc(hz);
        scr_uscale_ = dalloc(std::max<int64_t>(plan_.max_scr_rows, 1) * sizeof(float));
        RFG_CUDA(cudaMemsetAsync(scr_uhi_, 0, hz, stream_));
        RFG_CUDA(cudaMemsetAsync(scr_ulo_, 0, hz, stream_));
        RFG_CUDA(cudaMemsetAsync(scr_uscale_, 0, std::max<int64_t>(plan_.max_scr_rows, 1) * sizeof(float), stream_));
        adiag0_ = (double*)dalloc(std::max<int64_t>(plan_.n, 1) * sizeof(double));
        setup_tc();
    }
    // the child row of each front row, for either child: the inverse of emap, on the device
    dp_.imap = (int32_t*)dalloc(std::max<int64_t>(plan_.imap_elems, 1) * sizeof(int32_t));
    RFG_CUDA(cudaMemsetAsync(dp_.imap, 0xff, std::max<int64_t>(plan_.imap_elems, 1) * sizeof(int32_t), stream_));
    if (plan_.nfronts > 0) {
        k_imap_fill<<<(unsigned)plan_.nfronts, 128, 0, stream_>>>(dp_.fronts, dp_.emap, dp_.imap);
        RFG_CUDA(cudaGetLastError());
    }
    RFG_CUDA(cudaStreamSynchronize(stream_));
}

void Engine::set_attributes() {
    RFG_CUDA(cudaFuncSetAttribute(k_schur_dmma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DM_SMEM));
    RFG_CUDA(cudaFuncSetAttribute(k_schur_dmma64<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)D64_SMEM));
    RFG_CUDA(cudaFuncSetAttribute(k_schur_dmma64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)D64_SMEM));
    RFG_CUDA(cudaFuncSetAttribute(k_schur_big<float, float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)big_smem<float>()));
    RFG_CUDA(cudaFuncSetAttribute(k_panel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PANEL_SMEM));
    RFG_CUDA(cudaFuncSetAttribute(k_panel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PANEL_SMEM));
    RFG_CUDA(cudaFuncSetAttribute(k_pivot_block<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PB_SMEM));
    RFG_CUDA(cudaFuncSetAttribute(k_pivot_block<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PB_SMEM));
    RFG_CUDA(cudaFuncSetAttribute(k_block_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BI_SMEM));
    const size_t s32 = 2 * NB * (UT + 1) * sizeof(float);
    RFG_CUDA(cudaFuncSetAttribute(k_schur<float, float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s32));
    RFG_CUDA(cudaFuncSetAttribute(k_schur<float, float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s32));
}

int Engine::tc_error() const {
    if (!tc_err_) return 0;
    int e = 0;
    RFG_CUDA(cudaMemcpy(&e, tc_err_, sizeof(int), cudaMemcpyDeviceToHost));
    return e;
}

Engine::~Engine() {
    if (stream_) cudaStreamSynchronize(stream_);
    for (cudaGraphExec_t& g : factor_graph_)
        if (g) cudaGraphExecDestroy(g);
    for (auto& g : solve_graphs_) cudaGraphExecDestroy(g.exec);
    for (cudaEvent_t e : prof_ev_) cudaEventDestroy(e);
    for (void* p : allocs_) dev_free(p, stream_);
    for (void* p : {(void*)ref_r_, (void*)ref_dx_, (void*)ref_red_}) dev_free(p, stream_);
    if (stream_) cudaStreamSynchronize(stream_);
    if (side_) cudaStreamDestroy(side_);
    for (cudaEvent_t e : {ev_fork_, ev_join_, ev0_})
        if (e) cudaEventDestroy(e);
    if (ev1_) cudaEventDestroy(ev1_);
    if (stream_) cudaStreamDestroy(stream_);
}

void Engine::pivots_to_host(double* out) const {
    RFG_CUDA(cudaMemcpyAsync(out, d_, plan_.n * sizeof(double), cudaMemcpyDeviceToHost, stream_));
    RFG_CUDA(cudaStreamSynchronize(stream_));
}

// CTAs of an outer update's rest from which it runs beside the next block's steps: one per SM
// (thresholds of 40 and 600 measured the same; below, the rest is shorter than the fork and join).
// A 64-pivot step is a chain of three launches of a few CTAs, about 33 µs, and four of them wait
// for each outer update; a factorization takes, with the rest on the one stream and beside the steps,
// 3.42 and 3.33 ms at 22³, 17.22 and 16.47 at 33³, 71.6 and 70.6 at 45³, 336.3 and 334.7 at 60³. (One
// CTA per SM for the rest, which leaves half of every SM to the steps, was slower: 88 against 71 ms at
// 45³.)
constexpr int64_t AHEAD_MIN_CTAS = 148;

template <typename T>
void Engine::factor_impl() {
    using S = typename ScrType<T>::type;
    T* panel = (T*)panel_;
    T* upd = (T*)upd_;
    S* const sw0 = (S*)scr_w_;
    S* const sl0 = (S*)scr_l_;
    const Plan& P = plan_;
    int64_t launches = 0;
    size_t schur_smem = 2 * NB * (UT + 1) * sizeof(S);
    int64_t nprof = 0;
    prof_phase_.clear();
    // PROF_SKIP: the interval before a 128-tile outer update at profiling level 2 (not counted)
    constexpr int PROF_SKIP = 7;
    auto mark = [&](int phase, cudaStream_t on = nullptr) {
        // an event after each launch; the time since the previous event goes to its phase
        // (level 2: only the events around the 128-tile outer updates)
        if (!profile_) return;
        if (profile_ == 2 && phase != 6 && phase != PROF_SKIP) return;
        if (profile_ == 1 && phase == PROF_SKIP) return;
        if (prof_ev_.size() <= prof_phase_.size() + 1) {
            cudaEvent_t e;
            RFG_CUDA(cudaEventCreate(&e));
            prof_ev_.push_back(e);
        }
        // external: under stream capture the record becomes an event-record node of the graph
        RFG_CUDA(cudaEventRecordWithFlags(prof_ev_[prof_phase_.size() + 1], on ? on : stream_, cudaEventRecordExternal));
        prof_phase_.push_back(phase);
    };
    if (profile_) {
        if (prof_ev_.empty()) {
            cudaEvent_t e;
            RFG_CUDA(cudaEventCreate(&e));
            prof_ev_.push_back(e);
        }
        RFG_CUDA(cudaEventRecordWithFlags(prof_ev_[0], stream_, cudaEventRecordExternal));
    }
    RFG_CUDA(cudaMemsetAsync(status_, 0xff, std::max<int64_t>(P.nfronts, 1) * sizeof(int64_t), stream_));
    RFG_CUDA(cudaMemsetAsync(d_, 0, std::max<int64_t>(P.n, 1) * sizeof(double), stream_));
    if (h16_ && P.n > 0) {
        // RFG_TC_H16_FALLBACK_TEST: no diagonal, so that every row reports an invalid scale
        // and the engine takes its TF32 fallback (tests of that path)
        const bool fail_test = getenv("RFG_TC_H16_FALLBACK_TEST") != nullptr;
        if (fail_test) {
            RFG_CUDA(cudaMemsetAsync(adiag0_, 0, P.n * sizeof(double), stream_));
        } else {
            k_orig_diag<<<(unsigned)std::min<int64_t>((P.n + 255) / 256, 148 * 8), 256, 0, stream_>>>(
                (const double*)src_, (const int64_t*)diag_src_, P.n, adiag0_);
            launches++;
        }
    }
    if (P.panel_elems > 0) RFG_CUDA(cudaMemsetAsync(panel, 0, P.panel_elems * sizeof(T), stream_));
    mark(0);
    if (nseg_ > 0) {
        const int64_t nb = std::min<int64_t>((nseg_ + 255) / 256, 148 * 16);
        launch_pdl(true, k_scatter<T>, dim3((unsigned)nb), dim3(256), 0, stream_, panel, (const double*)src_,
                   (const int64_t*)dp_.seg_dst, (const int64_t*)dp_.seg_ptr, (const int64_t*)dp_.seg_src, (int64_t)0,
                   nseg_);
        launches++;
        mark(0);
    }
    if (P.nfronts > 0) {
        launch_pdl(true, k_capture_diag<T>, dim3((unsigned)P.nfronts), dim3(128), 0, stream_, (const T*)panel, adiag_,
                   (const DFront*)dp_.fronts, (const int64_t*)dp_.level_order, (int64_t)0);
        launches++;
        mark(0);
    }
    // Look-ahead (FP64): the part of an outer update that the next outer block's steps do not read
    // runs beside them on the side stream; the steps' launches go first wherever a CTA leaves an SM.
    // (With profiling on the launches are timed one after another.)
    const bool use_ahead = side_ != nullptr && profile_ == 0;
    const int prio = use_ahead ? high_prio_ : 0;
    int64_t ahead = -1;  // the outer block whose update is on the side stream
    bool pdl = true;     // false for the launch that follows a wait for the side stream
    auto join = [&] {
        if (ahead < 0) return;
        RFG_CUDA(cudaStreamWaitEvent(stream_, ev_join_, 0));
        ahead = -1;
        pdl = false;
    };
    auto overlap = [&] {
        const bool p = pdl;
        pdl = true;
        return p;
    };
    for (int64_t l = 0; l < P.nlevels; l++) {
        const int64_t lo = P.level_off[l], nl = P.level_off[l + 1] - lo;
        if (nl == 0) continue;
        if (P.asm_blocks[l] > 0) {
            launch_pdl(overlap(), k_assemble<T>, dim3((unsigned)P.asm_blocks[l]), dim3(256), 0, stream_, panel, upd,
                       (const DFront*)dp_.fronts, (const int64_t*)(dp_.level_order + lo),
                       (const int64_t*)(dp_.asm_pre + lo + l), nl, (const int32_t*)dp_.imap, status_);
            launches++;
            mark(1);
        }
        for (int64_t si = P.step_off[l]; si < P.step_off[l + 1]; si++) {
            const DStep& st = P.steps[si];
            // this outer block's W and L operands
            const int64_t sb = sizeof(T) == 8 ? ((st.s / KO) & 1) * std::max<int64_t>(P.max_scr_rows, 1) * NBO : 0;
            S* const sw = sw0 + sb;
            S* const sl = sl0 + sb;
            if (ahead >= 0 && st.s / KO >= ahead + 2) join();  // the buffer is about to be written again
            launch_pdl_prio(prio, overlap(), k_pivot_block<T>, dim3((unsigned)st.nact), dim3(PBT), PB_SMEM, stream_, panel, d_,
                       (const double*)adiag_, (const DFront*)dp_.fronts, (const int64_t*)dp_.level_order, st.fr_off,
                       st.s, status_, linv_);
            launches++;
            mark(2);
            if (st.n_panel > 0) {
                // this outer block's buffer of the split operands
                const int64_t so = use_tc_ ? ((st.s / KO) & 1) * std::max<int64_t>(plan_.max_scr_rows, 1) * NBO : 0;
                launch_pdl_prio(prio, true, k_panel<T>, dim3((unsigned)st.n_panel), dim3(PNT),
                           PANEL_SMEM, stream_, panel, (const double*)d_,
                           (const double*)linv_, (const DFront*)dp_.fronts, (const int64_t*)dp_.level_order, st.fr_off,
                           st.nact, (const int64_t*)(dp_.pre_panel + st.pre_off),
                           (const int64_t*)(dp_.pre_scr + st.scr_off), st.s, sw, sl, (const int64_t*)status_,
                           h16_ ? (float*)nullptr : (float*)scr_whi_ + so, (float*)scr_wlo_ + so,
                           (float*)scr_lhi_ + so, (float*)scr_llo_ + so,
                           (const uint8_t*)(dp_.panel_mode + st.pre_off), (const int64_t*)dp_.rows,
                           (const double*)adiag0_, h16_ ? (__half*)scr_uhi_ + so : (__half*)nullptr,
                           (__half*)scr_ulo_ + so, (float*)scr_uscale_,
                           tc_err_);
                launches++;
                mark(3);
            }
            if (st.n_inner > 0) {
                if constexpr (sizeof(T) == 8)
                    launch_pdl_prio(prio, true, k_schur_dmma64<false>, dim3((unsigned)st.n_inner), dim3(128), D64_SMEM,
                               stream_,
                               panel, upd, (const DFront*)dp_.fronts, (const int64_t*)dp_.level_order, st.fr_off,
                               st.nact, (const int64_t*)(dp_.pre_inner + st.pre_off), (const int64_t*)nullptr, 0,
                               (const int64_t*)(dp_.pre_scr + st.scr_off), st.s, (const double*)sw, (const double*)sl,
                               (const int64_t*)status_);
                else
                    launch_pdl(true, k_schur<T, S, false>, dim3((unsigned)st.n_inner), dim3(256), schur_smem, stream_,
                               panel, upd, (const DFront*)dp_.fronts, (const int64_t*)dp_.level_order, st.fr_off,
                               st.nact, (const int64_t*)(dp_.pre_inner + st.pre_off),
                               (const int64_t*)(dp_.pre_scr + st.scr_off), st.s, (const S*)sw, (const S*)sl,
                               (const int64_t*)status_);
                launches++;
                mark(4);
            }
            if (st.n_inner_tc > 0 && use_tc_) {
                launch_schur_tc_inner(st);
                launches++;
                mark(4);
            }
            if (st.n_outer + st.n_outer_tc > 0) {
                if constexpr (sizeof(T) == 8) {
                    // Two outer blocks' updates of one front must follow each other. The tiles of the next
                    // block's columns (part 1) keep the steps waiting; the rest (part 2), when a launch of it
                    // fills the GPU and steps follow, runs on the side stream beside them.
                    const int64_t rest = 2 * (st.n_outer_tc - st.n_outer_tc_a) + (st.n_outer - st.n_outer_a);
                    const bool split = use_ahead && si + 1 < P.step_off[l + 1] && rest >= AHEAD_MIN_CTAS;
                    join();
                    auto outer = [&](int part, cudaStream_t on, int pr, bool chained) {
                        auto cnt = [&](int64_t all, int64_t a) { return part == 0 ? all : part == 1 ? a : all - a; };
                        const int64_t n64 = cnt(st.n_outer, st.n_outer_a), n128 = cnt(st.n_outer_tc, st.n_outer_tc_a);
                        if (n64 > 0) {
                            launch_pdl_prio(pr, chained, k_schur_dmma64<true>, dim3((unsigned)n64), dim3(128), D64_SMEM, on,
                                            panel, upd, (const DFront*)dp_.fronts, (const int64_t*)dp_.level_order,
                                            st.fr_off, st.nact, (const int64_t*)(dp_.pre_outer + st.pre_off),
                                            (const int64_t*)(dp_.pre_outer_a + st.pre_off), part,
                                            (const int64_t*)(dp_.pre_scr + st.scr_off), st.s, (const double*)sw,
                                            (const double*)sl, (const int64_t*)status_);
                            chained = true;
                            launches++;
                            mark(5, on);
                        }
                        if (n128 > 0) {
                            mark(PROF_SKIP, on);
                            launch_pdl_prio(pr, chained, k_schur_dmma, dim3((unsigned)(2 * n128)), dim3(DM_THREADS), DM_SMEM,
                                            on, panel, upd, (const DFront*)dp_.fronts, (const int64_t*)dp_.level_order,
                                            st.fr_off, st.nact, (const int64_t*)(dp_.pre_outer_tc + st.pre_off),
                                            (const int64_t*)(dp_.pre_outer_tc_a + st.pre_off), part,
                                            (const int64_t*)(dp_.pre_scr + st.scr_off), st.s, (const double*)sw,
                                            (const double*)sl, (const int64_t*)status_);
                            launches++;
                            mark(6, on);
                            nprof += profile_ ? 1 : 0;
                        }
                    };
                    if (split) {
                        RFG_CUDA(cudaEventRecord(ev_fork_, stream_));
                        if (st.n_outer_a + st.n_outer_tc_a > 0) outer(1, stream_, prio, overlap());
                        RFG_CUDA(cudaStreamWaitEvent(side_, ev_fork_, 0));
                        outer(2, side_, 0, false);
                        RFG_CUDA(cudaEventRecord(ev_join_, side_));
                        ahead = st.s / KO;
                    } else {
                        outer(0, stream_, prio, overlap());
                    }
                } else {
                    if (st.n_outer > 0) {
                        launch_pdl(true, k_schur<T, S, true>, dim3((unsigned)st.n_outer), dim3(256), schur_smem,
                                   stream_, panel, upd, (const DFront*)dp_.fronts, (const int64_t*)dp_.level_order,
                                   st.fr_off, st.nact, (const int64_t*)(dp_.pre_outer + st.pre_off),
                                   (const int64_t*)(dp_.pre_scr + st.scr_off), st.s, (const S*)sw, (const S*)sl,
                                   (const int64_t*)status_);
                        launches++;
                        mark(5);
                    }
                    if (st.n_outer_tc > 0) {
                        mark(PROF_SKIP);
                        if (use_tc_)
                            launch_schur_tc(st);
                        else
                            launch_pdl(true, k_schur_big<T, S>, dim3((unsigned)st.n_outer_tc), dim3(256), big_smem<S>(),
                                       stream_, panel, upd, (const DFront*)dp_.fronts, (const int64_t*)dp_.level_order,
                                       st.fr_off, st.nact, (const int64_t*)(dp_.pre_outer_tc + st.pre_off),
                                       (const int64_t*)(dp_.pre_scr + st.scr_off), st.s, (const S*)sw, (const S*)sl,
                                       (const int64_t*)status_);
                        launches++;
                        mark(6);
                        nprof += profile_ ? 1 : 0;
                    }
                }
            }
        }
        join();
    }
    if (P.nblocks > 0) {
        launch_pdl(true, k_block_inverse, dim3((unsigned)P.nblocks), dim3(128), BI_SMEM, stream_, linv_,
                   (const uint8_t*)dp_.blk_width);
        launches++;
        mark(2);
    }
    RFG_CUDA(cudaGetLastError());
    last_factor.launches = launches;
    last_factor.schur_launches = nprof;
}

int64_t Engine::factor(const double* src, bool on_device) {
    if (nsrc_ > 0) {
        if (on_device)
            RFG_CUDA(cudaMemcpyAsync(src_, src, nsrc_ * sizeof(double), cudaMemcpyDeviceToDevice, stream_));
        else
            host_upload(src_, src, nsrc_ * sizeof(double), stream_);
    }
    RFG_CUDA(cudaEventRecord(ev0_, stream_));
    // The first numeric phase of an engine is launched directly: a handle that is factored
    // once (and freed) would not win back the cost of capturing and instantiating the
    // graph. Later calls capture it once and replay it.
    const bool direct = factor_calls_++ == 0 && !factor_graph_[profile_];
    if (use_graphs_ && !direct) {
        // with profiling on, the phase events are recorded by event nodes of the graph
        cudaGraphExec_t& ex = factor_graph_[profile_];
        if (!ex) {
            cudaGraph_t g;
            RFG_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
            if (prec_ == PREC_FP64)
                factor_impl<double>();
            else
                factor_impl<float>();
            RFG_CUDA(cudaStreamEndCapture(stream_, &g));
            RFG_CUDA(cudaGraphInstantiate(&ex, g, 0));
            RFG_CUDA(cudaGraphDestroy(g));
            prof_phase_graph_[profile_] = prof_phase_;
        }
        prof_phase_ = prof_phase_graph_[profile_];
        RFG_CUDA(cudaGraphLaunch(ex, stream_));
    } else if (prec_ == PREC_FP64) {
        factor_impl<double>();
    } else {
        factor_impl<float>();
    }
    RFG_CUDA(cudaEventRecord(ev1_, stream_));
    std::vector<int64_t> st(plan_.nfronts);
    if (plan_.nfronts > 0)
        RFG_CUDA(cudaMemcpyAsync(st.data(), status_, plan_.nfronts * sizeof(int64_t), cudaMemcpyDeviceToHost, stream_));
    int tc_err = 0;
    if (tc_err_) RFG_CUDA(cudaMemcpyAsync(&tc_err, tc_err_, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    RFG_CUDA(cudaStreamSynchronize(stream_));
    if (tc_err == 21 && h16_) {
        // a row of the FP16 split left its range (a front whose diagonal no longer bounds
        // its rows, e.g. after heavy cancellation): this engine factors with the TF32 split
        h16_ = false;
        RFG_CUDA(cudaMemsetAsync(tc_err_, 0, sizeof(int), stream_));
        for (cudaGraphExec_t& g : factor_graph_)
            if (g) {
                RFG_CUDA(cudaGraphExecDestroy(g));
                g = nullptr;
            }
        return factor(src, on_device);
    }
    if (tc_err)
        throw CudaError("tensor-core Schur update: a bounded wait gave up (code " + std::to_string(tc_err) +
                        "); the factor is invalid");
    float ms = 0.f;
    RFG_CUDA(cudaEventElapsedTime(&ms, ev0_, ev1_));
    last_factor.t_factor_ms = ms;
    last_factor.schur_ms = 0.0;
    last_factor.schur_flops = plan_.outer_big_flops;
    last_factor.schur_entries = plan_.outer_big_entries;
    last_factor.schur_opvals = plan_.outer_big_opvals;
    last_factor.h2d_bytes = on_device ? 0 : nsrc_ * (int64_t)sizeof(double);
    for (double& v : last_factor.phase_ms) v = 0.0;
    for (size_t i = 0; i < prof_phase_.size(); i++) {
        float e = 0.f;
        RFG_CUDA(cudaEventElapsedTime(&e, prof_ev_[i], prof_ev_[i + 1]));
        if (prof_phase_[i] < 7) last_factor.phase_ms[prof_phase_[i]] += e;
    }
    last_factor.schur_ms = last_factor.phase_ms[6];
    // the first failing front in postorder among those whose subtree was factored
    for (int64_t t = 0; t < plan_.nfronts; t++)
        if (st[t] >= 0) return st[t];
    return -1;
}

}  // namespace rfg
