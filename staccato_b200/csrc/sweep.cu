// Frequency-sweep kernels: fused assembly + partial-pivot complex LU + solve (+ refinement).
//
// One CTA owns one (ROM, frequency) system at a time and pulls the next one from a work
// counter (persistent launch; the host orders the work list largest systems first).
//
// Storage: the matrix lives in a per-CTA scratch slot (L2-resident while in flight); blocked
// right-looking LU.  The NB-column panel is staged in shared memory and factored by all warps with
// one CTA barrier per column: row interchanges are tracked as a logical permutation, so no row is
// physically moved while the column is being searched.  After the panel, every warp independently
// processes its own groups of CW trailing columns: apply the panel's interchanges, solve the
// unit-lower triangle for the U rows (warp shuffles), and update the remaining rows with
// register-tiled complex FMAs.  No CTA barrier separates the column groups.  FP64 sweeps run on
// sweep_lu64.cu (orders up to 512) and sweep_large.cu (above); the FP64 instances here re-solve the
// mixed form's non-converged systems of orders above 512, whose number only the device knows, and, with
// matrix and right-hand sides whole in shared memory, solve the smallest orders in FP64 where that is
// the faster form (fp64_smem_faster).
//
// Precision forms
//   FP64  (double2): reproduces LAPACK zgetrf/zgetrs as restated in the oracle bit for bit:
//          IZAMAX pivots (largest |re|+|im|, smallest row index on ties) and every entry
//          updated in increasing pivot-column order with the same fused multiply-adds.
//   MIXED (float2 factors, NB = 32): the FP64-assembled matrix is rounded to complex FP32
//          and factored; the solution is refined with residuals r = b - A(w) x computed in
//          FP64 from K, M, D on the fly (the same assembly arithmetic) and corrections solved
//          with the FP32 factors (back substitution by the reciprocals of U's diagonal), until
//          the predicted error rho * ||d_s|| / ||x||, rho = 2 ||d_s|| / ||d_s-1|| the observed
//          contraction, is at most tol for every right-hand side (default tol = 2^-34, which
//          keeps the true error below 1e-10 with a factor-2 margin on the test workloads), at
//          most max_refine corrections after the first solve.  Frequencies that do not
//          converge are listed on the device and re-solved by a second, FP64 launch when asked
//          (steps = -1).
//
// Reference sequence: src/analysis/KrylovROMSubstructure.cpp:1403-1453 (host, MKL), the
// cuBLAS batched sweep of test/krylovMidsizeTest/gpu/concurrent/batchedLU/src/main.cu:223-267
// (no pivoting), the classical stopping rule of iterative refinement on the correction size (Wilkinson; Moler 1967).
#include <algorithm>
#include <climits>
#include <type_traits>

#include "sweep_common.cuh"

namespace srom {


// ====================================================================================
// smem class (FP64): the whole n x n matrix and the right-hand sides in shared memory, unblocked right-looking LU,
// one warp searches each pivot.  Nothing passes through global memory between assembly and solution, and all 256
// threads share the right-hand sides: a system of few columns, or of many right-hand sides to a column, is bound by
// those latencies and not by the pivot chain that sweep_lu64.cu shortens (fp64_smem_faster has both sides' times).
// ====================================================================================
__device__ __forceinline__ void panel_factor_smem(double2 *P, int ldp, int m, int ncols, int *ipiv, int *s_info,
                                  double2 *Bs, int ldbs, int nrhs, int *s_bc) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int jj = 0; jj < ncols; ++jj) {
        if (warp == 0) {
            double best = -1.0;
            int bi = INT_MAX;
            for (int i = jj + lane; i < m; i += 32) {
                double v = cabs1(P[i + (int64_t)jj * ldp]);
                if (v > best) {
                    best = v;
                    bi = i;
                }
            }
#pragma unroll
            for (int off = 16; off; off >>= 1) {
                double ob = __shfl_xor_sync(FULL_MASK, best, off);
                int oi = __shfl_xor_sync(FULL_MASK, bi, off);
                if (ob > best || (ob == best && oi < bi)) {
                    best = ob;
                    bi = oi;
                }
            }
            // IZAMAX starts from the first entry: a NaN there is returned as the pivot.
            double first = cabs1(P[jj + (int64_t)jj * ldp]);
            if (bi == INT_MAX || first != first) bi = jj;
            double2 piv = P[bi + (int64_t)jj * ldp];
            bool nz = (piv.x != 0.0 || piv.y != 0.0);
            if (nz) {
                if (bi != jj) {
                    if (lane == 0) {
                        P[bi + (int64_t)jj * ldp] = P[jj + (int64_t)jj * ldp];
                        P[jj + (int64_t)jj * ldp] = piv;
                    }
                    if (Bs)
                        for (int c = lane; c < nrhs; c += 32)
                            swap2(Bs[jj + (int64_t)c * ldbs], Bs[bi + (int64_t)c * ldbs]);
                }
                __syncwarp();
                double2 inv = crecip(piv);
                for (int i = jj + 1 + lane; i < m; i += 32)
                    P[i + (int64_t)jj * ldp] = cmul(P[i + (int64_t)jj * ldp], inv);
            } else if (lane == 0 && *s_info == 0) {
                *s_info = jj + 1;
            }
            if (lane == 0) {
                s_bc[0] = bi;
                s_bc[1] = nz ? 1 : 0;
                ipiv[jj] = bi + 1;
            }
        }
        __syncthreads();
        const int p = s_bc[0];
        const bool doswap = s_bc[1] && p != jj;
        if (doswap)
            for (int c = tid; c < jj; c += NT) swap2(P[jj + (int64_t)c * ldp], P[p + (int64_t)c * ldp]);
        for (int c = jj + 1 + warp; c < ncols; c += NW) {
            double2 *col = P + (int64_t)c * ldp;
            if (doswap) {
                if (lane == 0) swap2(col[jj], col[p]);
                __syncwarp();
            }
            const double2 u = col[jj];
            const double2 *lcol = P + (int64_t)jj * ldp;
            for (int i = jj + 1 + lane; i < m; i += 32) col[i] = csubmul(col[i], lcol[i], u);
        }
        __syncthreads();
    }
}


// One row of the blocked substitution: b[i, c] -= sum_j A[i, j] b[j, c] over the block's
// columns j (increasing for the forward sweep, decreasing for the backward one), all
// right-hand sides.  With a stage (global A), the row's block entries are copied into the
// thread's own shared-memory column (stage[t * NT + tid]) by cp.async in two alternating
// batches of CB, so the whole batch is in flight before it is used; without a stage
// (A in shared memory) the entries are read directly.
template <typename T, bool BACKWARD>
__device__ __forceinline__ void solve_row_block_chunk(const T *A, int64_t lda, T *B, int ldb, int nrhs, int i,
                                                      int jb, int je, T *stage, int CB) {
    using C = CT<T>;
    const int bs = je - jb;
    const int tid = threadIdx.x;
    auto col = [&](int t) { return BACKWARD ? je - 1 - t : jb + t; };
    T acc[RMAX_SOLVE];
#pragma unroll
    for (int cc = 0; cc < RMAX_SOLVE; ++cc) acc[cc] = cc < nrhs ? B[i + (int64_t)cc * ldb] : C::zero();
    if (stage) {
        const int nb = (bs + CB - 1) / CB;
        auto issue = [&](int b) {
            T *dst = stage + (b & 1) * CB * NT;
            for (int t = 0; t < CB && b * CB + t < bs; ++t) cp_async_elem(dst + t * NT + tid, A + i + col(b * CB + t) * lda);
            cp_async_commit();
        };
        issue(0);
        for (int b = 0; b < nb; ++b) {
            if (b + 1 < nb) {
                issue(b + 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            const T *src = stage + (b & 1) * CB * NT;
            for (int t = 0; t < CB && b * CB + t < bs; ++t) {
                const T a = src[t * NT + tid];
                const int j = col(b * CB + t);
#pragma unroll
                for (int cc = 0; cc < RMAX_SOLVE; ++cc)
                    if (cc < nrhs) acc[cc] = C::subm(acc[cc], a, B[j + (int64_t)cc * ldb]);
            }
        }
    } else {
        for (int t = 0; t < bs; ++t) {
            const int j = col(t);
            const T a = A[i + j * lda];
#pragma unroll
            for (int cc = 0; cc < RMAX_SOLVE; ++cc)
                if (cc < nrhs) acc[cc] = C::subm(acc[cc], a, B[j + (int64_t)cc * ldb]);
        }
    }
#pragma unroll
    for (int cc = 0; cc < RMAX_SOLVE; ++cc)
        if (cc < nrhs) B[i + (int64_t)cc * ldb] = acc[cc];
}

template <typename T, bool BACKWARD>
__device__ __forceinline__ void solve_row_block(const T *A, int64_t lda, T *B, int ldb, int nrhs, int i, int jb,
                                                int je, T *stage, int CB) {
    for (int c0 = 0; c0 < nrhs; c0 += RMAX_SOLVE)
        solve_row_block_chunk<T, BACKWARD>(A, lda, B + (int64_t)c0 * ldb, ldb, min(RMAX_SOLVE, nrhs - c0), i, jb, je,
                                           stage, CB);
}

// zgetrs 'N' on an in-place LU (A, lda) with B (n x nrhs, ldb) in shared memory; the row
// interchanges have already been applied to B.  32-row blocks: the block's diagonal triangle
// is staged in shared memory (tile, 32 x 33) when A lives in global memory, one warp per
// right-hand side solves it with the values in registers (warp shuffles), then every thread
// takes rows below (above) the block and applies the block to all right-hand sides of the
// row.  Every entry of B receives its updates in the oracle's order.
template <typename T>
__device__ void lu_solve(const T *A, int64_t lda, int n, T *B, int ldb, int nrhs, T *tile, T *stage = nullptr,
                         int stage_cb = 0) {
    using C = CT<T>;
    constexpr int LDT = 33;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int jb = 0; jb < n; jb += 32) {
        const int je = min(jb + 32, n), bs = je - jb;
        const T *D = A + jb + jb * lda;
        int ldd = (int)lda;
        if (tile) {
            for (int j = warp; j < bs; j += NW)
                if (lane < bs) tile[lane + j * LDT] = D[lane + j * lda];
            D = tile;
            ldd = LDT;
            __syncthreads();
        }
        for (int c = warp; c < nrhs; c += NW) {
            T *b = B + (int64_t)c * ldb + jb;
            T v = lane < bs ? b[lane] : C::zero();
            for (int j = 0; j < bs; ++j) {
                const T bj = C::shfl(v, j, 32);
                if (lane > j && lane < bs) v = C::subm(v, D[lane + j * ldd], bj);
            }
            if (lane < bs) b[lane] = v;
        }
        __syncthreads();
        for (int i = je + tid; i < n; i += NT) solve_row_block<T, false>(A, lda, B, ldb, nrhs, i, jb, je, stage, stage_cb);
        __syncthreads();
    }
    for (int jend = n; jend > 0; jend -= 32) {
        const int jb = max(jend - 32, 0), bs = jend - jb;
        const T *D = A + jb + jb * lda;
        int ldd = (int)lda;
        if (tile) {
            for (int j = warp; j < bs; j += NW)
                if (lane < bs) tile[lane + j * LDT] = D[lane + j * lda];
            D = tile;
            ldd = LDT;
            __syncthreads();
        }
        for (int c = warp; c < nrhs; c += NW) {
            T *b = B + (int64_t)c * ldb + jb;
            T v = lane < bs ? b[lane] : C::zero();
            for (int j = bs - 1; j >= 0; --j) {
                if (lane == j) v = C::div(v, D[j + j * ldd]);
                const T bj = C::shfl(v, j, 32);
                if (lane < j) v = C::subm(v, D[lane + j * ldd], bj);
            }
            if (lane < bs) b[lane] = v;
        }
        __syncthreads();
        for (int i = tid; i < jb; i += NT) solve_row_block<T, true>(A, lda, B, ldb, nrhs, i, jb, jend, stage, stage_cb);
        __syncthreads();
    }
}

// zgetrs 'N' for a factor in global memory, streamed through shared memory: the SW columns
// of each block, from the block's first row (forward) or row 0 (backward) to the last row
// needed, are copied by cp.async into one of two strip buffers while the previous block is
// being processed.  One warp per right-hand side solves the block's triangle from the strip,
// then every thread updates its rows.  B (n x nrhs, ldb) is in shared memory with the
// interchanges already applied; the per-entry update order is the oracle's.  With dinv (the
// mixed form's correction solves) the back substitution multiplies by the reciprocals of
// U's diagonal instead of dividing: the divisions were the critical path of the triangle.
template <typename T, int SW>
__device__ void lu_solve_strips(const T *A, int64_t lda, int n, T *B, int ldb, int nrhs, T *strips,
                                const T *dinv = nullptr) {
    using C = CT<T>;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nblk = (n + SW - 1) / SW;
    // ---- forward: unit lower triangle ----
    auto issue_f = [&](int blk) {
        const int jb = blk * SW, bs = min(SW, n - jb), rows = n - jb;
        T *dst = strips + (blk & 1) * (SW * n);
        for (int e = tid; e < rows * bs; e += NT) {
            const int r = e % rows, c = e / rows;
            cp_async_elem(dst + c * n + r, A + (jb + r) + (int64_t)(jb + c) * lda);
        }
        cp_async_commit();
    };
    issue_f(0);
    for (int blk = 0; blk < nblk; ++blk) {
        const int jb = blk * SW, bs = min(SW, n - jb), rows = n - jb;
        if (blk + 1 < nblk) {
            issue_f(blk + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const T *S = strips + (blk & 1) * (SW * n);  // S[c * n + r] = A[jb + r, jb + c]
        for (int c = warp; c < nrhs; c += NW) {
            T *b = B + (int64_t)c * ldb + jb;
            T v = lane < bs ? b[lane] : C::zero();
            for (int j = 0; j < bs; ++j) {
                const T bj = C::shfl(v, j, 32);
                if (lane > j && lane < bs) v = C::subm(v, S[j * n + lane], bj);
            }
            if (lane < bs) b[lane] = v;
        }
        __syncthreads();
        for (int r = bs + tid; r < rows; r += NT) {
            for (int c0 = 0; c0 < nrhs; c0 += 4) {
                const int nc = min(4, nrhs - c0);
                T acc[4];
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) acc[cc] = cc < nc ? B[jb + r + (int64_t)(c0 + cc) * ldb] : C::zero();
#pragma unroll
                for (int j = 0; j < SW; ++j) {
                    if (j < bs) {
                        const T a = S[j * n + r];
#pragma unroll
                        for (int cc = 0; cc < 4; ++cc)
                            if (cc < nc) acc[cc] = C::subm(acc[cc], a, B[jb + j + (int64_t)(c0 + cc) * ldb]);
                    }
                }
#pragma unroll
                for (int cc = 0; cc < 4; ++cc)
                    if (cc < nc) B[jb + r + (int64_t)(c0 + cc) * ldb] = acc[cc];
            }
        }
        __syncthreads();
    }
    // ---- backward: upper triangle, blocks from the last ----
    auto issue_b = [&](int q) {  // q-th block from the end
        const int jend = n - q * SW, jb = max(jend - SW, 0), bs = jend - jb, rows = jend;
        T *dst = strips + (q & 1) * (SW * n);
        for (int e = tid; e < rows * bs; e += NT) {
            const int r = e % rows, c = e / rows;
            cp_async_elem(dst + c * n + r, A + r + (int64_t)(jb + c) * lda);
        }
        cp_async_commit();
    };
    issue_b(0);
    for (int q = 0; q < nblk; ++q) {
        const int jend = n - q * SW, jb = max(jend - SW, 0), bs = jend - jb;
        if (q + 1 < nblk) {
            issue_b(q + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const T *S = strips + (q & 1) * (SW * n);  // S[c * n + r] = A[r, jb + c]
        for (int c = warp; c < nrhs; c += NW) {
            T *b = B + (int64_t)c * ldb + jb;
            T v = lane < bs ? b[lane] : C::zero();
            for (int j = bs - 1; j >= 0; --j) {
                if (lane == j) v = dinv ? C::mul(v, dinv[jb + j]) : C::div(v, S[j * n + jb + j]);
                const T bj = C::shfl(v, j, 32);
                if (lane < j) v = C::subm(v, S[j * n + jb + lane], bj);
            }
            if (lane < bs) b[lane] = v;
        }
        __syncthreads();
        for (int r = tid; r < jb; r += NT) {
            for (int c0 = 0; c0 < nrhs; c0 += 4) {
                const int nc = min(4, nrhs - c0);
                T acc[4];
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) acc[cc] = cc < nc ? B[r + (int64_t)(c0 + cc) * ldb] : C::zero();
#pragma unroll
                for (int jj = 0; jj < SW; ++jj) {
                    const int j = bs - 1 - jj;
                    if (j >= 0) {
                        const T a = S[j * n + r];
#pragma unroll
                        for (int cc = 0; cc < 4; ++cc)
                            if (cc < nc) acc[cc] = C::subm(acc[cc], a, B[jb + j + (int64_t)(c0 + cc) * ldb]);
                    }
                }
#pragma unroll
                for (int cc = 0; cc < 4; ++cc)
                    if (cc < nc) B[r + (int64_t)(c0 + cc) * ldb] = acc[cc];
            }
        }
        __syncthreads();
    }
}


__global__ void __launch_bounds__(NT) sweep_fp64_smem_kernel(const RomDev *__restrict__ roms,
                                                              const Item *__restrict__ items,
                                                              int n_items, int *counter) {
    extern __shared__ double2 smem[];
    __shared__ int s_item, s_info, s_bc[2];
    for (;;) {
        const int it = next_item(counter, &s_item);
        if (it >= n_items) break;
        const Item w = items[it];
        const RomDev R = roms[w.rom];
        const int n = R.n;
        const int lda = n | 1;
        double2 *A = smem;
        double2 *B = A + (int64_t)n * lda;
        int *ipiv = reinterpret_cast<int *>(B + (int64_t)n * R.r);
        assemble_into<double2>(A, lda, R, R.omega[w.f], w.f);
        load_rhs(B, n, R);
        if (threadIdx.x == 0) s_info = 0;
        __syncthreads();
        panel_factor_smem(A, lda, n, n, ipiv, &s_info, B, n, R.r, s_bc);
        lu_solve<double2>(A, lda, n, B, n, R.r, nullptr);
        store_solution(B, n, R, w.f);
        if (R.LU) {
            double2 *LU = R.LU + (int64_t)w.f * n * n;
            for (int j = threadIdx.x >> 5; j < n; j += NW)
                for (int i = threadIdx.x & 31; i < n; i += 32) LU[i + (int64_t)j * n] = A[i + j * lda];
            for (int j = threadIdx.x; j < n; j += NT) R.ipiv[(int64_t)w.f * n + j] = ipiv[j];
        }
        if (threadIdx.x == 0) {
            if (R.info) R.info[w.f] = s_info;
            if (R.steps) R.steps[w.f] = 0;
            if (R.berr) R.berr[w.f] = 0.0;
        }
        __syncthreads();
    }
}

// ====================================================================================
// global class
// ====================================================================================

// Per-warp processing of the columns outside the panel after panel j0 has been factored.
//   * columns [0, j0) and the nrhs right-hand-side columns of B: apply the interchanges;
//   * columns [j0+nbc, n) in groups of CW: interchanges, U rows by forward substitution with
//     the unit-lower panel triangle, then A22 -= L21 U12 for logical rows [nbc, m).
template <typename T, int NB>
__device__ void trailing_update(T *A, int64_t lda, int n, int j0, int nbc, const T *P, int ldp,
                                const int *s_perm, const int *s_mdst, const int *s_msrc, int nmoved,
                                T *s_u, T *B, int ldbs, int nrhs, int *s_grp) {
    using C = CT<T>;
    constexpr int CW = CWG;                       // trailing columns per warp group
    constexpr int RQ = 2;                         // Schur rows per lane per pass
    constexpr int MV = (2 * NB + 31) / 32;
    constexpr int TR = 32 / NB;  // row segments per warp in the triangle solve
    constexpr int TC = CW / TR;  // columns per lane in the triangle solve
    static_assert(TR * TC == CW, "triangle solve covers the column group");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = n - j0;

    constexpr int CB = 8;  // swap-only columns per warp pass (loads in flight)
    for (int cb = warp * CB; cb < j0 + nrhs; cb += NW * CB) {
        T mv[MV][CB];
#pragma unroll
        for (int t = 0; t < CB; ++t) {
            const int c = cb + t;
            if (c < j0 + nrhs) {
                const T *col = c < j0 ? A + (int64_t)c * lda + j0 : B + (int64_t)(c - j0) * ldbs + j0;
#pragma unroll
                for (int q = 0; q < MV; ++q) {
                    const int e = lane + 32 * q;
                    if (e < nmoved) mv[q][t] = col[s_msrc[e]];
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < CB; ++t) {
            const int c = cb + t;
            if (c < j0 + nrhs) {
                T *col = c < j0 ? A + (int64_t)c * lda + j0 : B + (int64_t)(c - j0) * ldbs + j0;
#pragma unroll
                for (int q = 0; q < MV; ++q) {
                    const int e = lane + 32 * q;
                    if (e < nmoved) col[s_mdst[e]] = mv[q][t];
                }
            }
        }
        __syncwarp();
    }

    T *u = s_u + warp * NB * CW;
    const int trow = lane % NB, tgrp = lane / NB;
    // column groups are handed out dynamically so that warps finish a panel together
    for (;;) {
        int gi = 0;
        if (lane == 0) gi = atomicAdd(s_grp, 1);
        gi = __shfl_sync(FULL_MASK, gi, 0);
        const int c0 = j0 + nbc + gi * CW;
        if (c0 >= n) break;
        T mv[MV][CW];
        T uv[TC];
#pragma unroll
        for (int q = 0; q < MV; ++q) {
            const int e = lane + 32 * q;
            if (e < nmoved) {
                const int s = s_msrc[e];
#pragma unroll
                for (int cc = 0; cc < CW; ++cc)
                    if (c0 + cc < n) mv[q][cc] = A[(j0 + s) + (int64_t)(c0 + cc) * lda];
            }
        }
        const int prow = trow < nbc ? s_perm[trow] : 0;
#pragma unroll
        for (int t = 0; t < TC; ++t) {
            const int cc = tgrp * TC + t;
            uv[t] = (trow < nbc && c0 + cc < n) ? A[(j0 + prow) + (int64_t)(c0 + cc) * lda] : C::zero();
        }
        __syncwarp();
        for (int k = 0; k < nbc; ++k) {
            const bool act = trow > k && trow < nbc;
            const T lk = act ? P[prow + (int64_t)k * ldp] : C::zero();
#pragma unroll
            for (int t = 0; t < TC; ++t) {
                const T ukt = C::shfl(uv[t], k, NB);
                if (act) uv[t] = C::subm(uv[t], lk, ukt);
            }
        }
        if (trow < nbc) {
#pragma unroll
            for (int t = 0; t < TC; ++t) {
                const int cc = tgrp * TC + t;
                u[trow * CW + cc] = uv[t];
                if (c0 + cc < n) A[(j0 + trow) + (int64_t)(c0 + cc) * lda] = uv[t];
            }
        }
#pragma unroll
        for (int q = 0; q < MV; ++q) {
            const int e = lane + 32 * q;
            if (e < nmoved) {
                const int d = s_mdst[e];
                if (d >= nbc) {
#pragma unroll
                    for (int cc = 0; cc < CW; ++cc)
                        if (c0 + cc < n) A[(j0 + d) + (int64_t)(c0 + cc) * lda] = mv[q][cc];
                }
            }
        }
        __syncwarp();
        T nxt[RQ][CW];
        int npr[RQ];
        auto load_chunk = [&](int rb, T (&dst)[RQ][CW], int (&pr)[RQ]) {
#pragma unroll
            for (int q = 0; q < RQ; ++q) {
                const int l = rb + lane + 32 * q;
                pr[q] = l < m ? s_perm[l] : 0;
#pragma unroll
                for (int cc = 0; cc < CW; ++cc)
                    dst[q][cc] = (l < m && c0 + cc < n) ? A[(j0 + l) + (int64_t)(c0 + cc) * lda] : C::zero();
            }
        };
        if (nbc < m) load_chunk(nbc, nxt, npr);
        for (int rb = nbc; rb < m; rb += 32 * RQ) {
            T acc[RQ][CW];
            int pr[RQ];
#pragma unroll
            for (int q = 0; q < RQ; ++q) {
                pr[q] = npr[q];
#pragma unroll
                for (int cc = 0; cc < CW; ++cc) acc[q][cc] = nxt[q][cc];
            }
            if (rb + 32 * RQ < m) load_chunk(rb + 32 * RQ, nxt, npr);
            for (int k = 0; k < nbc; ++k) {
                T lv[RQ], uw[CW];
#pragma unroll
                for (int q = 0; q < RQ; ++q) lv[q] = P[pr[q] + (int64_t)k * ldp];
#pragma unroll
                for (int cc = 0; cc < CW; ++cc) uw[cc] = u[k * CW + cc];
                // c - a*b as two FMA layers over the whole tile: the same two roundings per
                // component as C::subm, but every first FMA is issued before any second one.
#pragma unroll
                for (int q = 0; q < RQ; ++q)
#pragma unroll
                    for (int cc = 0; cc < CW; ++cc) C::subm_first(acc[q][cc], lv[q], uw[cc]);
#pragma unroll
                for (int q = 0; q < RQ; ++q)
#pragma unroll
                    for (int cc = 0; cc < CW; ++cc) C::subm_second(acc[q][cc], lv[q], uw[cc]);
            }
#pragma unroll
            for (int q = 0; q < RQ; ++q) {
                const int l = rb + lane + 32 * q;
#pragma unroll
                for (int cc = 0; cc < CW; ++cc)
                    if (l < m && c0 + cc < n) A[(j0 + l) + (int64_t)(c0 + cc) * lda] = acc[q][cc];
            }
        }
        __syncwarp();
    }
}

// Shared-memory carve-up of the global-class kernels (bytes from the dynamic base).
// The u and panel regions come last: during the mixed form's refinement neither is in use, and
// together with whatever dynamic shared memory lies beyond `total` they form the staging ring
// of the correction solves (ring = [u, end of the dynamic allocation)).
// big: the large-order FP64 instances (orders whose panel does not fit shared memory): the
// panel lives in global scratch, the panel region holds the solve's 32 x 33 diagonal tile
// instead, and the mixed form's regions (work32, pos, dinv) are empty.
struct GlobalSmem {
    size_t work64, work32, perm, ptot, pos, ipiv, moved, dinv, u, panel, total;
    static __host__ __device__ size_t up(size_t b) { return (b + 255) / 256 * 256; }
    __host__ __device__ GlobalSmem(int ldp, int n_max, int r_max, bool big = false) {
        work64 = 0;
        work32 = work64 + up((size_t)n_max * r_max * 16);
        perm = work32 + (big ? 0 : up((size_t)n_max * r_max * 8));
        ptot = perm + up((size_t)ldp * 4);
        pos = ptot + up((size_t)ldp * 4);
        ipiv = pos + (big ? 0 : up((size_t)ldp * 4));
        moved = ipiv + up((size_t)ldp * 4);
        dinv = moved + up((size_t)2 * 2 * NB32 * 4);
        u = dinv + (big ? 0 : up((size_t)ldp * 16));      // reciprocals of diag(U), mixed form
        static_assert(sizeof(PanelXchg32) <= (size_t)NW * 2048, "the panel's exchange fits the u region");
        panel = u + up((size_t)NW * 2048);                // per warp NB x CWG complex
        total = panel + (big ? up((size_t)32 * 33 * 16)   // the solve's diagonal tile
                             : up((size_t)ldp * 256));    // ldp x 16 double2 == ldp x 32 float2
    }
};

// panel_factor_32 as a function of its own, its arguments shared-memory offsets so that its accesses are known to
// be shared ones: inlined into this kernel the same code took 1.3 times as long a column (256 rows: 1870 cycles
// against 1400; in the tensor-core kernel the inlined form is the faster one).
extern __shared__ __align__(256) unsigned char panel_sm[];
template <int RPT>
__device__ __noinline__ void panel_call(unsigned p_off, int ldp, int m, int ncols, unsigned perm_off, unsigned lg_off,
                                        int *s_pivlg, unsigned moved_off, PanelLists &PL, int info_off, unsigned x_off) {
    int *moved = reinterpret_cast<int *>(panel_sm + moved_off);
    panel_factor_32<RPT>(reinterpret_cast<float2 *>(panel_sm + p_off), ldp, m, ncols,
                         reinterpret_cast<int *>(panel_sm + perm_off), reinterpret_cast<int *>(panel_sm + lg_off), s_pivlg,
                         moved, moved + 2 * NB32, PL, info_off, *reinterpret_cast<PanelXchg32 *>(panel_sm + x_off));
}

// Blocked LU of the system already assembled in A (n x n, lda).  B (smem, ld n, nrhs
// columns, may be null) receives the interchanges; s_ptot (smem) the composite row
// permutation (final row l holds original row s_ptot[l]); s_ipiv the LAPACK pivots.
template <typename T, int NB, int RPT>
__device__ void factor_global(T *A, int64_t lda, int n, int ldp, unsigned char *sm, const GlobalSmem &L,
                              T *B, int nrhs, PanelLists &PL, PivotXchg<typename CT<T>::R> &X,
                              int *s_pivlg, T *P_global = nullptr) {
    // the panel: shared memory, or (large orders) the CTA's global scratch, L2-resident
    T *P = P_global ? P_global : reinterpret_cast<T *>(sm + L.panel);
    T *s_u = reinterpret_cast<T *>(sm + L.u);
    int *s_perm = reinterpret_cast<int *>(sm + L.perm);
    int *s_ptot = reinterpret_cast<int *>(sm + L.ptot);
    int *s_ipiv = reinterpret_cast<int *>(sm + L.ipiv);
    int *s_mdst = reinterpret_cast<int *>(sm + L.moved);
    int *s_msrc = s_mdst + 2 * NB32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < n; i += NT) s_ptot[i] = i;
    if (tid == 0) PL.info = 0;
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int nbc = min(NB, n - j0);
        const int m = n - j0;
        for (int c = warp; c < nbc; c += NW)
            for (int i = lane; i < m; i += 32) P[i + (int64_t)c * ldp] = A[(j0 + i) + (j0 + c) * lda];
        if (tid == 0) {
            PL.nmoved = 0;
            PL.grp = 0;
        }
        __syncthreads();
        if constexpr (std::is_same<T, float2>::value)  // the u region is free until the trailing update
            panel_call<RPT>((unsigned)L.panel, ldp, m, nbc, (unsigned)L.perm, (unsigned)L.pos, s_pivlg, (unsigned)L.moved,
                            PL, j0, (unsigned)L.u);
        else
            panel_factor_par<T, RPT>(P, ldp, m, nbc, s_perm, s_pivlg, s_mdst, s_msrc, PL, j0, X);
        const int nmoved = PL.nmoved;
        for (int c = warp; c < nbc; c += NW)
            for (int i = lane; i < m; i += 32) A[(j0 + i) + (j0 + c) * lda] = P[s_perm[i] + (int64_t)c * ldp];
        if (tid < nbc) s_ipiv[j0 + tid] = j0 + s_pivlg[tid] + 1;
        if (warp == NW - 1) {
            int v[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int e = lane + 32 * q;
                if (e < nmoved) v[q] = s_ptot[j0 + s_msrc[e]];
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int e = lane + 32 * q;
                if (e < nmoved) s_ptot[j0 + s_mdst[e]] = v[q];
            }
            __syncwarp();
        }
        trailing_update<T, NB>(A, lda, n, j0, nbc, P, ldp, s_perm, s_mdst, s_msrc, nmoved, s_u, B, n, nrhs, &PL.grp);
        __syncthreads();
    }
}


// Global-class kernel.  MIXED: complex-FP32 factors + FP64 refinement; systems that do not
// converge are appended to a.fb_items (when given) for the FP64 kernel launched after it.
// FP64: the bit-exact path; a.n_items_dev (when given) holds the item count (fallback list).
// BIG (FP64 only): the panel in global scratch (a.panel_off into the CTA's slot) and the
// tile-staged blocked solve (lu_solve), for orders up to NT * RPT whose panel does not fit
// shared memory.
template <bool MIXED, int RPT, bool BIG = false>
__global__ void __launch_bounds__(NT) sweep_global_kernel(GlobalArgs a) {
    static_assert(!(MIXED && BIG), "large orders are FP64 only");
    extern __shared__ __align__(256) unsigned char sm[];
    __shared__ int s_item;
    __shared__ int s_pivlg[NB32];
    __shared__ PanelLists PL;
    __shared__ PivotXchg<typename CT<typename std::conditional<MIXED, float2, double2>::type>::R> Xx;
    __shared__ double s_dx[RMAX_MIXED];
    using T = typename std::conditional<MIXED, float2, double2>::type;
    const GlobalSmem L(a.ldp, a.n_max, a.r_max, BIG);
    const int tid = threadIdx.x;
    const int n_items = a.n_items_dev ? *a.n_items_dev : a.n_items;
    int *s_ipiv = reinterpret_cast<int *>(sm + L.ipiv);

    for (;;) {
        const int it = next_item(a.counter, &s_item);
        if (it >= n_items) break;
        const Item wi = a.items[it];
        const RomDev R = a.roms[wi.rom];
        const int n = R.n;
        const double w = R.omega[wi.f];
        int steps = 0, info = 0;
        double berr = 0.0;
        bool write_status = true;
        if constexpr (MIXED) {
            float2 *A32 = reinterpret_cast<float2 *>(a.scratch + (int64_t)blockIdx.x * a.slot_bytes);
            double2 *X = reinterpret_cast<double2 *>(sm + L.work64);
            float2 *B32 = reinterpret_cast<float2 *>(sm + L.work32);
            int *s_pos = reinterpret_cast<int *>(sm + L.pos);
            int *s_ptot = reinterpret_cast<int *>(sm + L.ptot);
            assemble_into<float2>(A32, n, R, w, wi.f);
            __syncthreads();
            factor_global<float2, NB32, RPT>(A32, n, n, a.ldp, sm, L, nullptr, 0, PL, Xx, s_pivlg);
            info = PL.info;
            MixedWork W{X, B32, s_pos, s_ptot, reinterpret_cast<float2 *>(sm + L.dinv), sm + L.u,
                        a.smem_dyn - (int)L.u, s_dx, n};  // ring: u, panel and the rest of the allocation
            const RingSolve<RPT> solve{A32, n, n, W.ring, W.ring_bytes, W.s_dinv};
            mixed_refine<RPT>(a, R, wi, w, A32, W, solve, info, steps, berr, write_status);
        } else {
            double2 *A64 = R.LU ? R.LU + (int64_t)wi.f * n * n
                                : reinterpret_cast<double2 *>(a.scratch + (int64_t)blockIdx.x * a.slot_bytes);
            double2 *B = reinterpret_cast<double2 *>(sm + L.work64);
            assemble_into<double2>(A64, n, R, w, wi.f);
            load_rhs(B, n, R);
            __syncthreads();
            if constexpr (BIG) {
                double2 *Pg = reinterpret_cast<double2 *>(a.scratch + (int64_t)blockIdx.x * a.slot_bytes + a.panel_off);
                factor_global<double2, NB64, RPT>(A64, n, n, a.ldp, sm, L, B, R.r, PL, Xx, s_pivlg, Pg);
                info = PL.info;
                lu_solve<double2>(A64, n, n, B, n, R.r, reinterpret_cast<double2 *>(sm + L.panel));
            } else {
                factor_global<double2, NB64, RPT>(A64, n, n, a.ldp, sm, L, B, R.r, PL, Xx, s_pivlg);
                info = PL.info;
                lu_solve_strips<double2, 8>(A64, n, n, B, n, R.r, reinterpret_cast<double2 *>(sm + L.panel));
            }
            store_solution(B, n, R, wi.f);
            steps = a.steps_value;
            if (R.ipiv)
                for (int j = tid; j < n; j += NT) R.ipiv[(int64_t)wi.f * n + j] = s_ipiv[j];
        }
        if (tid == 0 && write_status) {
            if (R.info) R.info[wi.f] = info;
            if (R.steps) R.steps[wi.f] = steps;
            if (R.berr) R.berr[wi.f] = berr;
        }
        __syncthreads();
    }
}

// ====================================================================================
// host-side launch helpers
// ====================================================================================
// What the kernels of this file are allowed to ask for, one value for all sizes: another thread's smaller launch of the
// same kernel must not lower it between a launcher's call and its launch.
constexpr size_t SMEM_DYN = SMEM_OPTIN - GLOBAL_STATIC_SMEM;

size_t fp64_smem_bytes(int n, int r) {
    const size_t lda = (size_t)(n | 1);
    return sizeof(double2) * (lda * n + (size_t)n * r) + sizeof(int) * (size_t)n;
}

size_t global_smem_bytes(int n_max, int r_max, bool big) { return GlobalSmem(n_max | 1, n_max, r_max, big).total; }

bool global_panel_fits(int n_max, int r_max, int smem_optin) {
    return global_rpt(n_max) <= GLOBAL_MAX_RPT &&
           global_smem_bytes(n_max, r_max, false) + GLOBAL_STATIC_SMEM <= (size_t)smem_optin;
}

int64_t big_panel_offset(int n_max) { return ((int64_t)n_max * n_max * 16 + 255) / 256 * 256; }

int64_t big_slot_bytes(int n_max) { return big_panel_offset(n_max) + (int64_t)(n_max | 1) * NB64 * 16; }

size_t fp64_global_smem_bytes(int n_max, int r_max) { return global_smem_bytes(n_max, r_max, false); }

int global_rpt(int n_max) { return (n_max + NT - 1) / NT; }

// Where the shared-memory kernel is faster than the row kernel, by how the call's systems fill the GPU (a call alone,
// row kernel / shared-memory kernel, us or their ratio): one wave of the latter, two CTAs a multiprocessor where its
// shared memory holds two: order 1 and 1 right-hand side 30.7 / 24.1, 8 and 16 43 / 35, 24 and 200 505 / 283, 1 and 5000
// 2135 / 350, 222 systems of order 5 33 / 30.5; but 16 and 1 36 / 41, 48 and 16 0.78.  Two a multiprocessor (300 systems):
// order 4 and 32 right-hand sides 1.05, 8 and 64 0.94; four (600): order 2 and 64 1.04, 3 and 64 0.94; more (1200, 4000):
// order 1 and 16 1.09 / 1.00, 2 and 64 1.08 / 0.95, 4 and 256 1.10 / 0.97.  Within a first panel of 16 columns the row
// kernel has no second pass over the right-hand sides, hence the two lines up to order 32.
bool fp64_smem_faster(int n, int r, long long systems, int sms) {
    const long long q = (long long)(n - 1) * (n - 1);
    const int wave = sms * (2 * (fp64_smem_bytes(n, r) + 1088) <= (size_t)228 * 1024 ? 2 : 1);
    if (systems <= wave) return n <= 8 || (n <= 16 && 3LL * r >= n) || (n <= 32 && n > 16 && 5LL * r >= n);
    if (n > 10) return false;
    if (systems <= 2LL * sms + sms / 4) return r >= 2 * q;
    if (systems <= 4LL * sms + sms / 4) return r >= 32 * q;
    return r >= 16 + 26 * q;
}

cudaError_t launch_fp64_smem(const RomDev *roms, const Item *items, int n_items, int *counter,
                             size_t smem, int grid, cudaStream_t st) {
    auto k = sweep_fp64_smem_kernel;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_DYN);
    if (e != cudaSuccess) return e;
    k<<<grid, NT, smem, st>>>(roms, items, n_items, counter);
    return cudaGetLastError();
}

int fp64_smem_blocks_per_sm(size_t smem) {
    int b = 0;
    auto k = sweep_fp64_smem_kernel;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_DYN) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, NT, smem) != cudaSuccess) return 0;
    return b;
}

// The mixed kernel takes all the shared memory a CTA may have (one CTA per SM either way, by
// registers): what lies beyond its fixed regions deepens the correction solves' staging ring.
template <bool MIXED, int RPT, bool BIG = false>
static cudaError_t launch_global_t(const GlobalArgs &a0, int grid, cudaStream_t st) {
    auto k = sweep_global_kernel<MIXED, RPT, BIG>;
    GlobalArgs a = a0;
    size_t smem = global_smem_bytes(a.n_max, a.r_max, BIG);
    if (MIXED) {
        int dev = 0, optin = 0;
        cudaFuncAttributes fa{};
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k);
        if (e != cudaSuccess) return e;
        const size_t cap = (size_t)optin - fa.sharedSizeBytes;
        if (cap > smem) smem = cap / 256 * 256;
        // the correction solves' ring must hold two strips of 16 columns of the largest system
        const size_t ring = smem - GlobalSmem(a.ldp, a.n_max, a.r_max).u;
        if (ring < 2 * (size_t)16 * a.n_max * sizeof(float2)) return cudaErrorInvalidValue;
    }
    a.smem_dyn = (int)smem;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max(smem, SMEM_DYN));
    if (e != cudaSuccess) return e;
    k<<<grid, NT, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_global(bool mixed, const GlobalArgs &a0, int grid, cudaStream_t st) {
    GlobalArgs a = a0;
    a.ldp = a.n_max | 1;
    const int rpt = global_rpt(a.n_max);
    if (mixed && a.r_max > RMAX_MIXED) return cudaErrorInvalidValue;
    if (mixed) {
        if (rpt <= 1) return launch_global_t<true, 1>(a, grid, st);
        if (rpt == 2) return launch_global_t<true, 2>(a, grid, st);
        if (rpt == 3) return launch_global_t<true, 3>(a, grid, st);
    } else {
        if (rpt <= 3) return launch_global_t<false, 3>(a, grid, st);  // n > LU64_MAX_N
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_global_big(const GlobalArgs &a0, int grid, cudaStream_t st) {
    GlobalArgs a = a0;
    a.ldp = a.n_max | 1;
    if (a.slot_bytes < big_slot_bytes(a.n_max)) return cudaErrorInvalidValue;
    a.panel_off = big_panel_offset(a.n_max);
    const int rpt = global_rpt(a.n_max);
    return rpt <= GLOBAL_MAX_RPT ? launch_global_t<false, GLOBAL_MAX_RPT, true>(a, grid, st) : cudaErrorInvalidValue;
}

}  // namespace srom
