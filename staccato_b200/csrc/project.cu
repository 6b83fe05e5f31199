// ROM projection kernels: R_m = V^T A_m V for sparse FE matrices A_m sharing one CSR pattern,
// and the FP64 Gram-Schmidt orthonormalisation of the basis V.
//
// Reference: generateROM (src/analysis/KrylovROMSubstructure.cpp:709-765) computes
// Y = A V with mkl_sparse_z_mm (src/tools/MathLibrary.cpp:491-532) and R = V^H Y with
// cblas_zgemm ConjTrans (src/tools/MathLibrary.cpp:177-234), one matrix after another; the
// basis comes from block Gram-Schmidt with re-orthogonalisation (KrylovROMSubstructure.cpp:433-454).
//
// B200 layout: V is transposed once into row-major Vt (N x k) so that the k entries of a
// basis row are contiguous; the SpMM gives each warp one node (three rows), and every gathered
// Vt row feeds its rows and all matrices of the pattern (K and M share it);
// Y_m is written row-major.  R_m = Vt^T Y_m runs on the FP64 tensor cores
// (mma.sync m8n8k4 f64): each CTA reduces a contiguous row range into a private k x k
// partial, and a second kernel sums the partials in a fixed order (16 segments; deterministic).
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "project_kernels.h"

namespace srom {

constexpr int PRJ_MAX_MATS = 3;
constexpr int PRJ_WIN = 128;  // basis columns per SpMM pass and per side of a V^T Y window

// ---- V (column-major, ldv) -> Vt (row-major N x k) --------------------------------------
__global__ void transpose_kernel(const double *__restrict__ V, int64_t N, int k, int64_t ldv,
                                 double *__restrict__ Vt) {
    __shared__ double t[32][33];
    const int64_t r0 = (int64_t)blockIdx.x * 32;
    const int c0 = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int64_t r = r0 + threadIdx.x;
        const int c = c0 + y;
        if (r < N && c < k) t[y][threadIdx.x] = V[r + (int64_t)c * ldv];
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int64_t r = r0 + y;
        const int c = c0 + threadIdx.x;
        if (r < N && c < k) Vt[r * k + c] = t[threadIdx.x][y];
    }
}

// ---- Y_m = A_m V  (full CSR pattern, shared by the n_mats value arrays) -----------------
// A warp takes three consecutive rows.  FE matrices numbered node by node give the three
// DOF rows of a node the same column pattern; when the warp finds that (equal lengths and
// equal column lists, checked with a warp vote), every gathered Vt row feeds all three rows
// and all matrices, cutting the Vt gathers -- the dominant L2 traffic -- by three.  Otherwise
// the rows are processed one after the other.  The column indices and values of a row are
// staged 32 entries at a time in the warp's shared-memory slot (coalesced loads), so that
// the Vt gathers of SPMM_DEPTH consecutive entries are independent loads in flight together.
// Every Y entry is the sequential FMA chain over the row's entries in storage order.
//
// CTAs of four warps, a warp a node, more of them than are resident: the hardware hands out the next CTA as one
// ends.  With one resident wave that strides over the nodes, the long rows (a vertex node couples to 195 columns,
// the average to 80) fell to the same warps whenever the wave's length met a multiple of a mesh layer's.  Two
// matrices, 96 columns: 30,927 rows 160 -> 96 us, 41,175 rows 160 -> 121 us, 107,163 rows 316 -> 277 us; CTAs of
// eight warps 113 / 141 / 326 us, of two 99 / 125 / 282 us.
constexpr int SPMM_THREADS = 128;
constexpr int SPMM_MMA_CTAS = 4;  // resident CTAs an SM of spmm_mma_kernel (128 registers a thread)
constexpr int SPMM_WARPS = SPMM_THREADS / 32;
constexpr int SPMM_DEPTH = 4;

struct SpmmStage {
    int col[32];
    double val[3 * PRJ_MAX_MATS][32];
};

// Column window: the k (<= 32 CPL) basis columns starting at Vt (row stride ldv) into Y (row
// stride ldy); a basis wider than 128 columns is projected window by window.
template <int CPL, int NMAT, int NR>
__device__ __forceinline__ void spmm_rows(int64_t row, const int64_t *__restrict__ rowptr,
                                          const int *__restrict__ colind, int base, const ProjVals &vals,
                                          const double *__restrict__ Vt, int k, int ldv, double *__restrict__ Y,
                                          int ldy, int64_t y_stride, int lane, SpmmStage &st) {
    const int64_t e0 = rowptr[row] - base, e1 = rowptr[row + 1] - base;
    int64_t off[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) off[r] = (rowptr[row + r] - base) - e0;
    double acc[NR][NMAT][CPL];
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int m = 0; m < NMAT; ++m)
#pragma unroll
            for (int q = 0; q < CPL; ++q) acc[r][m][q] = 0.0;
    for (int64_t c0 = e0; c0 < e1; c0 += 32) {
        const int cnt = (int)min((int64_t)32, e1 - c0);
        __syncwarp();
        if (lane < cnt) {
            st.col[lane] = colind[c0 + lane] - base;
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int m = 0; m < NMAT; ++m) st.val[r * NMAT + m][lane] = vals.v[m][c0 + lane + off[r]];
        }
        __syncwarp();
        int j = 0;
        for (; j + SPMM_DEPTH <= cnt; j += SPMM_DEPTH) {
            double v[SPMM_DEPTH][CPL];
#pragma unroll
            for (int u = 0; u < SPMM_DEPTH; ++u) {
                const double *vr = Vt + (int64_t)st.col[j + u] * ldv;
#pragma unroll
                for (int q = 0; q < CPL; ++q) {
                    const int c = lane + 32 * q;
                    v[u][q] = c < k ? vr[c] : 0.0;
                }
            }
#pragma unroll
            for (int u = 0; u < SPMM_DEPTH; ++u)
#pragma unroll
                for (int r = 0; r < NR; ++r)
#pragma unroll
                    for (int m = 0; m < NMAT; ++m) {
                        const double a = st.val[r * NMAT + m][j + u];
#pragma unroll
                        for (int q = 0; q < CPL; ++q) acc[r][m][q] = fma(a, v[u][q], acc[r][m][q]);
                    }
        }
        for (; j < cnt; ++j) {
            const double *vr = Vt + (int64_t)st.col[j] * ldv;
#pragma unroll
            for (int q = 0; q < CPL; ++q) {
                const int c = lane + 32 * q;
                const double v = c < k ? vr[c] : 0.0;
#pragma unroll
                for (int r = 0; r < NR; ++r)
#pragma unroll
                    for (int m = 0; m < NMAT; ++m) acc[r][m][q] = fma(st.val[r * NMAT + m][j], v, acc[r][m][q]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int m = 0; m < NMAT; ++m)
#pragma unroll
            for (int q = 0; q < CPL; ++q) {
                const int c = lane + 32 * q;
                if (c < k) Y[m * y_stride + (row + r) * ldy + c] = acc[r][m][q];
            }
}

// Whether the rows r0 .. r0 + 2 have the same column list (a warp vote; the trip count is warp-uniform).
__device__ __forceinline__ bool same_columns(int64_t r0, const int64_t *__restrict__ rowptr,
                                             const int *__restrict__ colind, int base, int lane) {
    const int64_t a0 = rowptr[r0], a1 = rowptr[r0 + 1], a2 = rowptr[r0 + 2], a3 = rowptr[r0 + 3];
    const int64_t len = a1 - a0;
    bool same = (a2 - a1) == len && (a3 - a2) == len;
    for (int64_t t0 = 0; same && t0 < len; t0 += 32) {
        const int64_t t = t0 + lane;
        bool eq = true;
        if (t < len) {
            const int c0 = colind[a0 - base + t];
            eq = c0 == colind[a1 - base + t] && c0 == colind[a2 - base + t];
        }
        same = __all_sync(0xffffffffu, eq);
    }
    return same;
}

// Two matrices of one pattern, up to 48 basis columns, on the FP64 tensor cores: the three rows of a node and the two matrices are
// six of the eight rows of an m8n8k4 MMA whose k runs over four consecutive entries, and the gathered Vt rows
// are its B operand.  A lane reads two neighbouring columns at once (16 bytes, eight lanes a 128-byte line) and
// gives one to each of two MMAs, whose results for a lane are then four neighbouring columns.  With fused
// multiply-adds every entry's six values were broadcast to the lanes from shared memory, which took twice the
// arithmetic's time, and with fewer than 96 columns part of the lanes idle.  The gathers of 16 entries are in
// flight together with the next 32 entries' columns and values.  An MMA adds its four products in order, so
// the sums keep the order of the entries (Y's bits are those of spmm_rows); nodes whose rows differ in pattern
// go through spmm_rows.  k (at most 16 TP) and the row strides are even.  Bound by the gathers (a quarter-warp's 16-byte loads
// fall in four lines).  Tet10 block: 0.20 -> 0.14 ms at k = 32, 0.22 -> 0.20 ms at k = 48 (TP = 3 spills 48 bytes).  One or three
// matrices would fill three or nine rows of the eight: spmm_full_kernel.
template <int TP>
__global__ void __launch_bounds__(SPMM_THREADS, SPMM_MMA_CTAS) spmm_mma_kernel(int64_t N, const int64_t *__restrict__ rowptr,
                                                                   const int *__restrict__ colind, int base,
                                                                   ProjVals vals, const double *__restrict__ Vt, int k,
                                                                   int ldv, double *__restrict__ Y, int ldy,
                                                                   int64_t y_stride) {
    __shared__ SpmmStage stage[SPMM_WARPS];
    const int lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
    SpmmStage &st = stage[threadIdx.x >> 5];
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarp = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r0 = warp * 3; r0 < N; r0 += nwarp * 3) {
        const int nr = (int)min((int64_t)3, N - r0);
        const int64_t p0 = rowptr[r0], p1 = rowptr[r0 + 1], p2 = rowptr[min(r0 + 2, N)], p3 = rowptr[min(r0 + 3, N)];
        bool same = nr == 3 && p2 - p1 == p1 - p0 && p3 - p2 == p1 - p0;
        const int len = (int)(p1 - p0);
        if (same) {
            // MMA row lr: matrix row lr / 2 of the node, matrix lr & 1 (rows 6 and 7: none)
            const int rr = lr >> 1;
            const double *va = (lr & 1 ? vals.v[1] : vals.v[0]) + (p0 - base) + (int64_t)min(rr, 2) * len;
            const int *ci = colind + (p0 - base);
            const int live_a = lr < 6 ? len : 0;
            double acc[TP][2][2];
#pragma unroll
            for (int u = 0; u < TP; ++u) acc[u][0][0] = acc[u][0][1] = acc[u][1][0] = acc[u][1][1] = 0.0;
            int col = 0, col1 = 0, col2 = 0;
            double av[8];
            auto fetch = [&](int c0) {  // columns of the three rows and this lane's values of 32 entries
                const int e = min(c0 + lane, len - 1);
                col = ci[e] - base;
                col1 = ci[len + e] - base;
                col2 = ci[2 * len + e] - base;
#pragma unroll
                for (int g = 0; g < 8; ++g) av[g] = c0 + 4 * g + lk < live_a ? va[c0 + 4 * g + lk] : 0.0;
            };
            if (len > 0) fetch(0);
            for (int c0 = 0; c0 < len; c0 += 32) {
                same = __all_sync(0xffffffffu, col == col1 && col == col2);
                if (!same) break;
                const int mycol = col;
                double a[8];
#pragma unroll
                for (int g = 0; g < 8; ++g) a[g] = av[g];
                if (c0 + 32 < len) fetch(c0 + 32);
#pragma unroll
                for (int h = 0; h < 8; h += 4) {
                    if (c0 + 4 * h >= len) break;
                    double2 v[4][TP];
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const int cg = __shfl_sync(0xffffffffu, mycol, 4 * (h + g) + lk);
                        const double *vr = Vt + (int64_t)cg * ldv + 2 * lr;
                        const bool live = c0 + 4 * (h + g) + lk < len;
#pragma unroll
                        for (int u = 0; u < TP; ++u)
                            v[g][u] = live && 16 * u + 2 * lr < k ? *reinterpret_cast<const double2 *>(vr + 16 * u)
                                                                   : make_double2(0.0, 0.0);
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g)
#pragma unroll
                        for (int u = 0; u < TP; ++u) {
                            asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                                : "+d"(acc[u][0][0]), "+d"(acc[u][0][1]) : "d"(a[h + g]), "d"(v[g][u].x));
                            asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                                : "+d"(acc[u][1][0]), "+d"(acc[u][1][1]) : "d"(a[h + g]), "d"(v[g][u].y));
                        }
                }
            }
            if (same && lr < 6) {
                double *y = Y + (lr & 1) * y_stride + (r0 + rr) * ldy + 4 * lk;
#pragma unroll
                for (int u = 0; u < TP; ++u) {
                    const int c = 16 * u + 4 * lk;
                    if (c < k) *reinterpret_cast<double2 *>(y + 16 * u) = make_double2(acc[u][0][0], acc[u][1][0]);
                    if (c + 2 < k) *reinterpret_cast<double2 *>(y + 16 * u + 2) = make_double2(acc[u][0][1], acc[u][1][1]);
                }
            }
        }
        if (!same)
            for (int r = 0; r < nr; ++r)
                spmm_rows<(TP + 1) / 2, 2, 1>(r0 + r, rowptr, colind, base, vals, Vt, k, ldv, Y, ldy, y_stride, lane, st);
    }
}

template <int CPL, int NMAT>
__global__ void __launch_bounds__(SPMM_THREADS) spmm_full_kernel(int64_t N, const int64_t *__restrict__ rowptr,
                                                                 const int *__restrict__ colind, int base,
                                                                 ProjVals vals, const double *__restrict__ Vt, int k,
                                                                 int ldv, double *__restrict__ Y, int ldy,
                                                                 int64_t y_stride) {
    __shared__ SpmmStage stage[SPMM_WARPS];
    const int lane = threadIdx.x & 31;
    SpmmStage &st = stage[threadIdx.x >> 5];
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarp = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r0 = warp * 3; r0 < N; r0 += nwarp * 3) {
        const int nr = (int)min((int64_t)3, N - r0);
        const bool same = nr == 3 && same_columns(r0, rowptr, colind, base, lane);
        if (same) {
            spmm_rows<CPL, NMAT, 3>(r0, rowptr, colind, base, vals, Vt, k, ldv, Y, ldy, y_stride, lane, st);
        } else {
            for (int r = 0; r < nr; ++r)
                spmm_rows<CPL, NMAT, 1>(r0 + r, rowptr, colind, base, vals, Vt, k, ldv, Y, ldy, y_stride, lane, st);
        }
    }
}

// wave: at most one wave of resident CTAs (the node loop is grid-strided), else a warp a node
template <int CPL, int NMAT>
static void spmm_full_launch(int grid, bool wave, cudaStream_t st, int64_t N, const int64_t *rowptr, const int *colind,
                             int base, const ProjVals &vals, const double *Vt, int k, int ldv, double *Y, int ldy,
                             int64_t y_stride, int sms) {
    int per_sm = 0;
    if (wave && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, spmm_full_kernel<CPL, NMAT>, SPMM_THREADS, 0) ==
                    cudaSuccess && per_sm > 0)
        grid = std::min(grid, per_sm * sms);
    spmm_full_kernel<CPL, NMAT><<<grid, SPMM_THREADS, 0, st>>>(N, rowptr, colind, base, vals, Vt, k, ldv, Y, ldy,
                                                               y_stride);
}

template <int TP>
static void spmm_mma_launch(int grid, bool wave, cudaStream_t st, int64_t N, const int64_t *rowptr, const int *colind,
                            int base, const ProjVals &vals, const double *Vt, int k, int ldv, double *Y, int ldy,
                            int64_t y_stride, int sms) {
    if (wave) grid = std::min(grid, SPMM_MMA_CTAS * sms);
    spmm_mma_kernel<TP><<<grid, SPMM_THREADS, 0, st>>>(N, rowptr, colind, base, vals, Vt, k, ldv, Y, ldy, y_stride);
}

template <int CPL>
static void launch_spmm_full(int grid, bool wave, cudaStream_t st, int64_t N, const int64_t *rowptr, const int *colind,
                             int base, const ProjVals &vals, int n_mats, const double *Vt, int k, int ldv, double *Y,
                             int ldy, int64_t y_stride, int sms) {
    if (n_mats == 1) spmm_full_launch<CPL, 1>(grid, wave, st, N, rowptr, colind, base, vals, Vt, k, ldv, Y, ldy, y_stride, sms);
    else if (n_mats == 2) spmm_full_launch<CPL, 2>(grid, wave, st, N, rowptr, colind, base, vals, Vt, k, ldv, Y, ldy, y_stride, sms);
    else spmm_full_launch<CPL, 3>(grid, wave, st, N, rowptr, colind, base, vals, Vt, k, ldv, Y, ldy, y_stride, sms);
}

// Upper-triangle storage of a symmetric matrix (the reference's CSR,
// src/tools/MathLibrary.cpp:502-507): the mirrored entries (j, i), j != i, are added with
// FP64 atomics after the row pass above has written the stored half.
__global__ void spmm_upper_mirror_kernel(int64_t N, const int64_t *__restrict__ rowptr,
                                         const int *__restrict__ colind, int base, ProjVals vals, int n_mats,
                                         const double *__restrict__ Vt, int k, int ldv, double *__restrict__ Y,
                                         int ldy, int64_t y_stride) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarp = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t row = warp; row < N; row += nwarp) {
        const int64_t e0 = rowptr[row] - base, e1 = rowptr[row + 1] - base;
        for (int64_t e = e0; e < e1; ++e) {
            const int64_t col = colind[e] - base;
            if (col == row) continue;
            for (int c = lane; c < k; c += 32) {
                const double v = Vt[row * ldv + c];
                for (int m = 0; m < n_mats; ++m) atomicAdd(&Y[m * y_stride + col * ldy + c], vals.v[m][e] * v);
            }
        }
    }
}

// ---- R_m partial = Vt[rows]^T Y_m[rows] on FP64 tensor cores ------------------------------
// One launch covers nm matrices and one window of R: ka rows (basis columns of Vt, row stride
// ldv) by kb columns (columns of Y_m, row stride ldy), both <= 128.  The warps share
// out the matrices and the 8 x 8 tiles of the window.
// The rows of Vt and of the nm Y's are staged 32 at a time in shared memory (leading
// dimension padded by 4 keeps the fragment loads free of bank conflicts); the Vt chunk is
// staged once for all nm matrices, and the chunks are double-buffered with cp.async so the
// loads of chunk c + 1 overlap the MMAs of chunk c.  Each CTA takes a contiguous range of
// chunks and writes a private kap x kbp partial.
__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src));
}

struct VtyWindow {
    const double *Vt;  // first basis column of the window's rows
    int ka, ldv;
    const double *Y;   // first column of the window's columns (matrix 0)
    int kb, ldy;
    int64_t y_stride;  // between matrices
};

// A warp's share is two 8-row bands by half of the tiles across: eight fragment reads for twelve MMAs (one
// band by all tiles took thirteen, and the shared-memory datapath as long as the MMAs).  PAIRS: rows of even
// length, copied 16 bytes at a time.
template <int TH, int MAXT, bool PAIRS>
__global__ void __launch_bounds__(MAXT) vty_partial_kernel(int64_t N, VtyWindow w, int nm, int64_t chunks_per_cta,
                                                           double *__restrict__ partial) {
    extern __shared__ __align__(16) double sh[];
    const int kap = (w.ka + 7) & ~7, kbp = (w.kb + 7) & ~7;
    const int lda = kap + 4, ldb = kbp + 4;
    const int nband = kap / 8, ntile = kbp / 8, nbp = (nband + 1) / 2, th = (ntile + 1) / 2;
    const int a_sz = 32 * lda, b_sz = 32 * ldb;
    const int stage = a_sz + nm * b_sz;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    // lanes to a row, and rows to a warp's pass, of the copies: a whole warp a row left most lanes of narrow windows
    // idle (107,163 rows, one matrix: k = 8 0.140 ms, k = 16 0.140; with the lanes shared out 0.033 and 0.044)
    constexpr int PER = PAIRS ? 2 : 1;
    const int need = TH > 2 ? 32 : max(kap, kbp) / PER;  // TH > 2: more than 32 columns across
    const int lpr = need <= 4 ? 4 : need <= 8 ? 8 : need <= 16 ? 16 : 32, rpw = 32 / lpr;
    const int mloc = warp / (2 * nbp), band0 = warp % (2 * nbp) / 2 * 2, t0 = (warp & 1) * th;
    const bool second = band0 + 1 < nband;
    const int nt = min(th, ntile - t0);
    const int64_t n_chunks = (N + 31) / 32;
    const int64_t c_begin = (int64_t)blockIdx.x * chunks_per_cta;
    const int64_t c_end = min(n_chunks, c_begin + chunks_per_cta);

    auto issue = [&](int64_t ch, int buf) {
        double *dst0 = sh + buf * stage;
        const int64_t r0 = ch * 32;
        const int nr = (int)min((int64_t)32, N - r0);
        for (int row = warp * rpw + lane / lpr; row < 32 * (1 + nm); row += nw * rpw) {
            const int rr = row & 31, which = row >> 5;  // 0: Vt, else matrix which - 1
            const bool isa = which == 0;
            const int kk = isa ? w.ka : w.kb, kp = isa ? kap : kbp;
            double *dst = dst0 + (isa ? rr * lda : a_sz + (which - 1) * b_sz + rr * ldb);
            const double *src = isa ? w.Vt + (r0 + rr) * w.ldv : w.Y + (which - 1) * w.y_stride + (r0 + rr) * w.ldy;
            for (int c = PER * (lane % lpr); c < kp; c += lpr * PER) {
                const unsigned d = (unsigned)__cvta_generic_to_shared(dst + c);
                if (rr < nr && c < kk) {
                    if constexpr (PAIRS) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + c));
                    else cp_async8(dst + c, src + c);
                } else {
#pragma unroll
                    for (int h = 0; h < PER; ++h) dst[c + h] = 0.0;
                }
            }
        }
        asm volatile("cp.async.commit_group;");
    };

    double acc[2][TH][2];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int t = 0; t < TH; ++t) acc[x][t][0] = acc[x][t][1] = 0.0;
    if (c_begin < c_end) issue(c_begin, 0);
    for (int64_t ch = c_begin; ch < c_end; ++ch) {
        const int buf = (int)((ch - c_begin) & 1);
        if (ch + 1 < c_end) {
            issue(ch + 1, buf ^ 1);
            asm volatile("cp.async.wait_group 1;");
        } else {
            asm volatile("cp.async.wait_group 0;");
        }
        __syncthreads();
        {
            const double *sV = sh + buf * stage + 8 * band0 + (lane >> 2);
            const double *sY = sh + buf * stage + a_sz + mloc * b_sz + 8 * t0 + (lane >> 2);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                const int rr = 4 * kk + (lane & 3);
                const double a0 = sV[rr * lda], a1 = second ? sV[rr * lda + 8] : 0.0;
#pragma unroll
                for (int t = 0; t < TH; ++t) {
                    if (t < nt) {
                        const double b = sY[rr * ldb + 8 * t];
                        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                                     : "+d"(acc[0][t][0]), "+d"(acc[0][t][1])
                                     : "d"(a0), "d"(b));
                        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                                     : "+d"(acc[1][t][0]), "+d"(acc[1][t][1])
                                     : "d"(a1), "d"(b));
                    }
                }
            }
        }
        __syncthreads();
    }
    // lane holds D[row = lane/4][col = 2*(lane%4) + {0,1}] of tile (band, t)
    double *P = partial + ((int64_t)mloc * gridDim.x + blockIdx.x) * kap * kbp;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        if (x == 1 && !second) break;
        const int ra = 8 * (band0 + x) + (lane >> 2);
#pragma unroll
        for (int t = 0; t < TH; ++t) {
            if (t < nt) {
                const int cb = 8 * (t0 + t) + 2 * (lane & 3);
                P[ra + (int64_t)cb * kap] = acc[x][t][0];
                P[ra + (int64_t)(cb + 1) * kap] = acc[x][t][1];
            }
        }
    }
}

// Sum of part[blk * stride] over the CTA partials, by RED_SEG threads an element (threadIdx.y): segment y
// takes blk = y, y + RED_SEG, ..., and the segments are added in order (deterministic).  With one thread an
// element the few thousand elements of a small result left the GPU idle on one chain of nblk loads
// (43 us for two 96 x 96 results of 148 partials, 59 us for a Gram-Schmidt panel).  Valid in segment 0.
constexpr int RED_SEG = 16;
__device__ __forceinline__ double sum_partials(const double *__restrict__ part, int nblk, int64_t stride, bool live) {
    __shared__ double red[RED_SEG][33];
    double s = 0.0;
    if (live) {
#pragma unroll 5
        for (int blk = threadIdx.y; blk < nblk; blk += RED_SEG) s += part[(int64_t)blk * stride];
    }
    red[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    s = 0.0;
    if (threadIdx.y == 0) {
#pragma unroll
        for (int y = 0; y < RED_SEG; ++y) s += red[y][threadIdx.x];
    }
    return s;
}

// out.r[m][a + b * ldr] = sum over the CTA partials
__global__ void reduce_partials_kernel(const double *__restrict__ partial, int nblk, int nmat, int ka, int kb,
                                       int kap, int kbp, ProjOut out, int ldr) {
    const int64_t e = (int64_t)blockIdx.x * 32 + threadIdx.x;
    const bool live = e < (int64_t)nmat * ka * kb;
    const int m = live ? (int)(e / ((int64_t)ka * kb)) : 0;
    const int rem = live ? (int)(e % ((int64_t)ka * kb)) : 0;
    const int a = rem % ka, b = rem / ka;
    const double s = sum_partials(partial + (int64_t)m * nblk * kap * kbp + a + (int64_t)b * kap, nblk, (int64_t)kap * kbp, live);
    if (live && threadIdx.y == 0) out.r[m][a + (int64_t)b * ldr] = s;
}

// ---- block Gram-Schmidt with re-orthogonalisation --------------------------------------
// The columns of V (column-major, N x k, ldv) are taken in panels P of GS_B columns.  One pass
// over a panel with the orthonormal columns Q = V[:, :j0] before it:
//     C = [Q P]^T P                 (one reduction: H = Q^T P on top, G = P^T P below)
//     R^T R = G - H^T H             (Cholesky; the Gram matrix of P - Q H by Pythagoras)
//     P <- (P - Q H) R^-1
// and `passes` passes are made (two keep the basis orthonormal to rounding level).  This is
// the reference's block scheme -- block projection against V repeated, then an orthonormal
// basis of the block (KrylovROMSubstructure.cpp:433-475, :513-534) -- with the QR of the block
// taken through its Gram matrix so that every pass is one reduction and one row update.
constexpr int GS_B = 32;        // panel width
constexpr int GS_WIN = 128;     // columns of [Q P] per reduction launch (16 bands of 8)
constexpr int GS_LDR = 36;      // staged column stride (32 rows + 4: conflict-free fragments)
constexpr int GS_THREADS = 512;
constexpr int GS_HCHUNK = 128;  // rows of H staged per round of the row update

// part[blk][x0 + i][c] = sum over this CTA's rows of V[r, x0 + i] * V[r, j0 + c]
// (i < w, c < b), on the FP64 tensor cores; chunks of 32 rows through a ring of GS_STAGES cp.async
// stages (one CTA an SM: with two stages too little was in flight to reach the L2's rate).  PAIRS: V and ldv
// allow 16-byte copies of two rows.  The panel is staged once where the window ends with it.
constexpr int GS_STAGES = 4;
template <bool PAIRS>
__global__ void __launch_bounds__(GS_THREADS) gs_gram_kernel(const double *__restrict__ V, int64_t N, int64_t ldv,
                                                             int x0, int w, int j0, int b, int rows_c,
                                                             int64_t chunks_per_cta, double *__restrict__ part) {
    extern __shared__ __align__(16) double sh[];
    const int wp = (w + 7) & ~7, bp = (b + 7) & ~7;
    const bool own = x0 + w == j0 + b && w >= b;  // the window's last columns are the panel
    const int po = own ? w - b : wp;              // staged column of the panel's first
    const int cols = own ? po + bp : wp + bp;     // wp <= cols, as w = po + b
    const int stage = (GS_WIN + GS_B) * GS_LDR;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nband = wp / 8, ntile = bp / 8;
    const int64_t n_chunks = (N + 31) / 32;
    const int64_t c_begin = (int64_t)blockIdx.x * chunks_per_cta;
    const int64_t c_end = min(n_chunks, c_begin + chunks_per_cta);

    auto issue = [&](int64_t ch) {
        if (ch < c_end) {
            double *dst0 = sh + (int)((ch - c_begin) % GS_STAGES) * stage;
            const int64_t r0 = ch * 32;
            const int nr = (int)min((int64_t)32, N - r0);
            constexpr int LPC = PAIRS ? 16 : 32;  // lanes a column
            for (int col = threadIdx.x / LPC; col < cols; col += GS_THREADS / LPC) {
                const int rr = (threadIdx.x % LPC) * (32 / LPC);
                const bool isp = col >= po;
                const int cc = isp ? col - po : col;
                const bool ok = isp ? cc < b : cc < w;
                double *dst = dst0 + col * GS_LDR + rr;
                const double *src = V + r0 + rr + (int64_t)(isp ? j0 + cc : x0 + cc) * ldv;
                const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
                if (PAIRS && ok && rr + 1 < nr) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src));
                } else {
#pragma unroll
                    for (int h = 0; h < 32 / LPC; ++h) {
                        if (ok && rr + h < nr)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + 8 * h), "l"(src + h));
                        else
                            dst[h] = 0.0;
                    }
                }
            }
        }
        asm volatile("cp.async.commit_group;");
    };

    double acc[4][2];
#pragma unroll
    for (int t = 0; t < 4; ++t) acc[t][0] = acc[t][1] = 0.0;
    for (int q = 0; q < GS_STAGES - 1; ++q) issue(c_begin + q);
    for (int64_t ch = c_begin; ch < c_end; ++ch) {
        const int buf = (int)((ch - c_begin) % GS_STAGES);
        asm volatile("cp.async.wait_group %0;" ::"n"(GS_STAGES - 2));
        __syncthreads();  // the chunk is in; everyone is done with the one before, whose place the next takes
        issue(ch + GS_STAGES - 1);
        if (warp < nband) {
            const double *sX = sh + buf * stage;
            const double *sP = sX + po * GS_LDR;
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                const int rr = 4 * kk + (lane & 3);
                const double a = sX[(8 * warp + (lane >> 2)) * GS_LDR + rr];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if (t < ntile) {
                        const double bv = sP[(8 * t + (lane >> 2)) * GS_LDR + rr];
                        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                                     : "+d"(acc[t][0]), "+d"(acc[t][1])
                                     : "d"(a), "d"(bv));
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;");
    if (warp < nband) {
        const int i = x0 + 8 * warp + (lane >> 2);
        double *P = part + (int64_t)blockIdx.x * rows_c * GS_B;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int c = 8 * t + 2 * (lane & 3);
            if (i < rows_c) {  // tiles past b hold zeros
                P[(int64_t)i * GS_B + c] = acc[t][0];
                P[(int64_t)i * GS_B + c + 1] = acc[t][1];
            }
        }
    }
}

// C[i][c] = sum_blk part[blk][i][c]
__global__ void gs_reduce_kernel(const double *__restrict__ part, int nblk, int rows_c, double *__restrict__ Cm) {
    const int64_t tot = (int64_t)rows_c * GS_B, e = (int64_t)blockIdx.x * 32 + threadIdx.x;
    const double s = sum_partials(part + e, nblk, tot, e < tot);
    if (e < tot && threadIdx.y == 0) Cm[e] = s;
}

// One CTA: G' = G - H^T H, Cholesky R^T R = G', Rinv = R^-1 (upper), written to rinv[a][c].  Thread (a, c)
// holds rows a, a + 8, a + 16, a + 24 of column c.  The elimination multiplies by the pivot's reciprocal (one
// a step, 31 dependent steps) and the rows are scaled by 1 / sqrt(pivot) at the end; Rinv's columns take a lane
// each, right-looking, in registers.
constexpr int GS_CT = 256, GS_CR = GS_B * GS_B / GS_CT;
__global__ void __launch_bounds__(GS_CT) gs_chol_kernel(const double *__restrict__ Cm, int j0, int b,
                                                        double *__restrict__ rinv) {
    __shared__ double G[GS_B][GS_B + 1];
    __shared__ double rd[GS_B];  // 1 / R[j][j]
    const int a0 = threadIdx.x / GS_B, c = threadIdx.x % GS_B;
    double g[GS_CR];
#pragma unroll
    for (int q = 0; q < GS_CR; ++q) g[q] = 0.0;
#pragma unroll 4
    for (int i = 0; i < j0; ++i) {
        const double hc = Cm[(int64_t)i * GS_B + c];
#pragma unroll
        for (int q = 0; q < GS_CR; ++q) g[q] = fma(Cm[(int64_t)i * GS_B + a0 + 8 * q], hc, g[q]);
    }
    bool tiny = false;
#pragma unroll
    for (int q = 0; q < GS_CR; ++q) {
        const int a = a0 + 8 * q;
        // unit diagonal past a short panel
        g[q] = a < b && c < b ? Cm[(int64_t)(j0 + a) * GS_B + c] - g[q] : (a == c ? 1.0 : 0.0);
        tiny = tiny || (a == c && g[q] < 0x1p-900);
        G[a][c] = g[q];
    }
    // G = L D L^T by rows: row j is final before step j, and R[j][c] = G[j][c] / sqrt(G[j][j])
    auto step = [&](int j, double t) {
#pragma unroll
        for (int q = 0; q < GS_CR; ++q) {
            const int a = a0 + 8 * q;
            if (a > j && c > j) {
                g[q] = fma(-G[j][a], t, g[q]);
                G[a][c] = g[q];  // read only as row a of a later step
            }
        }
        __syncthreads();
    };
    // columns of norm below about 1e-154 have pivots whose reciprocal overflows: panels with a small diagonal entry (a
    // pivot is smaller by 2^-53 at most, short of breaking down) divide.  (Chosen pivot by pivot, the test cost every
    // panel 1.5 us.)
    if (__syncthreads_or(tiny)) {
        for (int j = 0; j + 1 < b; ++j) step(j, G[j][c] / G[j][j]);
    } else {
        for (int j = 0; j + 1 < b; ++j) step(j, G[j][c] * __drcp_rn(G[j][j]));
    }
    if (a0 == 0) rd[c] = 1.0 / sqrt(G[c][c]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < GS_CR; ++q) {
        const int a = a0 + 8 * q;
        if (a < c) G[a][c] = g[q] * rd[a];
    }
    __syncthreads();
    if (threadIdx.x < GS_B) {
        // column c of R^-1: x_i = (e_c - sum_{l > i} R[i][l] x_l) / R[i][i] from the last row
        double x[GS_B];
#pragma unroll
        for (int i = 0; i < GS_B; ++i) x[i] = i == c && c < b ? 1.0 : 0.0;
#pragma unroll
        for (int l = GS_B - 1; l >= 0; --l) {
            // rows below the diagonal stay out: at a pivot that broke down (a column dependent on those before it)
            // rd[l] and G[.][l] are not finite, and 0 times them would spread to the columns before
            if (l <= c) {
                x[l] *= rd[l];
#pragma unroll
                for (int i = 0; i < l; ++i) x[i] = fma(-G[i][l], x[l], x[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < GS_B; ++i) rinv[i * GS_B + c] = i <= c ? x[i] : 0.0;
    }
}

// p <- (p - q H) Rinv with q = V[r, :j0] and p = V[r, j0:j0+b]: 16 rows a warp, both products on the FP64
// tensor cores (H from shared memory, the rows of V straight from global memory in fragment order, p - q H
// through shared memory into the second product's A operand).  HBM / L2 bound; as fused multiply-adds with H
// broadcast from shared memory every row cost eight 16-byte reads for 16 multiply-adds.
constexpr int GS_UW = 8;             // warps of a CTA, 16 rows each
constexpr int GS_LDB = GS_B + 4;     // 4 modulo 16 doubles: conflict-free fragments
__device__ __forceinline__ void gs_dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}
__global__ void __launch_bounds__(32 * GS_UW, 3) gs_update_kernel(double *__restrict__ V, int64_t N, int64_t ldv, int j0, int b,
                                                        const double *__restrict__ Cm, const double *__restrict__ rinv) {
    __shared__ double Hs[GS_HCHUNK * GS_LDB];  // rows of H; later the warps' p - q H
    __shared__ double Rs[GS_B * GS_LDB];
    static_assert(GS_UW * 16 <= GS_HCHUNK, "the warps' rows fit the place of H");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane >> 2, lk = lane & 3;
    for (int e = threadIdx.x; e < GS_B * GS_B; e += blockDim.x) Rs[e / GS_B * GS_LDB + e % GS_B] = rinv[e];
    const int64_t r0 = ((int64_t)blockIdx.x * GS_UW + warp) * 16;
    double acc[2][4][2];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t r = r0 + 8 * x + lr;
                const int c = 8 * t + 2 * lk + h;
                acc[x][t][h] = (r < N && c < b) ? V[r + (int64_t)(j0 + c) * ldv] : 0.0;
            }
    for (int i0 = 0; i0 < j0; i0 += GS_HCHUNK) {
        const int ni = min(GS_HCHUNK, j0 - i0);  // a multiple of GS_B
        __syncthreads();
        for (int e = threadIdx.x; e < ni * GS_B; e += blockDim.x)
            Hs[e / GS_B * GS_LDB + e % GS_B] = Cm[(int64_t)i0 * GS_B + e];
        __syncthreads();
#pragma unroll 4
        for (int i = 0; i < ni; i += 4) {
            double q[2], h[4];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int64_t r = r0 + 8 * x + lr;
                q[x] = r < N ? -V[r + (int64_t)(i0 + i + lk) * ldv] : 0.0;
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) h[t] = Hs[(i + lk) * GS_LDB + 8 * t + lr];
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int t = 0; t < 4; ++t) gs_dmma(acc[x][t], q[x], h[t]);
        }
    }
    __syncthreads();
    double *T = Hs + warp * 16 * GS_LDB;
    bool finite = true;
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                T[(8 * x + lr) * GS_LDB + 8 * t + 2 * lk + h] = acc[x][t][h];
                finite = finite && fabs(acc[x][t][h]) <= DBL_MAX;
                acc[x][t][h] = 0.0;
            }
    finite = __all_sync(0xffffffffu, finite);
    __syncwarp();
    if (!finite) {
        // a column that broke down in the pass before, or came in not finite: the zeros below Rinv's diagonal would
        // carry it into the columns before it in the same 8-column tile, so these sums end at the diagonal
#pragma unroll 1
        for (int e = lane; e < 16 * b; e += 32) {
            const int row = e & 15, c = e >> 4;
            double s = 0.0;
#pragma unroll 1
            for (int k = 0; k <= c; ++k) s = fma(T[row * GS_LDB + k], Rs[k * GS_LDB + c], s);
            if (r0 + row < N) V[r0 + row + (int64_t)(j0 + c) * ldv] = s;
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < GS_B; k += 4) {
        double p[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) p[x] = T[(8 * x + lr) * GS_LDB + k + lk];
#pragma unroll
        for (int t = k / 8; t < 4; ++t) {  // Rinv is upper triangular
            const double rv = Rs[(k + lk) * GS_LDB + 8 * t + lr];
#pragma unroll
            for (int x = 0; x < 2; ++x) gs_dmma(acc[x][t], p[x], rv);
        }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t r = r0 + 8 * x + lr;
                const int c = 8 * t + 2 * lk + h;
                if (r < N && c < b) V[r + (int64_t)(j0 + c) * ldv] = acc[x][t][h];
            }
}

// ---- complex projection R = Z^H A V through the real kernels ------------------------------
// With A = Ar + i Ai and the basis stored as the real N x 2k rows [Re V | Im V], the real SpMM
// over the two value arrays (Ar, Ai) gives P_r = Ar [Vr | Vi] and P_i = Ai [Vr | Vi]; then
// Y = A V has Re Y = Ar Vr - Ai Vi and Im Y = Ar Vi + Ai Vr (combined in place into P_r's rows
// as [Re Y | Im Y]), and the real V^T Y kernel on W = [Re Z | Im Z] gives G = W^T [Re Y | Im Y],
// whose four k x k blocks combine into Z^H Y = (Zr^T Yr + Zi^T Yi) + i (Zr^T Yi - Zi^T Yr).

// V (complex, column-major, ldv) -> Wt (real, row-major N x 2k: [Re V(row) | Im V(row)])
__global__ void transpose_split_kernel(const double2 *__restrict__ V, int64_t N, int k, int64_t ldv,
                                       double *__restrict__ Wt) {
    __shared__ double2 t[32][33];
    const int64_t r0 = (int64_t)blockIdx.x * 32;
    const int c0 = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int64_t r = r0 + threadIdx.x;
        const int c = c0 + y;
        if (r < N && c < k) t[y][threadIdx.x] = V[r + (int64_t)c * ldv];
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int64_t r = r0 + y;
        const int c = c0 + threadIdx.x;
        if (r < N && c < k) {
            const double2 v = t[threadIdx.x][y];
            Wt[r * 2 * k + c] = v.x;
            Wt[r * 2 * k + k + c] = v.y;
        }
    }
}

// complex values -> separate real and imaginary arrays
__global__ void split_values_kernel(const double2 *__restrict__ a, int64_t nnz, double *__restrict__ re,
                                    double *__restrict__ im) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += (int64_t)gridDim.x * blockDim.x) {
        const double2 v = a[e];
        re[e] = v.x;
        im[e] = v.y;
    }
}

// rows of P_r = [Ar Vr | Ar Vi] and P_i = [Ai Vr | Ai Vi] -> rows of P_r = [Re Y | Im Y]
__global__ void combine_y_kernel(double *__restrict__ Pr, const double *__restrict__ Pi, int64_t N, int k) {
    const int64_t tot = N * k;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / k;
        const int c = (int)(e % k);
        double *pr = Pr + r * 2 * k;
        const double *pi = Pi + r * 2 * k;
        const double yr = pr[c] - pi[k + c];
        const double yi = pr[k + c] + pi[c];
        pr[c] = yr;
        pr[k + c] = yi;
    }
}

// G (2k x 2k, column-major) -> R (k x k complex, column-major)
__global__ void combine_r_kernel(const double *__restrict__ G, int k, double2 *__restrict__ R) {
    const int k2 = 2 * k;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < k * k; e += gridDim.x * blockDim.x) {
        const int a = e % k, b = e / k;
        const double re = G[a + (int64_t)b * k2] + G[(k + a) + (int64_t)(k + b) * k2];
        const double im = G[a + (int64_t)(k + b) * k2] - G[(k + a) + (int64_t)b * k2];
        R[a + (int64_t)b * k] = make_double2(re, im);
    }
}

cudaError_t launch_transpose_split(const double2 *V, int64_t N, int k, int64_t ldv, double *Wt, cudaStream_t st) {
    dim3 grid((unsigned)((N + 31) / 32), (unsigned)((k + 31) / 32)), block(32, 8);
    transpose_split_kernel<<<grid, block, 0, st>>>(V, N, k, ldv, Wt);
    return cudaGetLastError();
}

cudaError_t launch_split_values(const double2 *a, int64_t nnz, double *re, double *im, int sms, cudaStream_t st) {
    const int grid = (int)std::min<int64_t>((nnz + 255) / 256, (int64_t)sms * 8);
    if (grid > 0) split_values_kernel<<<grid, 256, 0, st>>>(a, nnz, re, im);
    return cudaGetLastError();
}

cudaError_t launch_combine_y(double *Pr, const double *Pi, int64_t N, int k, int sms, cudaStream_t st) {
    const int grid = (int)std::min<int64_t>((N * k + 255) / 256, (int64_t)sms * 8);
    if (grid > 0) combine_y_kernel<<<grid, 256, 0, st>>>(Pr, Pi, N, k);
    return cudaGetLastError();
}

cudaError_t launch_combine_r(const double *G, int k, double2 *R, cudaStream_t st) {
    combine_r_kernel<<<(k * k + 255) / 256, 256, 0, st>>>(G, k, R);
    return cudaGetLastError();
}

// ---- host launchers -------------------------------------------------------------------------
cudaError_t launch_transpose(const double *V, int64_t N, int k, int64_t ldv, double *Vt, cudaStream_t st) {
    dim3 grid((unsigned)((N + 31) / 32), (unsigned)((k + 31) / 32)), block(32, 8);
    transpose_kernel<<<grid, block, 0, st>>>(V, N, k, ldv, Vt);
    return cudaGetLastError();
}

cudaError_t launch_spmm(int64_t N, const int64_t *rowptr, const int *colind, int base, int upper, ProjVals vals,
                        int n_mats, const double *Vt, int k, double *Y, int64_t y_stride, int sms, cudaStream_t st) {
    const int threads = SPMM_THREADS;
    const int64_t warps_needed = (N + 2) / 3;
    const int grid = (int)std::min<int64_t>((warps_needed * 32 + threads - 1) / threads, 1 << 30);
    // window by window (PRJ_WIN columns of the basis at a time), each into its columns of Y
    for (int j0 = 0; j0 < k; j0 += PRJ_WIN) {
        const int kw = std::min(PRJ_WIN, k - j0);
        const double *Vw = Vt + j0;
        double *Yw = Y + j0;
        // Narrow windows of many nodes have little work a CTA and average out in one wave: 107,163 rows, a CTA a
        // four nodes against one wave: k = 32 166 / 149 us (one matrix), 152 / 141 (two), 262 / 252 (three), k = 64 236 /
        // 225 (two; one matrix 158 / 196).  At 41,175 rows k = 32 takes 58 / 66 us, 67 / 76 and 115 / 149.
        const bool wave = (kw <= 32 || (n_mats == 2 && kw <= 64)) && warps_needed > (int64_t)160 * sms;
        // two matrices, even rows (the window starts on a multiple of 128 columns), up to 48 columns: the tensor
        // cores.  Beyond, a node's gathers no longer fit one warp's registers and its values and columns are read
        // once a 48-column part (Tet10 block: 0.20 against 0.22 ms at 48 columns, 0.26 against 0.22 at 64)
        if (n_mats == 2 && kw <= 48 && (k & 1) == 0 && (y_stride & 1) == 0) {
            auto go = kw <= 32 ? spmm_mma_launch<2> : spmm_mma_launch<3>;
            go(grid, wave, st, N, rowptr, colind, base, vals, Vw, kw, k, Yw, k, y_stride, sms);
        } else if (kw <= 32) launch_spmm_full<1>(grid, wave, st, N, rowptr, colind, base, vals, n_mats, Vw, kw, k, Yw, k, y_stride, sms);
        else if (kw <= 64) launch_spmm_full<2>(grid, wave, st, N, rowptr, colind, base, vals, n_mats, Vw, kw, k, Yw, k, y_stride, sms);
        else if (kw <= 96) launch_spmm_full<3>(grid, wave, st, N, rowptr, colind, base, vals, n_mats, Vw, kw, k, Yw, k, y_stride, sms);
        else launch_spmm_full<4>(grid, wave, st, N, rowptr, colind, base, vals, n_mats, Vw, kw, k, Yw, k, y_stride, sms);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (upper) {
            spmm_upper_mirror_kernel<<<std::min(grid, 16 * sms), threads, 0, st>>>(N, rowptr, colind, base, vals, n_mats, Vw, kw, k,
                                                                                   Yw, k, y_stride);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

// Matrices per launch of vty_partial_kernel: a matrix takes two warps a pair of 8-row bands, and a launch at most
// 24 warps (768 threads, <= 85 registers a thread) for windows up to 12 tiles wide, 16 (512) for wider ones.
constexpr int vty_warps(int nband) { return 2 * ((nband + 1) / 2); }
constexpr int vty_max_warps(int ntile) { return ntile > 12 ? 16 : 24; }
constexpr int vty_group(int nband, int ntile, int n_mats) {
    return std::max(1, std::min(n_mats, vty_max_warps(ntile) / vty_warps(nband)));
}
constexpr size_t vty_smem(int nband, int ntile, int nm) {  // two chunks of 32 rows, leading dimensions padded by 4
    return sizeof(double) * (size_t)2 * 32 * ((8 * nband + 4) + (size_t)nm * (8 * ntile + 4));
}
// every window and matrix count: the launch's threads within its bound, its shared memory within a CTA's 227 KB
constexpr bool vty_fits() {
    for (int nband = 1; nband <= PRJ_WIN / 8; ++nband)
        for (int ntile = 1; ntile <= PRJ_WIN / 8; ++ntile)
            for (int n_mats = 1; n_mats <= PRJ_MAX_MATS; ++n_mats) {
                const int nm = vty_group(nband, ntile, n_mats);
                if (nm * vty_warps(nband) > vty_max_warps(ntile) || vty_smem(nband, ntile, nm) > (size_t)227 * 1024)
                    return false;
            }
    return true;
}
static_assert(vty_fits(), "vty_partial_kernel's launches fit their bounds");

size_t vty_partial_doubles(int k, int n_mats, int nblk) {
    const int kp = (std::min(k, PRJ_WIN) + 7) & ~7;
    return (size_t)nblk * n_mats * kp * kp;
}

template <int TH, int MAXT>
static cudaError_t vty_launch(int64_t N, const VtyWindow &w, int nm, int nblk, double *partial, cudaStream_t st) {
    const int nband = (w.ka + 7) / 8, ntile = (w.kb + 7) / 8;
    const int threads = 32 * nm * vty_warps(nband);
    const size_t smem = vty_smem(nband, ntile, nm);
    // rows of even length: every row of Vt and Y starts on 16 bytes
    const bool pairs = ((w.ldv | w.ldy | w.ka | w.kb) & 1) == 0 && (w.y_stride & 1) == 0 &&
                       ((reinterpret_cast<uintptr_t>(w.Vt) | reinterpret_cast<uintptr_t>(w.Y)) & 15) == 0;
    auto kf = pairs ? vty_partial_kernel<TH, MAXT, true> : vty_partial_kernel<TH, MAXT, false>;
    // one value for all sizes: another thread's smaller launch must not lower it between this call and this launch
    cudaError_t e = cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    const int64_t n_chunks = (N + 31) / 32;
    const int64_t per = (n_chunks + nblk - 1) / nblk;
    kf<<<nblk, threads, smem, st>>>(N, w, nm, per, partial);
    return cudaGetLastError();
}

// R_m = Vt^T Y_m (k x k, leading dimension k) window by window: PRJ_WIN x PRJ_WIN blocks of R,
// each one DMMA pass over the rows plus a deterministic reduction into its block.
cudaError_t launch_vty(int64_t N, int k, const double *Vt, const double *Y, int64_t y_stride, int n_mats,
                       int nblk, double *partial, ProjOut out, cudaStream_t st) {
    for (int i0 = 0; i0 < k; i0 += PRJ_WIN) {
        const int ka = std::min(PRJ_WIN, k - i0);
        const int kap = (ka + 7) & ~7;
        for (int j0 = 0; j0 < k; j0 += PRJ_WIN) {
            const int kb = std::min(PRJ_WIN, k - j0);
            const int kbp = (kb + 7) & ~7, ntile = kbp / 8;
            const int group = vty_group(kap / 8, ntile, n_mats);
            for (int m0 = 0; m0 < n_mats; m0 += group) {
                const int nm = std::min(group, n_mats - m0);
                const VtyWindow w{Vt + i0, ka, k, Y + m0 * y_stride + j0, kb, k, y_stride};
                double *Pm = partial + (int64_t)m0 * nblk * kap * kbp;
                cudaError_t e;
                if (ntile <= 4) e = vty_launch<2, 32 * vty_max_warps(4)>(N, w, nm, nblk, Pm, st);
                else if (ntile <= 8) e = vty_launch<4, 32 * vty_max_warps(8)>(N, w, nm, nblk, Pm, st);
                else if (ntile <= 12) e = vty_launch<6, 32 * vty_max_warps(12)>(N, w, nm, nblk, Pm, st);
                else e = vty_launch<8, 32 * vty_max_warps(16)>(N, w, nm, nblk, Pm, st);
                if (e != cudaSuccess) return e;
            }
            ProjOut o{};
            for (int m = 0; m < n_mats; ++m) o.r[m] = out.r[m] + i0 + (int64_t)j0 * k;
            const int64_t tot = (int64_t)n_mats * ka * kb;
            reduce_partials_kernel<<<(int)((tot + 31) / 32), dim3(32, RED_SEG), 0, st>>>(partial, nblk, n_mats, ka, kb, kap,
                                                                                       kbp, o, k);
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

size_t gs_workspace_doubles(int k, int nblk) {
    const size_t rows_c = (size_t)((k + 7) & ~7) + GS_B;
    return (size_t)nblk * rows_c * GS_B + rows_c * GS_B + (size_t)GS_B * GS_B;
}

cudaError_t launch_gram_schmidt(double *V, int64_t N, int k, int64_t ldv, int passes, double *work, int nblk,
                                cudaStream_t st) {
    const int rows_max = ((k + 7) & ~7) + GS_B;
    double *part = work;
    double *Cm = part + (size_t)nblk * rows_max * GS_B;
    double *rinv = Cm + (size_t)rows_max * GS_B;
    const size_t smem = sizeof(double) * (size_t)GS_STAGES * (GS_WIN + GS_B) * GS_LDR;
    const bool pairs = (reinterpret_cast<uintptr_t>(V) & 15) == 0 && (ldv & 1) == 0;
    auto gram = pairs ? gs_gram_kernel<true> : gs_gram_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(gram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int64_t n_chunks = (N + 31) / 32;
    const int64_t per = (n_chunks + nblk - 1) / nblk;
    const int ugrid = (int)((N + 16 * GS_UW - 1) / (16 * GS_UW));
    passes = std::max(passes, 1);
    for (int j0 = 0; j0 < k; j0 += GS_B) {
        const int b = std::min(GS_B, k - j0);
        const int rows_c = j0 + ((b + 7) & ~7);  // rows of C: Q's j0 columns, then P's (padded)
        for (int pass = 0; pass < passes; ++pass) {
            for (int x0 = 0; x0 < j0 + b; x0 += GS_WIN) {
                const int w = std::min(GS_WIN, j0 + b - x0);
                gram<<<nblk, GS_THREADS, smem, st>>>(V, N, ldv, x0, w, j0, b, rows_c, per, part);
            }
            const int64_t tot = (int64_t)rows_c * GS_B;
            gs_reduce_kernel<<<(int)((tot + 31) / 32), dim3(32, RED_SEG), 0, st>>>(part, nblk, rows_c, Cm);
            gs_chol_kernel<<<1, GS_CT, 0, st>>>(Cm, j0, b, rinv);
            gs_update_kernel<<<ugrid, 32 * GS_UW, 0, st>>>(V, N, ldv, j0, b, Cm, rinv);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

}  // namespace srom
