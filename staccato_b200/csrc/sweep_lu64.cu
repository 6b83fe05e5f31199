// FP64 sweep of orders up to 512: one CTA a (ROM, frequency) system, one thread a matrix row,
// Schur updates on the FP64 tensor cores (mma.sync m8n8k4 f64).
//
// Per system: [A | B] (the assembled matrix with the right-hand sides as further columns) in the
// CTA's global scratch slot (or A in the caller's LU buffer), then per 16-column panel
//   1. panel   thread t loads row t's 16 entries into registers and keeps them there for the 16
//              elimination steps.  A step: two warp reductions (redux) find the pivot, every
//              warp's candidate publishes its row in shared memory before the one CTA barrier (from
//              eight warps on the pivot's owner alone, behind a second one), and
//              all rows take the rank-1 update from registers and the published row.  Rows are not
//              moved: a logical permutation (s_perm) follows LAPACK's interchanges.  The multipliers
//              go to the shared-memory panel P (physical row order), the U rows to the matrix.
//   2. U12     a chunk of trailing columns, a thread a column: the panel's interchanges, the unit
//              triangle of the panel in 120 multiply-adds from registers, the result to the matrix
//              and to shared memory as the MMA's B operand.
//   3. Schur   16 x 16 warp tiles of the chunk's remaining rows, accumulators loaded from and
//              stored to the matrix in the MMA's fragment layout.
// With the right-hand sides as columns of the trailing matrix the forward substitution is part of
// the factorisation, so L is neither written (unless the caller keeps the factors) nor read again;
// the backward substitution then streams U once.
//
// Rounding: bit-identical to the restated zgetrf / zgetrs.  c - a b is two fused multiply-adds a
// component, first the a.y terms, then the a.x ones.  An m8n8k4 MMA rounds as the four fused
// multiply-adds of its k entries in increasing k, so the chain of a component over increasing k is
// exactly the MMA over the interleaved operands
//     re: a' = (a.y, -a.x) of k, k+1    b' = (b.y, b.x) of k, k+1
//     im: a' = (-a.y, -a.x) of k, k+1   b' = (b.x, b.y) of k, k+1.
//
// What bounds it: the chain of pivot steps (about 1300 cycles a column alone: reduction, reciprocal,
// publishing the row, scaling) at orders up to about 200; above, the same chain and the Schur tiles that come from and
// go to L2 (n = 512, 148 systems: issue slots 24 % busy, FP64 tensor pipe 33 %, L2 hit rate 50 %, stalls shared between
// shared-memory and global loads and barriers).
// Systems an SM, so that one's pivot chain overlaps the others' Schur updates: two up to n = 256 and four up to 128
// by registers (128 a thread, 68 to 84 bytes of spills), five at n = 64 and six up to 60 by shared memory (168
// registers a thread).
// Measured on a B200, whole sweeps, against the kernels that it replaced (whole matrix in shared
// memory, unblocked, up to n of about 112; 16-column panels with register-tiled fused multiply-adds,
// one system an SM, above): n = 64, 500 systems, 318 -> 122 us; n = 189, 1000 systems, 4.9 -> 2.3 ms;
// n = 256, r = 8, 2048 systems, 17.0 -> 9.3 ms.  The whole-matrix kernel stays for the smallest orders and widest
// right-hand sides (fp64_smem_faster in sweep.cu).
#include <algorithm>
#include <climits>

#include "sweep_common.cuh"

namespace srom {
namespace lu64 {

constexpr int NB = 16;  // panel width

// blocks an SM by registers; CW: columns of a chunk
template <int NT_>
struct Cfg;
template <>
struct Cfg<64> {
    static constexpr int CW = 64, BLOCKS = 6;
};
template <>
struct Cfg<128> {
    static constexpr int CW = 64, BLOCKS = 4;
};
template <>
struct Cfg<256> {
    static constexpr int CW = 128, BLOCKS = 2;
};
template <>
struct Cfg<512> {
    static constexpr int CW = 256, BLOCKS = 1;
};

// Leading dimensions that are 4 modulo 8 (in 16-byte entries): the two k rows a fragment load
// touches then fall in different halves of the 32 banks.
__host__ __device__ constexpr int ld4(int n) { return (n + 3) / 8 * 8 + 4; }
// Leading dimension of the scratch matrix: columns start on 128-byte lines.
__host__ __device__ constexpr int lda_of(int n) { return lu64_lda(n); }

template <int NT_>
struct Smem {
    static constexpr int NWT = NT_ / 32;
    static_assert(2 * NWT * (NB + 2) * 16 + 2 * NT_ * 4 + 384 <= NB * ld4(Cfg<NT_>::CW) * 16, "the panel's exchange fits the U region");
    size_t u, p, rows, keys, at, l11, perm, pivlg, dsrc, ddst, total;
    static __host__ __device__ size_t up(size_t b) { return (b + 127) / 128 * 128; }
    __host__ __device__ explicit Smem(int n_max) {
        u = 0;                                                     // NB x ld4(CW): the chunk's U rows,
        rows = 0;                                                  // or, in the panel, published rows,
        keys = rows + up((size_t)2 * NWT * NB * 16);               // candidates, reciprocals
        at = keys + up((size_t)4 * NWT * 16);                      // and the logical order
        p = u + up((size_t)NB * ld4(Cfg<NT_>::CW) * 16);           // NB x ld4(n): multipliers
        l11 = p + up((size_t)NB * ld4(n_max) * 16);                // the panel's unit triangle
        perm = l11 + up((size_t)NB * NB * 16);
        pivlg = perm + up((size_t)n_max * 4);
        dsrc = pivlg + up((size_t)n_max * 4);
        ddst = dsrc + up((size_t)2 * NB * 4);
        total = ddst + up((size_t)2 * NB * 4);
    }
    // the backward substitution's areas in the u and p regions: two diagonal blocks, the divisors
    // and as many right-hand sides as fit
    static constexpr size_t TILES = (size_t)2 * NB * (NB + 1) * 16;
    __host__ __device__ size_t work() const { return l11; }
};

struct Shared {
    int item, info, nmoved;
    int first;
};

__device__ __forceinline__ void dmma(double2 &c, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c.x), "+d"(c.y)
        : "d"(a), "d"(b));
}

__device__ __forceinline__ double neg_if(double v, unsigned sign) {
    return __hiloint2double(__double2hiint(v) ^ (int)sign, __double2loint(v));
}

// 1 / z with crecip's operations: Smith's two cases are one sequence on the larger and the smaller
// component, so that lanes on different cases do not diverge.
__device__ __forceinline__ double2 crecip_uniform(double2 z) {
    const bool xb = fabs(z.x) >= fabs(z.y);
    const double p = xb ? z.x : z.y, q = xb ? z.y : z.x;
    const double t = __ddiv_rn(q, p);
    const double d = __dadd_rn(p, __dmul_rn(q, t));
    const double u = __drcp_rn(d), v = __ddiv_rn(t, d);
    return xb ? make_double2(u, -v) : make_double2(v, -u);
}

// Exchanged through shared memory at the one barrier of a step, two buffers by the step's parity.
template <int NT_>
struct Exchange {
    static constexpr int NWT = NT_ / 32;
    int4 *cand;    // [2][NWT]: key (low, high word), physical row, 1 if the warp saw a NaN
    double2 *inv;  // [2][NWT]: reciprocal of the candidate
    double2 *rows; // [2][NWT][NB]: the candidate's row
    int *at;       // at[logical row] = physical row, of the rows that are not yet pivots
    int *lg;       // its inverse: lg[physical row]
};

// Elimination steps [jj0, jj1) of the panel at j0; a[0] holds this thread's row's entry of column jj,
// a[c] of column jj + c (c < W): every update also shifts the row by one column, so the loop body is
// the same code for every step.
//
// A step is one dependent chain (find the pivot, invert it, scale, update the next column), and the
// code is laid out to keep that short: no divergent branch on the common path, the search on one
// 64-bit key a row (value bits + 1; 0 for none) with ties and NaNs in a path of their own, and the
// reciprocal, the longest part, computed by every lane for its own entry before the barrier, where the
// reduction and the previous step's update of the columns past the next one run in its shadow.
// Warps without a row of the panel (tid >= m) only follow the pivots: with several systems an SM the steps are
// bound by instruction issue, and most panels are shorter than the thread count: 1000 systems of order 189 went
// from 2.30 to 2.21 ms with it, of order 150 from 1.49 to 1.40 ms.
template <int NT_, int W>
__device__ __forceinline__ void panel_steps(double2 (&a)[NB], int jj0, int jj1, int nbc, int j0, double2 *A,
                                            int64_t lda, double2 *P, int ldp, const Exchange<NT_> &X, int *s_pivlg,
                                            int *s_perm, Shared &S, int m, bool &done) {
    constexpr int NWT = NT_ / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // LATE: the pivot's row is published by its owner, behind a second barrier, instead of every warp's
    // candidate's before the first.  A lane's 16-byte stores take the shared-memory datapath as long as a whole
    // warp's (16 cycles each): with eight warps or more they cost more than the barrier (order 189: 2.21 -> 2.18 ms,
    // 256 with r = 8: 2.67 -> 2.63 ms a 592 systems).
    constexpr bool LATE = NWT >= 8;
    const bool live = warp * 32 < m;
    double2 lp = make_double2(0.0, 0.0);
    const double2 *up = nullptr;  // the previous step's pivot row
    for (int jj = jj0; jj < jj1; ++jj) {
        const int buf = jj & 1;
        int4 *cand = X.cand + buf * NWT;
        double2 *inv = X.inv + buf * NWT;
        double2 *rw = X.rows + (size_t)buf * NWT * NB;
        auto store_row = [&](int w) {
#pragma unroll
            for (int c = 0; c < W; ++c) rw[w * NB + c] = a[c];
        };
        bool nan = false;
        unsigned long long key = 0;
        unsigned hi = 0, lo = 0, bh = 0;
        double2 rec = make_double2(0.0, 0.0);
        if (live) {
            const double v = cabs1(a[0]);
            nan = !done && v != v;
            key = done || v != v ? 0 : (unsigned long long)__double_as_longlong(v) + 1;
            hi = (unsigned)(key >> 32);
            lo = (unsigned)key;
            bh = __reduce_max_sync(FULL_MASK, hi);
            rec = crecip_uniform(key ? a[0] : make_double2(1.0, 0.5));  // off the zero operands' path
            if (jj > jj0) {
#pragma unroll
                for (int c = 1; c + 1 < W; ++c) a[c] = csubmul(a[c + 1], lp, up[c + 1]);
            }
            const unsigned who = __ballot_sync(FULL_MASK, key != 0 && hi == bh);
            // flag: a NaN, or rows of equal value (high words compared), for the path below to sort out
            const int odd = __any_sync(FULL_MASK, nan) || (who & (who - 1));
            if (lane == (who ? __ffs(who) - 1 : 0)) {
                cand[warp] = make_int4((int)lo, (int)hi, tid, odd);
                if constexpr (!LATE) {
                    inv[warp] = rec;
                    store_row(warp);
                }
            }
        }
        __syncthreads();
        unsigned long long bkey;
        int bph;
        bool slow;
        auto key_of = [](const int4 &c) { return ((unsigned long long)(unsigned)c.y << 32) | (unsigned)c.x; };
        if constexpr (NWT <= 4) {
            const int4 c = cand[0];
            bkey = key_of(c);
            bph = c.z;
            slow = c.w;
#pragma unroll
            for (int i = 1; i < NWT; ++i) {
                const int4 d = cand[i];
                const unsigned long long k = key_of(d);
                slow = slow || d.w || (k == bkey && k != 0);
                bph = k > bkey ? d.z : bph;
                bkey = k > bkey ? k : bkey;
            }
        } else {
            const int4 c = lane < NWT ? cand[lane] : make_int4(0, 0, 0, 0);
            const unsigned mh = __reduce_max_sync(FULL_MASK, (unsigned)c.y);
            const unsigned w = __ballot_sync(FULL_MASK, (unsigned)c.y == mh && (c.x | c.y) != 0);
            slow = __any_sync(FULL_MASK, c.w) || (w & (w - 1));
            const int src = w ? __ffs(w) - 1 : 0;
            bph = __shfl_sync(FULL_MASK, c.z, src);
            bkey = ((unsigned long long)mh << 32) | (unsigned)__shfl_sync(FULL_MASK, c.x, src);
        }
        bool nz = true;
        int wl = bph >> 5;
        if (slow || bkey <= 1) {
            // The full rule.  IZAMAX takes the smallest logical row of the largest value and starts from
            // the first entry: a NaN there is the pivot, all-NaN likewise; LAPACK interchanges nothing
            // for a zero pivot (the row at logical position jj is then the pivot).
            if (tid == 0) S.first = 0;
            __syncthreads();
            const int first = X.at[jj];
            if (tid == first && nan) S.first = 1;
            const unsigned bl = __reduce_max_sync(FULL_MASK, hi == bh ? lo : 0u);
            const int lg = key != 0 && hi == bh && lo == bl ? X.lg[tid] : INT_MAX;
            const int low = __reduce_min_sync(FULL_MASK, lg);
            if (low == INT_MAX ? lane == 0 : lg == low) {
                cand[warp] = make_int4((int)lo, (int)hi, tid, 0);
                inv[warp] = rec;
                store_row(warp);
            }
            __syncthreads();
            bkey = 0;
            bph = first;
            for (int i = 0; i < NWT; ++i) {
                const unsigned long long k = key_of(cand[i]);
                const int ph = cand[i].z;
                if (k > bkey || (k == bkey && k != 0 && X.lg[ph] < X.lg[bph])) {
                    bkey = k;
                    bph = ph;
                }
            }
            wl = bph >> 5;
            if (S.first || bkey <= 1) {
                bph = first;
                wl = 0;
                __syncthreads();
                if (tid == first) {
                    inv[0] = crecip_uniform(a[0]);
                    store_row(0);
                }
            }
            __syncthreads();
            nz = rw[wl * NB].x != 0.0 || rw[wl * NB].y != 0.0;
        } else if constexpr (LATE) {
            wl = 0;
            if (tid == bph) {
                inv[0] = rec;
                store_row(0);
            }
            __syncthreads();
        }
        const double2 *pr = rw + wl * NB;
        if (live) {
            lp = nz ? cmul(a[0], inv[wl]) : a[0];
            a[0] = csubmul(a[1], lp, pr[1]);
            done = done || tid == bph;
            if (!done) P[tid + jj * ldp] = lp;
            up = pr;
        }
        if (warp == (m < NT_ - 31 ? NWT - 1 : (wl + 1) % NWT)) {  // a warp without rows, if there is one
            if (lane < nbc - jj) A[(j0 + jj) + (int64_t)(j0 + jj + lane) * lda] = pr[lane];
            if (lane == 0) {
                // the interchange of logical rows jj and lg[bph]
                const int first = X.at[jj], lgp = X.lg[bph];
                X.at[lgp] = first;
                X.lg[first] = lgp;
                s_perm[jj] = bph;
                s_pivlg[j0 + jj] = lgp;
                if (!nz && S.info == 0) S.info = j0 + jj + 1;
            }
        }
    }
    if (live && jj1 > jj0) {
#pragma unroll
        for (int c = 1; c + 1 < W; ++c) a[c] = csubmul(a[c + 1], lp, up[c + 1]);
    }
}

// Column c of [A | B]: columns of B (ld ldb) follow the n columns of A.
__device__ __forceinline__ double2 *col_ptr(double2 *A, int64_t lda, double2 *B, int64_t ldb, int n, int c) {
    return c < n ? A + (int64_t)c * lda : B + (int64_t)(c - n) * ldb;
}

template <int NT_>
__device__ __forceinline__ void factor(double2 *A, int64_t lda, double2 *B, int64_t ldb, int n, int r, bool keep_l,
                                       unsigned char *sm, const Smem<NT_> &L, int ldp, Shared &S) {
    constexpr int NWT = NT_ / 32, CW = Cfg<NT_>::CW, LDU = ld4(CW);
    double2 *U = reinterpret_cast<double2 *>(sm + L.u);
    double2 *P = reinterpret_cast<double2 *>(sm + L.p);
    const Exchange<NT_> X{reinterpret_cast<int4 *>(sm + L.keys), reinterpret_cast<double2 *>(sm + L.keys) + 2 * NWT,
                          reinterpret_cast<double2 *>(sm + L.rows), reinterpret_cast<int *>(sm + L.at),
                          reinterpret_cast<int *>(sm + L.at) + NT_};
    double2 *l11 = reinterpret_cast<double2 *>(sm + L.l11);
    int *s_perm = reinterpret_cast<int *>(sm + L.perm);
    int *s_pivlg = reinterpret_cast<int *>(sm + L.pivlg);
    int *s_dsrc = reinterpret_cast<int *>(sm + L.dsrc);
    int *s_ddst = reinterpret_cast<int *>(sm + L.ddst);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ncols = n + r;
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int nbc = min(NB, n - j0), m = n - j0;
        // ---- panel
        {
            double2 a[NB];
#pragma unroll
            for (int c = 0; c < NB; ++c)
                a[c] = (tid < m && c < nbc) ? A[(j0 + tid) + (int64_t)(j0 + c) * lda] : make_double2(0.0, 0.0);
            bool done = tid >= m;
            if (tid == 0) S.nmoved = 0;
            if (tid < m) {
                X.at[tid] = tid;
                X.lg[tid] = tid;
            }
            if (warp * 32 >= m && lane == 0) X.cand[warp] = X.cand[NWT + warp] = make_int4(0, 0, tid, 0);
            panel_steps<NT_, 16>(a, 0, min(4, nbc), nbc, j0, A, lda, P, ldp, X, s_pivlg, s_perm, S, m, done);
            panel_steps<NT_, 12>(a, 4, min(8, nbc), nbc, j0, A, lda, P, ldp, X, s_pivlg, s_perm, S, m, done);
            panel_steps<NT_, 8>(a, 8, min(12, nbc), nbc, j0, A, lda, P, ldp, X, s_pivlg, s_perm, S, m, done);
            panel_steps<NT_, 4>(a, 12, nbc, nbc, j0, A, lda, P, ldp, X, s_pivlg, s_perm, S, m, done);
        }
        __syncthreads();
        if (tid < m) {
            // the composite permutation: pivot rows, then the others in their logical places; a row that
            // left its place went to a pivot position or was displaced from one
            const int ph = tid < nbc ? s_perm[tid] : X.at[tid];
            s_perm[tid] = ph;
            if (ph != tid) {
                const int e = atomicAdd(&S.nmoved, 1);
                s_ddst[e] = tid;
                s_dsrc[e] = ph;
            }
        }
        __syncthreads();
        const int nmoved = S.nmoved;
        for (int e = tid; e < NB * NB; e += NT_) {
            const int i = e % NB, k = e / NB;
            l11[e] = (i > k && i < nbc) ? P[s_perm[i] + k * ldp] : make_double2(0.0, 0.0);
        }
        if (keep_l) {
            // the multipliers in logical row order, and LAPACK's interchanges on the columns left of
            // the panel (a warp a column; at most 32 rows move)
            for (int c = warp; c < nbc; c += NWT)
                for (int i = c + 1 + lane; i < m; i += 32) A[(j0 + i) + (int64_t)(j0 + c) * lda] = P[s_perm[i] + c * ldp];
            for (int c = warp; c < j0; c += NWT) {
                double2 *col = A + (int64_t)c * lda + j0;
                double2 v = make_double2(0.0, 0.0);
                if (lane < nmoved) v = col[s_dsrc[lane]];
                __syncwarp();
                if (lane < nmoved) col[s_ddst[lane]] = v;
            }
        }
        const int mt = m - NB;  // rows below the panel (when the panel is full)
        // A chunk's U rows between shared memory and the matrix: 16 lanes a column, so that the rows of
        // a column are one access.  They are stored only after the chunk's Schur update, which still
        // reads the rows that the interchanges displace from there.
        const int ui = lane & 15, uc = warp * 2 + (lane >> 4);
        auto fetch = [&](int c0, int nc) {
            if (ui < nbc)
                for (int c = uc; c < nc; c += 2 * NWT)
                    cp_async_elem(U + ui * LDU + c, col_ptr(A, lda, B, ldb, n, c0 + c) + j0 + s_perm[ui]);
            cp_async_commit();
        };
        auto flush = [&](int c0, int nc) {
            if (ui < nbc)
                for (int c = uc; c < nc; c += 2 * NWT) col_ptr(A, lda, B, ldb, n, c0 + c)[j0 + ui] = U[ui * LDU + c];
        };
        // chunks of nearly equal width, a multiple of 16 and at most CW
        const int left = ncols - (j0 + nbc);
        const int nchunk = (left + CW - 1) / CW;
        const int cw = ((left + nchunk - 1) / nchunk + 15) / 16 * 16;
        int c0 = j0 + nbc;
        for (; c0 < ncols; c0 += cw) {
            const int nc = min(cw, ncols - c0);
            __syncthreads();  // the panel's triangle; the previous chunk's Schur update
            // ---- U12 of the chunk, a thread a column
            if (c0 > j0 + nbc) {
                flush(c0 - cw, cw);
                __syncthreads();
            }
            fetch(c0, nc);
            cp_async_wait<0>();
            __syncthreads();
            if (tid < nc) {
                double2 x[NB];
#pragma unroll
                for (int i = 0; i < NB; ++i) x[i] = i < nbc ? U[i * LDU + tid] : make_double2(0.0, 0.0);
#pragma unroll
                for (int k = 0; k < NB - 1; ++k)
#pragma unroll
                    for (int i = k + 1; i < NB; ++i) x[i] = csubmul(x[i], l11[k * NB + i], x[k]);
#pragma unroll
                for (int i = 0; i < NB; ++i) U[i * LDU + tid] = x[i];
            }
            __syncthreads();
            // ---- Schur update of rows [16, m) of the chunk: a warp takes a strip of 16 columns (or a
            // segment of its rows, so that every warp has as many tiles) tile by tile, 16 x 16, the next
            // tile's entries loaded while this one's MMAs run.  A tile's rows are read from their
            // physical places and written to their logical ones.
            if (mt <= 0) continue;
            const int nrt = (mt + 15) / 16, nstrip = (nc + 15) / 16;
            int nseg = NWT;
            while (nseg > 1 && (nstrip * (nseg / 2)) % NWT == 0) nseg /= 2;
            const int lr = lane >> 2, lk = (lane >> 1) & 1;
            const bool odd = lane & 1;
            const unsigned sgn_re = odd ? 0x80000000u : 0u;
            for (int task = warp; task < nstrip * nseg; task += NWT) {
                const int strip = task / nseg, seg = task - strip * nseg;
                const int t0 = nrt * seg / nseg, t1 = nrt * (seg + 1) / nseg;
                if (t0 >= t1) continue;
                double2 *cp[4];
                bool okc[4];
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    const int cc = strip * 16 + 8 * (z >> 1) + 2 * (lane & 3) + (z & 1);
                    okc[z] = cc < nc;
                    cp[z] = col_ptr(A, lda, B, ldb, n, c0 + min(cc, nc - 1)) + j0;
                }
                const double2 *pb = U + lk * LDU + strip * 16 + lr, *pp = P + lk * ldp;
                double2 nx[2][4];
                int nph[2];
                auto load = [&](int t) {
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        nph[x] = s_perm[NB + min(t * 16 + 8 * x + lr, mt - 1)];
#pragma unroll
                        for (int z = 0; z < 4; ++z) nx[x][z] = cp[z][nph[x]];
                    }
                };
                load(t0);
                for (int t = t0; t < t1; ++t) {
                    double2 re[2][2], im[2][2];  // [row tile][column tile]: components of the two columns
                    const double2 *pa[2];
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        pa[x] = pp + nph[x];
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            re[x][y] = make_double2(nx[x][2 * y].x, nx[x][2 * y + 1].x);
                            im[x][y] = make_double2(nx[x][2 * y].y, nx[x][2 * y + 1].y);
                        }
                    }
                    if (t + 1 < t1) load(t + 1);
#pragma unroll
                    for (int k = 0; k < NB; k += 2) {
                        double are[2], aim[2], bre[2], bim[2];
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const double2 v = pa[x][k * ldp];
                            const double w = odd ? v.x : v.y;
                            are[x] = neg_if(w, sgn_re);
                            aim[x] = neg_if(w, 0x80000000u);
                        }
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            const double2 v = pb[k * LDU + 8 * y];
                            bre[y] = odd ? v.x : v.y;
                            bim[y] = odd ? v.y : v.x;
                        }
#pragma unroll
                        for (int x = 0; x < 2; ++x)
#pragma unroll
                            for (int y = 0; y < 2; ++y) {
                                dmma(re[x][y], are[x], bre[y]);
                                dmma(im[x][y], aim[x], bim[y]);
                            }
                    }
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const int row = t * 16 + 8 * x + lr;
                        if (row < mt) {
#pragma unroll
                            for (int y = 0; y < 2; ++y) {
                                if (okc[2 * y]) cp[2 * y][NB + row] = make_double2(re[x][y].x, im[x][y].x);
                                if (okc[2 * y + 1]) cp[2 * y + 1][NB + row] = make_double2(re[x][y].y, im[x][y].y);
                            }
                        }
                    }
                }
            }
        }
        __syncthreads();
        flush(c0 - cw, ncols - (c0 - cw));
        __syncthreads();
    }
}

// The parts of Smith's division by a diagonal entry that do not depend on the dividend: t, d and
// 1 / d; big: |re| >= |im|.  ok: d lies where quotient() may use 1 / d
struct Divisor {
    double t, d, rd;
    int big, ok;
};
__device__ __forceinline__ bool mid_range(double v) {  // |v| in about [2^-400, 2^400]
    return ((((unsigned)__double2hiint(v) >> 20) & 0x7ffu) - 623u) < 800u;
}
__device__ __forceinline__ Divisor divisor_of(double2 b) {
    Divisor D;
    D.big = fabs(b.x) >= fabs(b.y);
    const double p = D.big ? b.x : b.y, q = D.big ? b.y : b.x;
    D.t = __ddiv_rn(q, p);
    D.d = __dadd_rn(p, __dmul_rn(q, D.t));
    D.rd = __drcp_rn(D.d);
    D.ok = mid_range(D.d);
    return D;
}
// v / diagonal entry by Smith's method; both divisions by d correctly rounded from rd = 1 / d correctly rounded: a quotient within one unit in the last
// place, then Markstein's theorem (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", 1990): with r = n - q d (exact in one fused multiply-add), q + r rd
// rounds to n / d.  Operands outside the middle of the exponent range take the division itself.
__device__ __forceinline__ double2 quotient(double2 v, const Divisor &D) {
    const double p = D.big ? v.x : v.y, q = D.big ? v.y : v.x;
    const double re = __dadd_rn(p, __dmul_rn(q, D.t));
    double im = __dsub_rn(q, __dmul_rn(p, D.t));
    im = D.big ? im : -im;
    double qr = __dmul_rn(re, D.rd), qi = __dmul_rn(im, D.rd);
    qr = __fma_rn(__fma_rn(-qr, D.d, re), D.rd, qr);
    qi = __fma_rn(__fma_rn(-qi, D.d, im), D.rd, qi);
    qr = __fma_rn(__fma_rn(-qr, D.d, re), D.rd, qr);
    qi = __fma_rn(__fma_rn(-qi, D.d, im), D.rd, qi);
    if (!(D.ok && mid_range(re) && mid_range(im))) {
        qr = __ddiv_rn(re, D.d);
        qi = __ddiv_rn(im, D.d);
    }
    return make_double2(qr, qi);
}

// x = U^-1 y for nr right-hand sides (Bs: shared memory, n x nr, ld n), U in A.  Blocks of 16 rows
// from the last: the triangle by one warp a right-hand side, then a thread a row takes the block's
// columns in decreasing order (the oracle's), its 16 entries of U loaded ahead of the triangle; with
// several right-hand sides the rows are updated by MMAs over the same order.
// tile: two buffers of NB x (NB + 1), the next block's diagonal block copied in while this one is
// solved.  A division is on the path of every row: its divisor's parts are prepared for all rows at
// once (dv), which leaves five dependent multiply-adds.
template <int NT_, bool MMA>
__device__ __forceinline__ void back_substitute(const double2 *A, int64_t lda, int n, double2 *Bs, int nr, double2 *tile,
                                                const Divisor *dv) {
    constexpr int NWT = NT_ / 32, LDT = NB + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int last = (n - 1) / NB * NB;
    auto fetch = [&](int jb) {
        if (jb >= 0) {
            double2 *t = tile + ((jb / NB) & 1) * NB * LDT;
            for (int e = tid; e < NB * NB; e += NT_) {
                const int i = e % NB, j = e / NB;
                if (i < j && jb + j < n) cp_async_elem(t + i + j * LDT, A + (jb + i) + (int64_t)(jb + j) * lda);
            }
        }
        cp_async_commit();
    };
    fetch(last);
    for (int jb = last; jb >= 0; jb -= NB) {
        const int bs = min(NB, n - jb);
        double2 u[NB];
        if constexpr (!MMA) {
#pragma unroll
            for (int j = 0; j < NB; ++j)
                u[j] = (tid < jb && j < bs) ? A[tid + (int64_t)(jb + j) * lda] : make_double2(0.0, 0.0);
        }
        fetch(jb - NB);
        cp_async_wait<1>();
        __syncthreads();
        const double2 *tl = tile + ((jb / NB) & 1) * NB * LDT;
        for (int c = warp; c < nr; c += NWT) {
            double2 *b = Bs + (int64_t)c * n + jb;
            double2 v = lane < bs ? b[lane] : make_double2(0.0, 0.0);
            const Divisor D = dv[jb + min(lane, bs - 1)];
            double2 nt = tl[lane % NB + (bs - 1) * LDT];
            for (int j = bs - 1; j >= 0; --j) {
                const double2 ut = nt;
                if (j > 0) nt = tl[lane % NB + (j - 1) * LDT];
                if (lane == j) v = quotient(v, D);
                const double2 bj = CT<double2>::shfl(v, j, 32);
                if (lane < j) v = csubmul(v, ut, bj);
            }
            if (lane < bs) b[lane] = v;
        }
        __syncthreads();
        if constexpr (MMA) {
          if (bs == NB) {
            // 8 rows x 8 right-hand sides a warp tile, k running down from the block's last column
            const int lr = lane >> 2, lk = (lane >> 1) & 1;
            const bool odd = lane & 1;
            const unsigned sgn_re = odd ? 0x80000000u : 0u;
            const int nrt = (jb + 7) / 8, nct = (nr + 7) / 8;
            for (int t = warp; t < nrt * nct; t += NWT) {
                const int row = (t % nrt) * 8 + lr, cc = t / nrt * 8;
                double2 re, im, *cp[2], *pb = Bs + (int64_t)min(cc + lr, nr - 1) * n + jb + (NB - 1) - lk;
                const double2 *pa = A + min(row, jb - 1) + (int64_t)(jb + NB - 1 - lk) * lda;
                double2 av[NB / 2];
#pragma unroll
                for (int k = 0; k < NB / 2; ++k) av[k] = pa[-(int64_t)(2 * k) * lda];
#pragma unroll
                for (int h = 0; h < 2; ++h) cp[h] = Bs + (int64_t)min(cc + 2 * (lane & 3) + h, nr - 1) * n + min(row, jb - 1);
                re = make_double2(cp[0]->x, cp[1]->x);
                im = make_double2(cp[0]->y, cp[1]->y);
#pragma unroll
                for (int k = 0; k < NB / 2; ++k) {
                    const double2 b = pb[-2 * k];
                    const double w = odd ? av[k].x : av[k].y;
                    dmma(re, neg_if(w, sgn_re), odd ? b.x : b.y);
                    dmma(im, neg_if(w, 0x80000000u), odd ? b.y : b.x);
                }
                if (row < jb) {
                    if (cc + 2 * (lane & 3) < nr) *cp[0] = make_double2(re.x, im.x);
                    if (cc + 2 * (lane & 3) + 1 < nr) *cp[1] = make_double2(re.y, im.y);
                }
            }
          } else {
            for (int e = tid; e < jb * nr; e += NT_) {
                double2 *b = Bs + (int64_t)(e / jb) * n;
                double2 acc = b[e % jb];
                for (int j = bs - 1; j >= 0; --j) acc = csubmul(acc, A[e % jb + (int64_t)(jb + j) * lda], b[jb + j]);
                b[e % jb] = acc;
            }
          }
        } else if (tid < jb) {
            for (int c = 0; c < nr; ++c) {
                double2 *b = Bs + (int64_t)c * n;
                double2 acc = b[tid];
#pragma unroll
                for (int j = NB - 1; j >= 0; --j)
                    if (j < bs) acc = csubmul(acc, u[j], b[jb + j]);
                b[tid] = acc;
            }
        }
        // the next block's barrier orders these rows before their readers
    }
    cp_async_wait<0>();
    __syncthreads();
}

// A(w) into A and the right-hand sides into B.
template <int NT_>
__device__ __forceinline__ void assemble(const RomDev &R, int f, double2 *__restrict__ A, int64_t lda,
                                      double2 *__restrict__ B, int64_t ldb) {
    const int tid = threadIdx.x, n = R.n, r = R.r;
    const double2 *K = R.K, *M = R.M, *D = R.D, *rhs = R.rhs;
    const int64_t ldk = R.ldk, ldr = R.ldb;
    const double w = R.omega[f], s = -__dmul_rn(w, w), eta = R.eta;
    const uint64_t pol = l2_keep_policy();
    constexpr int NWT = NT_ / 32;
    const int lane = tid & 31, jfirst = sweep_start(f, n);
    if constexpr (NT_ > 64) {
        // a warp a column, from column sweep_start(f) on
        for (int jj = tid >> 5; jj < n; jj += NWT) {
            const int j = jj + jfirst < n ? jj + jfirst : jj + jfirst - n;
#pragma unroll 4
            for (int i = lane; i < n; i += 32) {
                const int64_t e = i + (int64_t)j * ldk;
                A[i + j * lda] = assemble_entry(ld_keep(K + e, pol), ld_keep(M + e, pol), D, e, eta, s, w);
            }
        }
    } else {
        // a column is one or two pieces of 32 rows: a warp takes every second piece, UN of them in flight
        constexpr int UN = 4;
        const int nch = (n + 31) / 32, dj = NWT / nch, dch = NWT % nch;
        int j = (tid >> 5) / nch, ch = (tid >> 5) % nch;
        while (j < n) {
            double2 k[UN], m[UN];
            int ii[UN], jj[UN];  // row (n or more: none) and column
#pragma unroll
            for (int q = 0; q < UN; ++q) {
                const int i = ch * 32 + lane, jw = j + jfirst < n ? j + jfirst : j + jfirst - n;
                ii[q] = j < n ? i : n;
                jj[q] = jw;
                if (ii[q] < n) {
                    k[q] = ld_keep(K + i + (int64_t)jw * ldk, pol);
                    m[q] = ld_keep(M + i + (int64_t)jw * ldk, pol);
                }
                j += dj;
                ch += dch;
                if (ch >= nch) {
                    ch -= nch;
                    ++j;
                }
            }
#pragma unroll
            for (int q = 0; q < UN; ++q)
                if (ii[q] < n)
                    A[ii[q] + (int64_t)jj[q] * lda] = assemble_entry(k[q], m[q], D, ii[q] + (int64_t)jj[q] * ldk, eta, s, w);
        }
    }
    for (int c = tid >> 5; c < r; c += NT_ / 32)
        for (int q = tid & 31; q < n; q += 32) B[q + c * ldb] = rhs[q + (int64_t)c * ldr];
}

template <int NT_>
__global__ void __launch_bounds__(NT_, Cfg<NT_>::BLOCKS) sweep_lu64_kernel(GlobalArgs a) {
    constexpr int NWT = NT_ / 32;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ Shared S;
    const Smem<NT_> L(a.n_max);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ldp = ld4(a.n_max);
    const int n_items = a.n_items_dev ? *a.n_items_dev : a.n_items;
    unsigned char *slot = a.scratch + (int64_t)blockIdx.x * a.slot_bytes;
    for (;;) {
        if (tid == 0) S.item = atomicAdd(a.counter, 1);
        __syncthreads();
        const int it = S.item;
        __syncthreads();
        if (it >= n_items) break;
        const Item wi = a.items[it];
        const RomDev &R = a.roms[wi.rom];
        const int n = R.n, r = R.r;
        const int64_t lds = lda_of(n);
        double2 *Bg = reinterpret_cast<double2 *>(slot);  // n x r, ld lds, then the matrix
        double2 *A = R.LU ? R.LU + (int64_t)wi.f * n * n : Bg + lds * r;
        const int64_t lda = R.LU ? n : lds;
        assemble<NT_>(R, wi.f, A, lda, Bg, lds);
        if (tid == 0) S.info = 0;
        __syncthreads();
        factor<NT_>(A, lda, Bg, lds, n, r, R.LU != nullptr, sm, L, ldp, S);
        // ---- backward substitution, as many right-hand sides at a time as shared memory holds
        double2 *tile = reinterpret_cast<double2 *>(sm + L.u);
        Divisor *dv = reinterpret_cast<Divisor *>(sm + L.u + L.TILES);
        double2 *Bs = reinterpret_cast<double2 *>(sm + L.u + L.TILES + (size_t)n * sizeof(Divisor));
        const int cap = max(1, (int)((L.work() - L.TILES - (size_t)n * sizeof(Divisor)) / ((size_t)n * 16)));
        if (tid < n) dv[tid] = divisor_of(A[tid + (int64_t)tid * lda]);
        for (int c0 = 0; c0 < r; c0 += cap) {
            const int nr = min(cap, r - c0);
            for (int c = warp; c < nr; c += NWT)
                for (int i = lane; i < n; i += 32) Bs[i + (int64_t)c * n] = Bg[i + (int64_t)(c0 + c) * lds];
            __syncthreads();
            // the row update on the MMA from three right-hand sides on (its tile holds eight)
            if (nr >= 3) back_substitute<NT_, true>(A, lda, n, Bs, nr, tile, dv);
            else back_substitute<NT_, false>(A, lda, n, Bs, nr, tile, dv);
            double2 *X = R.X + ((int64_t)wi.f * r + c0) * n;
            for (int e = tid; e < n * nr; e += NT_) X[e] = Bs[e];
            __syncthreads();
        }
        if (R.ipiv) {
            const int *pl = reinterpret_cast<const int *>(sm + L.pivlg);
            if (tid < n) R.ipiv[(int64_t)wi.f * n + tid] = tid / NB * NB + pl[tid] + 1;
        }
        if (tid == 0) {
            if (R.info) R.info[wi.f] = S.info;
            if (R.steps) R.steps[wi.f] = a.steps_value;
            if (R.berr) R.berr[wi.f] = 0.0;
        }
        __syncthreads();
    }
}

template <int NT_>
static cudaError_t launch(const GlobalArgs &a, int grid, cudaStream_t st) {
    auto k = sweep_lu64_kernel<NT_>;
    const size_t smem = Smem<NT_>(a.n_max).total;
    // one value for all sizes: another thread's smaller launch must not lower it between this call and this launch
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Smem<NT_>(NT_).total);
    if (e != cudaSuccess) return e;
    k<<<grid, NT_, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace lu64

template <int NT_>
static int blocks_per_sm(int n_max) {
    const size_t smem = lu64::Smem<NT_>(n_max).total + sizeof(lu64::Shared) + 1024;
    return std::max(1, std::min(lu64::Cfg<NT_>::BLOCKS, (int)((size_t)228 * 1024 / smem)));
}

int lu64_blocks_per_sm(int threads, int n_max) {
    switch (threads) {
        case 64: return blocks_per_sm<64>(n_max);
        case 128: return blocks_per_sm<128>(n_max);
        case 256: return blocks_per_sm<256>(n_max);
        default: return blocks_per_sm<512>(n_max);
    }
}

cudaError_t launch_lu64(int threads, const GlobalArgs &a, int grid, cudaStream_t st) {
    if (a.n_max > threads) return cudaErrorInvalidValue;
    switch (threads) {
        case 64: return lu64::launch<64>(a, grid, st);
        case 128: return lu64::launch<128>(a, grid, st);
        case 256: return lu64::launch<256>(a, grid, st);
        case 512: return lu64::launch<512>(a, grid, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace srom
