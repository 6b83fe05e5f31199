// FP64 sweep of large orders (513 to 2560): several multiprocessors a system.
//
// The systems of a group (at most one a multiprocessor's worth of scratch) advance together, panel by
// panel, with three launches a 32-column panel:
//   panel   a cluster of up to eight CTAs a system, a thread a row (320 rows a CTA): the row's 32 entries
//           stay in registers, every warp publishes its pivot candidate in its CTA's shared memory, one
//           cluster barrier a column, and all threads read the winner's row from its CTA (distributed
//           shared memory).  Rows are not moved; the logical order is kept in shared memory.
//   U12     a CTA a chunk of 64 trailing columns of [A | B]: the panel's interchanges and
//           U12 = L11^-1 x, a thread a column;
//   Schur   a CTA a tile of 128 rows and 64 columns on the FP64 tensor cores.  (One launch for U12 and
//           Schur, a CTA a chunk with all its rows, was a quarter slower: too few CTAs of equal length.)
// The right-hand sides are columns of the trailing matrix, so only the backward substitution follows
// (one CTA a system).  Arithmetic and order of updates are those of sweep_lu64.cu, bit-identical to the
// restated zgetrf / zgetrs.
//
// What bounds it: the FP64 rate in the update (a panel reads and writes the trailing matrix once: 4.9 ps
// an entry at the copy bandwidth against 7.1 for its 32 multiply-adds; with 16 columns a panel it was the
// bandwidth, and the update took half as long again), and with few systems the chain of pivot columns.  One CTA a system, as before, left a sweep of fewer
// frequencies than multiprocessors idle on the others and took one system's whole time at least.
// n = 2520, 12 frequencies, one right-hand side (B200): 748 ms with one CTA a system, 32 ms now.
#include <algorithm>
#include <climits>

#include "sweep_common.cuh"

namespace srom {
namespace large {

constexpr int NB = 32;        // panel width
constexpr int HB = 16;        // rows of a backward block; half a panel's triangle
constexpr int PT = 320;       // threads (rows) of a panel CTA
constexpr int PW = PT / 32;
constexpr int VT = 128;       // threads of a U12 CTA
constexpr int UT = 256;       // threads of a Schur CTA
constexpr int UW = UT / 32;
constexpr int CW = 64;        // columns of a U12 chunk and of a Schur tile
constexpr int RT = 128;       // rows of a Schur tile
constexpr int LDU = CW + 4, LDP = RT + 4;  // 4 modulo 8: see sweep_lu64.cu
constexpr int BT = 512;       // threads of a backward substitution CTA

__host__ __device__ constexpr int lda_of(int n) { return (n + 7) / 8 * 8; }

// A system's slot: B (n x r, ld lda_of(n)), the matrix (unless the caller keeps the factors), the panel's
// multipliers in logical row order (NB columns of ld lda_of(n)), its unit triangle and its bookkeeping.
struct State {
    int info, nmoved;
    int piv[NB];       // physical rows of the pivots
    int dsrc[NB], ddst[NB];  // rows displaced from the panel's top: from, to (nmoved of them)
};
struct Slot {
    size_t mat, p, l11, state, pivlg, total;
    __host__ __device__ Slot(int n_max, int r_max) {
        auto up = [](size_t b) { return (b + 255) / 256 * 256; };
        const size_t ld = lda_of(n_max);
        mat = up(ld * r_max * 16);
        p = mat + up(ld * n_max * 16);
        l11 = p + up((size_t)NB * ld * 16);
        state = l11 + up((size_t)NB * NB * 16);
        pivlg = state + up(sizeof(State));
        total = pivlg + up((size_t)n_max * 4);
    }
};

struct Args {
    const RomDev *roms;
    const Item *items;
    unsigned char *scratch;
    int64_t slot_bytes;
    int n_max, r_max;
};

// One system as the kernels address it.
struct Sys {
    RomDev R;
    int f, n, r;
    double2 *A, *B, *P, *l11;
    int64_t lda, ldb;
    State *st;
    int *pivlg;
};
__device__ __forceinline__ Sys system_of(const Args &a, int i) {
    Sys s;
    const Item wi = a.items[i];
    s.R = a.roms[wi.rom];
    s.f = wi.f;
    s.n = s.R.n;
    s.r = s.R.r;
    const Slot L(a.n_max, a.r_max);
    unsigned char *p = a.scratch + (int64_t)i * a.slot_bytes;
    s.ldb = lda_of(s.n);
    s.B = reinterpret_cast<double2 *>(p);
    s.A = s.R.LU ? s.R.LU + (int64_t)s.f * s.n * s.n : reinterpret_cast<double2 *>(p + L.mat);
    s.lda = s.R.LU ? s.n : s.ldb;
    s.P = reinterpret_cast<double2 *>(p + L.p);
    s.l11 = reinterpret_cast<double2 *>(p + L.l11);
    s.st = reinterpret_cast<State *>(p + L.state);
    s.pivlg = reinterpret_cast<int *>(p + L.pivlg);
    return s;
}
__device__ __forceinline__ double2 *col_ptr(const Sys &s, int c) {
    return c < s.n ? s.A + (int64_t)c * s.lda : s.B + (int64_t)(c - s.n) * s.ldb;
}

// ---------------------------------------------------------------------------- assembly
__global__ void __launch_bounds__(256) large_assemble_kernel(Args a) {
    const Sys s = system_of(a, blockIdx.y);
    const int lane = threadIdx.x & 31;
    const double w = s.R.omega[s.f], m2 = -__dmul_rn(w, w);
    const uint64_t pol = l2_keep_policy();
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < s.n + s.r; c += (gridDim.x * blockDim.x) >> 5) {
        double2 *col = col_ptr(s, c);
        if (c < s.n) {
#pragma unroll 4
            for (int i = lane; i < s.n; i += 32) {
                const int64_t e = i + (int64_t)c * s.R.ldk;
                col[i] = assemble_entry(ld_keep(s.R.K + e, pol), ld_keep(s.R.M + e, pol), s.R.D, e, s.R.eta, m2, w);
            }
        } else {
            for (int i = lane; i < s.n; i += 32) col[i] = s.R.rhs[i + (int64_t)(c - s.n) * s.R.ldb];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) s.st->info = 0;
}

// ---------------------------------------------------------------------------- panel
__device__ __forceinline__ uint32_t su32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t mapa(uint32_t addr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ int4 ld_cluster(uint32_t addr) {
    int4 v;
    asm volatile("ld.shared::cluster.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ double2 ld_cluster_d2(uint32_t addr) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr) : "memory");
    return v;
}
template <int CS>
__device__ __forceinline__ void cluster_sync() {
    if constexpr (CS == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// 1 / z with crecip's operations, Smith's two cases as one sequence (see sweep_lu64.cu)
__device__ __forceinline__ double2 crecip_uniform(double2 z) {
    const bool xb = fabs(z.x) >= fabs(z.y);
    const double p = xb ? z.x : z.y, q = xb ? z.y : z.x;
    const double t = __ddiv_rn(q, p);
    const double d = __dadd_rn(p, __dmul_rn(q, t));
    const double u = __drcp_rn(d), v = __ddiv_rn(t, d);
    return xb ? make_double2(u, -v) : make_double2(v, -u);
}

struct PanelSmem {
    int4 cand[2][PW];         // key (low, high word), physical row, 1 if the warp saw a NaN or a tie
    double2 inv[2][PW];       // reciprocal of the candidate
    double2 rows[2][PW][NB];  // the candidate's row
    double2 local[PW][NB];    // a warp's copy of the pivot's reciprocal (entry 0) and row
    int first;                // slow path: the first row's entry is a NaN
};

// Dynamic shared memory after PanelSmem: the multipliers of the CTA's rows (NB x PT), then at, lg (n_max
// ints each: the logical order, a copy in every CTA).
template <int CS, int W>
__device__ __forceinline__ void panel_steps(double2 (&a)[NB], double2 *l, int nbc, int j0, const Sys &s, PanelSmem &X,
                                            int *at, int *lgo, int rank, bool &done) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = rank * PT + tid;
    constexpr int NC = CS * PW, PER = (NC + 31) / 32;
    const int jj1 = min(NB - W + 4, nbc);
    for (int jj = NB - W; jj < jj1; ++jj) {
        const int buf = jj & 1;
        auto store_row = [&](int w) {
#pragma unroll
            for (int c = 0; c < W; ++c) X.rows[buf][w][c] = a[c];
        };
        const double v = cabs1(a[0]);
        const bool nan = !done && v != v;
        const unsigned long long key = done || v != v ? 0 : (unsigned long long)__double_as_longlong(v) + 1;
        const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
        const unsigned bh = __reduce_max_sync(FULL_MASK, hi);
        const double2 rec = crecip_uniform(key ? a[0] : make_double2(1.0, 0.5));
        const unsigned who = __ballot_sync(FULL_MASK, key != 0 && hi == bh);
        const int odd = __any_sync(FULL_MASK, nan) || (who & (who - 1));
        if (lane == (who ? __ffs(who) - 1 : 0)) {
            X.cand[buf][warp] = make_int4((int)lo, (int)hi, row, odd);
            X.inv[buf][warp] = rec;
            store_row(warp);
        }
        cluster_sync<CS>();
        // every warp reads all candidates of the cluster
        int4 c = make_int4(0, 0, 0, 0);
        int flag = 0, at_c = 0;
        bool tie = false;
        auto key_of = [](const int4 &q) { return ((unsigned long long)(unsigned)q.y << 32) | (unsigned)q.x; };
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int e = lane + 32 * q;
            if (e < NC) {
                const int4 d = ld_cluster(mapa(su32(&X.cand[buf][e % PW]), e / PW));
                flag |= d.w;
                tie = tie || (q > 0 && d.y == c.y && (d.x | d.y) != 0);
                if (q == 0 || key_of(d) > key_of(c)) {
                    c = d;
                    at_c = e;
                }
            }
        }
        const unsigned mh = __reduce_max_sync(FULL_MASK, (unsigned)c.y);
        const unsigned w = __ballot_sync(FULL_MASK, (unsigned)c.y == mh && (c.x | c.y) != 0);
        const bool slow = __any_sync(FULL_MASK, flag || (tie && (unsigned)c.y == mh)) || (w & (w - 1));
        const int src = w ? __ffs(w) - 1 : 0;
        int bph = __shfl_sync(FULL_MASK, c.z, src);
        int wl = __shfl_sync(FULL_MASK, at_c, src);
        unsigned long long bkey = ((unsigned long long)mh << 32) | (unsigned)__shfl_sync(FULL_MASK, c.x, src);
        bool nz = true;
        if (slow || bkey <= 1) {
            // the full rule of sweep_lu64.cu: ties by logical row, NaN first, no interchange for a zero pivot
            if (tid == 0) X.first = 0;
            cluster_sync<CS>();
            const int first = at[jj];
            if (row == first && nan) X.first = 1;
            const unsigned bl = __reduce_max_sync(FULL_MASK, hi == bh ? lo : 0u);
            const int lg = key != 0 && hi == bh && lo == bl ? lgo[row] : INT_MAX;
            const int m = __reduce_min_sync(FULL_MASK, lg);
            if (m == INT_MAX ? lane == 0 : lg == m) {
                X.cand[buf][warp] = make_int4((int)lo, (int)hi, row, 0);
                X.inv[buf][warp] = rec;
                store_row(warp);
            }
            cluster_sync<CS>();
            bkey = 0;
            bph = first;
            wl = 0;
            for (int e = 0; e < NC; ++e) {
                const int4 d = ld_cluster(mapa(su32(&X.cand[buf][e % PW]), e / PW));
                const unsigned long long k = key_of(d);
                if (k > bkey || (k == bkey && k != 0 && lgo[d.z] < lgo[bph])) {
                    bkey = k;
                    bph = d.z;
                    wl = e;
                }
            }
            const int fn = ld_cluster(mapa(su32(&X.first) & ~15u, first / PT)).x;  // X.first is 16-byte aligned
            if (fn || bkey <= 1) {
                bph = first;
                wl = first / PT * PW;
                cluster_sync<CS>();
                if (row == first) {
                    X.inv[buf][0] = crecip_uniform(a[0]);
                    store_row(0);
                }
            }
            cluster_sync<CS>();
            const double2 piv = ld_cluster_d2(mapa(su32(&X.rows[buf][wl % PW][0]), wl / PW));
            nz = piv.x != 0.0 || piv.y != 0.0;
        }
        const int wr = wl / PW, ww = wl % PW;
        // a warp fetches the pivot's reciprocal and row once, one entry a lane, into its own copy (with
        // every lane reading the whole row from the other CTA, those reads took most of a step)
        double2 *u = X.local[warp];
        if (lane < W) u[lane] = ld_cluster_d2(mapa(lane == 0 ? su32(&X.inv[buf][ww]) : su32(&X.rows[buf][ww][lane]), wr));
        __syncwarp();
        const double2 lp = nz ? cmul(a[0], u[0]) : a[0];
        l[jj * PT + tid] = lp;
#pragma unroll
        for (int c2 = 0; c2 + 1 < W; ++c2) a[c2] = csubmul(a[c2 + 1], lp, u[c2 + 1]);
        done = done || row == bph;
        if (rank == wr && warp == (ww + 1) % PW && lane < nbc - jj)
            s.A[(j0 + jj) + (int64_t)(j0 + jj + lane) * s.lda] = X.rows[buf][ww][lane];
        if (warp == PW - 1 && lane == 0) {  // the interchange of logical rows jj and lgo[bph], in every CTA
            const int first = at[jj], lgp = lgo[bph];
            at[lgp] = first;
            lgo[first] = lgp;
            lgo[bph] = jj;
            if (rank == 0) {
                s.st->piv[jj] = bph;
                s.pivlg[j0 + jj] = lgp;
                if (!nz && s.st->info == 0) s.st->info = j0 + jj + 1;
            }
        }
    }
}

template <int CS>
__global__ void __launch_bounds__(PT, 1) large_panel_kernel(Args a, int j0) {
    extern __shared__ __align__(128) unsigned char sm[];
    const Sys s = system_of(a, blockIdx.y);
    const int n = s.n, m = n - j0;
    if (m <= 0) return;  // the whole cluster: one system a cluster
    PanelSmem &X = *reinterpret_cast<PanelSmem *>(sm);
    double2 *l = reinterpret_cast<double2 *>(sm + (sizeof(PanelSmem) + 127) / 128 * 128);
    int *at = reinterpret_cast<int *>(l + NB * PT), *lgo = at + a.n_max;
    const int tid = threadIdx.x, rank = CS == 1 ? 0 : (int)blockIdx.x, row = rank * PT + tid;
    const int nbc = min(NB, m);
    double2 v[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c)
        v[c] = (row < m && c < nbc) ? s.A[(j0 + row) + (int64_t)(j0 + c) * s.lda] : make_double2(0.0, 0.0);
    bool done = row >= m;
    for (int i = tid; i < m; i += PT) {
        at[i] = i;
        lgo[i] = i;
    }
    cluster_sync<CS>();
    panel_steps<CS, 32>(v, l, nbc, j0, s, X, at, lgo, rank, done);
    panel_steps<CS, 28>(v, l, nbc, j0, s, X, at, lgo, rank, done);
    panel_steps<CS, 24>(v, l, nbc, j0, s, X, at, lgo, rank, done);
    panel_steps<CS, 20>(v, l, nbc, j0, s, X, at, lgo, rank, done);
    panel_steps<CS, 16>(v, l, nbc, j0, s, X, at, lgo, rank, done);
    panel_steps<CS, 12>(v, l, nbc, j0, s, X, at, lgo, rank, done);
    panel_steps<CS, 8>(v, l, nbc, j0, s, X, at, lgo, rank, done);
    panel_steps<CS, 4>(v, l, nbc, j0, s, X, at, lgo, rank, done);
    cluster_sync<CS>();  // the last interchange; no CTA leaves while another reads its shared memory
    // multipliers in logical row order: the unit triangle, and the rows below the panel
    if (row < m) {
        const int lg = lgo[row];
        const int64_t ldp = lda_of(n);
        if (lg < nbc) {
            for (int k = 0; k < NB; ++k) s.l11[k * NB + lg] = k < lg ? l[k * PT + tid] : make_double2(0.0, 0.0);
        } else {
#pragma unroll 8
            for (int k = 0; k < NB; ++k) s.P[(lg - NB) + k * ldp] = l[k * PT + tid];
        }
        if (s.R.LU)
            for (int k = 0; k < min(lg, nbc); ++k) s.A[(j0 + lg) + (int64_t)(j0 + k) * s.lda] = l[k * PT + tid];
    }
    if (rank == 0 && tid < 32) {
        // rows displaced from the panel's top, and the triangle's empty columns of a short last panel
        const int lg = tid < nbc ? lgo[tid] : 0;
        const unsigned mv = __ballot_sync(FULL_MASK, tid < nbc && lg >= nbc);
        if (tid < nbc && lg >= nbc) {
            const int e = __popc(mv & ((1u << tid) - 1));
            s.st->dsrc[e] = tid;
            s.st->ddst[e] = lg;
        }
        if (tid == 0) s.st->nmoved = __popc(mv);
        for (int e = tid; e < NB * NB; e += 32)
            if (e % NB >= nbc) s.l11[e] = make_double2(0.0, 0.0);
    }
}

// LAPACK's interchanges of the panel at j0 on the columns left of it (kept factors only): a warp a
// column, a lane one of the panel's places and one of the places that displaced rows go to.
__global__ void __launch_bounds__(256) large_left_kernel(Args a, int j0) {
    const Sys s = system_of(a, blockIdx.y);
    if (!s.R.LU || s.n <= j0) return;
    const int lane = threadIdx.x & 31, nbc = min(NB, s.n - j0), nm = s.st->nmoved;
    const int piv = lane < nbc ? s.st->piv[lane] : 0;
    const int src = lane < nm ? s.st->dsrc[lane] : 0, dst = lane < nm ? s.st->ddst[lane] : 0;
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < j0; c += (gridDim.x * blockDim.x) >> 5) {
        double2 *col = s.A + (int64_t)c * s.lda + j0;
        const double2 v = col[piv], d = col[src];
        __syncwarp();
        if (lane < nbc) col[lane] = v;
        if (lane < nm) col[dst] = d;
    }
}

// ---------------------------------------------------------------------------- update
__device__ __forceinline__ void dmma(double2 &c, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c.x), "+d"(c.y)
        : "d"(a), "d"(b));
}
__device__ __forceinline__ double neg_if(double v, unsigned sign) {
    return __hiloint2double(__double2hiint(v) ^ (int)sign, __double2loint(v));
}

constexpr size_t U12_SMEM = (size_t)16 * (2 * NB * LDU + NB * NB);
constexpr size_t SCHUR_SMEM = (size_t)16 * NB * (LDU + LDP);

// The panel's interchanges and U12 = L11^-1 x on a chunk of trailing columns.
__global__ void __launch_bounds__(VT) large_u12_kernel(Args a, int j0) {
    extern __shared__ __align__(128) unsigned char sm[];
    double2 *U = reinterpret_cast<double2 *>(sm);  // NB x LDU: pivot rows, then U12
    double2 *T = U + NB * LDU;                     // NB x LDU: the panel's top rows
    double2 *l11 = T + NB * LDU;
    const Sys s = system_of(a, blockIdx.y);
    const int n = s.n, m = n - j0, nbc = min(NB, m);
    const int c0 = j0 + nbc + blockIdx.x * CW, nc = min(CW, n + s.r - c0);
    if (m <= 0 || nc <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nm = s.st->nmoved;
    {
        const int piv = lane < nbc ? s.st->piv[lane] : 0;
        if (lane < nbc)
            for (int c = warp; c < nc; c += VT / 32) {
                const double2 *col = col_ptr(s, c0 + c) + j0;
                cp_async_elem(U + lane * LDU + c, col + piv);
                cp_async_elem(T + lane * LDU + c, col + lane);
            }
        for (int e = tid; e < NB * NB; e += VT) cp_async_elem(l11 + e, s.l11 + e);
        cp_async_commit();
    }
    cp_async_wait<0>();
    __syncthreads();
    // a thread a column, in halves of the triangle; the other threads move the displaced rows down
    if (tid < CW) {
        if (tid < nc) {
#pragma unroll 1
            for (int h = 0; h < 2 && h * HB < nbc; ++h) {
                double2 x[HB];
#pragma unroll
                for (int i = 0; i < HB; ++i) x[i] = h * HB + i < nbc ? U[(h * HB + i) * LDU + tid] : make_double2(0.0, 0.0);
                for (int k = 0; k < h * HB; ++k) {
                    const double2 uk = U[k * LDU + tid];
#pragma unroll
                    for (int i = 0; i < HB; ++i) x[i] = csubmul(x[i], l11[k * NB + h * HB + i], uk);
                }
                const double2 *d = l11 + h * HB * NB + h * HB;
#pragma unroll
                for (int k = 0; k < HB - 1; ++k)
#pragma unroll
                    for (int i = k + 1; i < HB; ++i) x[i] = csubmul(x[i], d[k * NB + i], x[k]);
#pragma unroll
                for (int i = 0; i < HB; ++i) U[(h * HB + i) * LDU + tid] = x[i];
            }
        }
    } else {
        for (int e = tid - CW; e < nm * nc; e += VT - CW) {
            const int q = e % nm, c = e / nm;
            col_ptr(s, c0 + c)[j0 + s.st->ddst[q]] = T[s.st->dsrc[q] * LDU + c];
        }
    }
    __syncthreads();
    if (lane < nbc)
        for (int c = warp; c < nc; c += VT / 32) col_ptr(s, c0 + c)[j0 + lane] = U[lane * LDU + c];
}

// A22 -= L21 U12 for a tile of RT rows and CW columns.  Warp w takes 16-column strip w & 3 and four of
// the tile's eight 16-row pieces; a piece's entries are loaded while the one before it is multiplied (the
// first one's while the operands are staged).
__global__ void __launch_bounds__(UT, 2) large_schur_kernel(Args a, int j0) {
    extern __shared__ __align__(128) unsigned char sm[];
    double2 *U = reinterpret_cast<double2 *>(sm);  // NB x LDU
    double2 *PS = U + NB * LDU;                    // NB x LDP
    const Sys s = system_of(a, blockIdx.z);
    const int n = s.n, mt = n - j0 - NB;
    const int t0 = blockIdx.x * RT, c0 = j0 + NB + blockIdx.y * CW, nc = min(CW, n + s.r - c0);
    if (t0 >= mt || nc <= 0) return;
    const int rows = min(RT, mt - t0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t ldp = lda_of(n);
    for (int c = warp; c < nc; c += UW) cp_async_elem(U + lane * LDU + c, col_ptr(s, c0 + c) + j0 + lane);
    for (int e = tid; e < NB * RT; e += UT) {
        const int i = e % RT, k = e / RT;
        if (i < rows) cp_async_elem(PS + k * LDP + i, s.P + t0 + i + k * ldp);
    }
    cp_async_commit();
    const int strip = warp & 3, half = warp >> 2;
    const int lr = lane >> 2, lk = (lane >> 1) & 1;
    const bool odd = lane & 1;
    const unsigned sgn_re = odd ? 0x80000000u : 0u;
    double2 *cp[4];
    bool okc[4];
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const int cc = strip * 16 + 8 * (z >> 1) + 2 * (lane & 3) + (z & 1);
        okc[z] = cc < nc;
        cp[z] = col_ptr(s, c0 + min(cc, nc - 1)) + j0 + NB + t0;
    }
    const double2 *pb = U + lk * LDU + strip * 16 + lr;
    const int p0 = half * 4, p1 = strip * 16 < nc ? min(p0 + 4, (rows + 15) / 16) : 0;
    double2 nx[2][4];
    auto load = [&](int p) {
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int row = min(p * 16 + 8 * x + lr, rows - 1);
#pragma unroll
            for (int z = 0; z < 4; ++z) nx[x][z] = cp[z][row];
        }
    };
    if (p0 < p1) load(p0);
    cp_async_wait<0>();
    __syncthreads();
    for (int p = p0; p < p1; ++p) {
        double2 re[2][2], im[2][2];  // [row tile][column tile]: components of the two columns
        const double2 *pa = PS + lk * LDP + p * 16 + lr;
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                re[x][y] = make_double2(nx[x][2 * y].x, nx[x][2 * y + 1].x);
                im[x][y] = make_double2(nx[x][2 * y].y, nx[x][2 * y + 1].y);
            }
        if (p + 1 < p1) load(p + 1);
#pragma unroll 8
        for (int k = 0; k < NB; k += 2) {
            double are[2], aim[2], bre[2], bim[2];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const double2 v = pa[k * LDP + 8 * x];
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
            const int row = p * 16 + 8 * x + lr;
            if (row < rows) {
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    if (okc[2 * y]) cp[2 * y][row] = make_double2(re[x][y].x, im[x][y].x);
                    if (okc[2 * y + 1]) cp[2 * y + 1][row] = make_double2(re[x][y].y, im[x][y].y);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------- backward substitution
// One CTA a system: 16-row blocks from the last, the triangle by one warp a right-hand side, then a
// thread a row takes the block's columns in decreasing order; the next rows' entries of U are loaded while
// the triangle is solved.
__global__ void __launch_bounds__(BT, 1) large_back_kernel(Args a) {
    extern __shared__ __align__(128) unsigned char sm[];
    const Sys s = system_of(a, blockIdx.x);
    const int n = s.n, r = s.r, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double2 *Bs = reinterpret_cast<double2 *>(sm);  // n x r
    double2 *tile = Bs + (int64_t)n * r;            // HB x (HB + 1)
    constexpr int LDT = HB + 1;
    for (int c = warp; c < r; c += BT / 32)
        for (int i = lane; i < n; i += 32) Bs[i + (int64_t)c * n] = s.B[i + (int64_t)c * s.ldb];
    for (int jb = (n - 1) / HB * HB; jb >= 0; jb -= HB) {
        const int bs = min(HB, n - jb);
        double2 u[HB];
#pragma unroll
        for (int j = 0; j < HB; ++j)
            u[j] = (tid < jb && j < bs) ? s.A[tid + (int64_t)(jb + j) * s.lda] : make_double2(0.0, 0.0);
        if (tid < HB * HB && tid % HB < bs && tid / HB < bs)
            tile[tid % HB + tid / HB * LDT] = s.A[(jb + tid % HB) + (int64_t)(jb + tid / HB) * s.lda];
        __syncthreads();
        for (int c = warp; c < r; c += BT / 32) {
            double2 *b = Bs + (int64_t)c * n + jb;
            double2 v = lane < bs ? b[lane] : make_double2(0.0, 0.0);
            const double2 dg = lane < bs ? tile[lane + lane * LDT] : make_double2(1.0, 0.5);
            // Smith's division by the diagonal: its parts without the dividend, once a lane
            const bool big = fabs(dg.x) >= fabs(dg.y);
            const double p = big ? dg.x : dg.y, q = big ? dg.y : dg.x;
            const double t = __ddiv_rn(q, p), d = __dadd_rn(p, __dmul_rn(q, t));
            for (int j = bs - 1; j >= 0; --j) {
                if (lane == j) {
                    const double x = big ? v.x : v.y, y = big ? v.y : v.x;
                    const double re = __dadd_rn(x, __dmul_rn(y, t)), im = __dsub_rn(y, __dmul_rn(x, t));
                    v = make_double2(__ddiv_rn(re, d), __ddiv_rn(big ? im : -im, d));
                }
                const double2 bj = CT<double2>::shfl(v, j, 32);
                if (lane < j) v = csubmul(v, tile[lane + j * LDT], bj);
            }
            if (lane < bs) b[lane] = v;
        }
        __syncthreads();
        for (int i = tid; i < jb; i += BT) {
            if (i != tid) {
#pragma unroll
                for (int j = 0; j < HB; ++j) u[j] = j < bs ? s.A[i + (int64_t)(jb + j) * s.lda] : make_double2(0.0, 0.0);
            }
            for (int c = 0; c < r; ++c) {
                double2 *b = Bs + (int64_t)c * n;
                double2 acc = b[i];
#pragma unroll
                for (int j = HB - 1; j >= 0; --j)
                    if (j < bs) acc = csubmul(acc, u[j], b[jb + j]);
                b[i] = acc;
            }
        }
        __syncthreads();
    }
    double2 *Xo = s.R.X + (int64_t)s.f * n * r;
    for (int e = tid; e < n * r; e += BT) Xo[e] = Bs[e];
    if (s.R.ipiv)
        for (int j = tid; j < n; j += BT) s.R.ipiv[(int64_t)s.f * n + j] = j / NB * NB + s.pivlg[j] + 1;
    if (tid == 0) {
        if (s.R.info) s.R.info[s.f] = s.st->info;
        if (s.R.steps) s.R.steps[s.f] = 0;
        if (s.R.berr) s.R.berr[s.f] = 0.0;
    }
}

static size_t panel_smem(int n_max) {
    return (sizeof(PanelSmem) + 127) / 128 * 128 + sizeof(double2) * NB * PT + (size_t)2 * n_max * 4;
}
static size_t back_smem(int n_max, int r_max) { return sizeof(double2) * ((size_t)n_max * r_max + HB * (HB + 1)); }

template <int CS>
static cudaError_t launch_panel(const Args &a, int systems, int j0, cudaStream_t st) {
    auto k = large_panel_kernel<CS>;
    const size_t smem = panel_smem(a.n_max);
    // one value for all sizes: another thread's smaller launch must not lower it between this call and this launch
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)panel_smem(LARGE_MAX_N));
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CS, systems, 1);
    cfg.blockDim = dim3(PT, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a, j0);
}

}  // namespace large

int64_t large_slot_bytes(int n_max, int r_max) { return (int64_t)large::Slot(n_max, r_max).total; }

cudaError_t launch_large(const LargeArgs &g, cudaStream_t st) {
    using namespace large;
    const size_t bsm = back_smem(g.n_max, g.r_max);
    if (g.n_max > LARGE_MAX_N || g.slot_bytes < large_slot_bytes(g.n_max, g.r_max) || bsm > SMEM_OPTIN)
        return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(large_u12_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)U12_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(large_schur_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SCHUR_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(large_back_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_OPTIN);
    if (e != cudaSuccess) return e;
    for (int i0 = 0; i0 < g.n_items; i0 += g.group) {
        const int ns = std::min(g.group, g.n_items - i0);
        const Args a{g.roms, g.items + i0, g.scratch, g.slot_bytes, g.n_max, g.r_max};
        // a warp a column; enough CTAs to fill the GPU
        large_assemble_kernel<<<dim3(std::max(1, std::min((g.n_max + g.r_max + 7) / 8, 8 * g.sms / ns)), ns), 256, 0, st>>>(a);
        for (int j0 = 0; j0 < g.n_max; j0 += NB) {
            const int m = g.n_max - j0;
            const int cs = (m + PT - 1) / PT;
            e = cs <= 1   ? launch_panel<1>(a, ns, j0, st)
                : cs <= 2 ? launch_panel<2>(a, ns, j0, st)
                : cs <= 4 ? launch_panel<4>(a, ns, j0, st)
                          : launch_panel<8>(a, ns, j0, st);
            if (e != cudaSuccess) return e;
            if (g.keep && j0 > 0)
                large_left_kernel<<<dim3(std::max(1, std::min((j0 + 7) / 8, 8 * g.sms / ns)), ns), 256, 0, st>>>(a, j0);
            const int nbc = std::min(NB, m), left = m - nbc + g.r_max;
            // systems of smaller order in the group have their last, short panel earlier: their right-hand
            // sides start nearer to it, so the chunks are counted from the panel's first column
            large_u12_kernel<<<dim3((left + NB + CW - 1) / CW, ns), VT, U12_SMEM, st>>>(a, j0);
            if (m > NB)
                large_schur_kernel<<<dim3((m - NB + RT - 1) / RT, (left + CW - 1) / CW, ns), UT, SCHUR_SMEM, st>>>(a, j0);
        }
        large_back_kernel<<<ns, BT, bsm, st>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

}  // namespace srom
