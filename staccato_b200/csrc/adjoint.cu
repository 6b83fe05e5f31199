// Adjoint (backward) sweep: parameter gradients of a real objective J(x(w_1..w_F)).
//
// For every frequency, with the FP64 factors P A = L U kept by the forward sweep
// (SROM_FLAG_KEEP_FACTORS) and the cotangent gbar_f = 2 dJ/d conj(x_f):
//     A^H lambda = gbar      (U^H y = gbar, L^H z = y, lambda = P^T z)
//     dJ/dp_j  += -Re( sum_c lambda_c^H dA_j(w) x_c ),
// where dA_j(w) = (c0 + c1 (i w) + c2 (-w^2)) G_j and G_j is either dense or U diag(s) W^T
// (low rank; the stiffness-scaling parameters of a modal ROM are rank-8 blocks).
// The reference has no adjoint; this is the backward call of the sweep.
//
// Two parts.  The solves (adjoint_solve_kernel): one CTA of four warps a frequency, several a
// multiprocessor.  The terms: lambda^H U and W^T x of all frequencies and all rank terms are two
// complex GEMMs, G x of all frequencies is one a dense parameter (zgemm.cu), and a warp a
// (frequency, parameter) combines them; so U, W and G are read once a GEMM tile instead of once a
// frequency.  Small calls, bound by launches, take their terms in the solve kernel (fused_terms).
// Per-frequency contributions are summed in a fixed order: the gradient is deterministic.
//
// What bounds it: the solves read the kept factors once (F n^2 16 bytes from HBM) behind a chain of 2 n
// dependent steps a frequency; 32-row blocks keep that chain at one warp's 32 steps a block with the
// products of the rows before it spread over all warps.  n = 128, 2000 frequencies, 16 rank-8
// parameters and one dense (B200, the whole backward call): 2.4 ms with the dot products of every
// row and every term taken by single warps, 0.40 ms now; the factors alone are 0.08 ms at the copy
// bandwidth.  Workspace beyond what the caller gives: the products of a pass (up to about 256 MB, kept in
// the handle) and lambda (F n r) when it is not asked for.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "adjoint_kernels.h"
#include "srom_device.cuh"
#include "zgemm.h"

namespace srom {

constexpr int ADJ_NT = 128;
constexpr int ADJ_NW = ADJ_NT / 32;
constexpr int ADJ_B = 32;             // rows of a block
constexpr int ADJ_LDT = ADJ_B + 1;
constexpr int ADJ_RC = 2;             // right-hand sides a pass of the block products
constexpr int ADJ_CPW = ADJ_B / ADJ_NW;  // columns of a block a warp

__device__ __forceinline__ double2 conj2(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {  // c + a*b
    return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ double2 shfl2(double2 v, int src) {
    return make_double2(__shfl_sync(FULL_MASK, v.x, src), __shfl_sync(FULL_MASK, v.y, src));
}

__device__ __forceinline__ double2 warp_sum2(double2 v) {
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        v.x += __shfl_xor_sync(FULL_MASK, v.x, off);
        v.y += __shfl_xor_sync(FULL_MASK, v.y, off);
    }
    return v;
}

// Y[j0 + j] -= sum_{i in [lo, hi)} conj(LU[i, j0 + j]) Y[i] for the block's columns j < bs and all
// right-hand sides: every warp takes ADJ_CPW columns, lanes over the rows, all columns' loads of a row
// step in flight together.
__device__ __forceinline__ void block_products(const double2 *__restrict__ LU, int n, int j0, int bs, int lo, int hi,
                                               double2 *Y, int r) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int jw = warp * ADJ_CPW;
    if (jw >= bs || lo >= hi) return;
    for (int c0 = 0; c0 < r; c0 += ADJ_RC) {
        double2 s[ADJ_CPW][ADJ_RC];
#pragma unroll
        for (int q = 0; q < ADJ_CPW; ++q)
#pragma unroll
            for (int c = 0; c < ADJ_RC; ++c) s[q][c] = make_double2(0.0, 0.0);
        for (int i = lo + lane; i < hi; i += 32) {
            double2 a[ADJ_CPW], y[ADJ_RC];
#pragma unroll
            for (int q = 0; q < ADJ_CPW; ++q)
                a[q] = jw + q < bs ? conj2(LU[i + (int64_t)(j0 + jw + q) * n]) : make_double2(0.0, 0.0);
#pragma unroll
            for (int c = 0; c < ADJ_RC; ++c) y[c] = c0 + c < r ? Y[i + (int64_t)(c0 + c) * n] : make_double2(0.0, 0.0);
#pragma unroll
            for (int q = 0; q < ADJ_CPW; ++q)
#pragma unroll
                for (int c = 0; c < ADJ_RC; ++c) s[q][c] = cfma(a[q], y[c], s[q][c]);
        }
#pragma unroll
        for (int q = 0; q < ADJ_CPW; ++q)
#pragma unroll
            for (int c = 0; c < ADJ_RC; ++c) {
                if (c0 + c >= r) break;
                const double2 v = warp_sum2(s[q][c]);
                if (lane == 0 && jw + q < bs) {
                    double2 &y = Y[j0 + jw + q + (int64_t)(c0 + c) * n];
                    y.x -= v.x;
                    y.y -= v.y;
                }
            }
    }
}

// The power of two that keeps a pivot's reciprocal in the normal range: y = v / u is (sc v) (1 / (sc u)).
__device__ __forceinline__ double pivot_scale(double2 u) {
    const double m = fmax(fabs(u.x), fabs(u.y));
    return m < 0x1p-1000 ? 0x1p600 : m > 0x1p1000 ? 0x1p-600 : 1.0;
}

// The block's diagonal triangle, conjugated and transposed: tile[i * ADJ_LDT + j] = conj(LU[j0 + j, j0 + i])
__device__ __forceinline__ void load_tile(const double2 *__restrict__ LU, int n, int j0, int bs, double2 *tile) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = warp; c < bs; c += ADJ_NW)
        if (lane < bs) tile[c * ADJ_LDT + lane] = conj2(LU[(j0 + lane) + (int64_t)(j0 + c) * n]);
}

// coef(w) = c0 + c1 (i w) + c2 (-w^2); -Re(coef S)
__device__ __forceinline__ double contribution(const DParamDev &P, double w, double2 S) {
    const double2 coef = make_double2(P.c0.x - w * P.c1.y - w * w * P.c2.x, P.c0.y + w * P.c1.x - w * w * P.c2.y);
    return -(coef.x * S.x - coef.y * S.y);
}

// All terms of one frequency by its CTA, from lambda and x (n x r each) in shared memory: a warp a rank term, a dense
// matrix's columns shared out over the warps.  part: ADJ_NW entries a term.
__device__ __forceinline__ void frequency_terms(const AdjointArgs &a, int f, double w, int n, int r, const double2 *lam,
                                                const double2 *x, double2 *part) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = 0; t < a.n_terms; ++t) {
        const DParamTerm T = a.terms[t];
        const DParamDev &P = a.params[T.param];
        const bool dense = P.kind != 0;
        if (!dense && t % ADJ_NW != warp) continue;
        double2 S = make_double2(0.0, 0.0);
        if (dense) {
            for (int i = lane; i < n; i += 32)
                for (int c = 0; c < r; ++c) {
                    double2 g = make_double2(0.0, 0.0);
#pragma unroll 4
                    for (int l = warp; l < n; l += ADJ_NW) g = cfma(P.G[i + (int64_t)l * n], x[l + c * n], g);
                    S = cfma(conj2(lam[i + c * n]), g, S);
                }
            S = warp_sum2(S);
        } else {
            const double2 *u = P.U + (int64_t)T.k * n, *v = (P.W ? P.W : P.U) + (int64_t)T.k * n;
            const double s = P.s ? P.s[T.k] : 1.0;
            for (int c = 0; c < r; ++c) {
                double2 p = make_double2(0.0, 0.0), q = p;
                for (int i = lane; i < n; i += 32) {
                    p = cfma(conj2(lam[i + c * n]), u[i], p);
                    q = cfma(v[i], x[i + c * n], q);
                }
                p = warp_sum2(p);
                q = warp_sum2(q);
                S = cfma(make_double2(s * p.x, s * p.y), q, S);
            }
        }
        if (lane == 0) part[t * ADJ_NW + (dense ? warp : 0)] = S;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < a.n_params; j += ADJ_NT) {
        const DParamDev &P = a.params[j];
        double2 S = make_double2(0.0, 0.0);
        for (int t = P.term0; t < P.term0 + P.nterm; ++t)
            for (int q = 0; q < (P.kind != 0 ? ADJ_NW : 1); ++q) {
                S.x += part[t * ADJ_NW + q].x;
                S.y += part[t * ADJ_NW + q].y;
            }
        a.partial[(int64_t)f * a.n_params + j] = contribution(P, w, S);
    }
}

// TERMS: the CTA takes its frequency's terms too (small calls; n r <= ADJ_B ADJ_LDT), and lambda may be null.
template <bool TERMS>
__global__ void __launch_bounds__(ADJ_NT, 4) adjoint_solve_kernel(AdjointArgs a) {
    extern __shared__ double2 sh[];
    __shared__ int s_item, s_scaled;
    const RomDev R = *a.rom;
    const int n = R.n, r = R.r;
    double2 *Y = sh;                                          // n x r
    double2 *dinv = Y + (int64_t)n * r;                       // reciprocals of the block's conj(diag U)
    double2 *tile = dinv + ADJ_B;                             // ADJ_B x ADJ_LDT
    int *perm = reinterpret_cast<int *>(tile + ADJ_B * ADJ_LDT);  // original row of a position
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (;;) {
        if (tid == 0) s_item = atomicAdd(a.counter, 1);
        __syncthreads();
        const int f = s_item;
        __syncthreads();
        if (f >= R.F) break;
        const double2 *LU = R.LU + (int64_t)f * n * n;
        const int *ipiv = R.ipiv + (int64_t)f * n;
        for (int c = warp; c < r; c += ADJ_NW)
            for (int i = lane; i < n; i += 32) Y[i + (int64_t)c * n] = a.gbar[(int64_t)f * a.ldg_f + i + (int64_t)c * a.ldg];
        for (int i = tid; i < n; i += ADJ_NT) perm[i] = i;
        __syncthreads();
        // U^H y = gbar, blocks from the first; the last warp meanwhile follows the interchanges
        for (int j0 = 0; j0 < n; j0 += ADJ_B) {
            const int bs = min(ADJ_B, n - j0);
            load_tile(LU, n, j0, bs, tile);
            if (warp == ADJ_NW - 1) {
                const double2 u = lane < bs ? conj2(LU[(j0 + lane) + (int64_t)(j0 + lane) * n]) : make_double2(1.0, 0.0);
                const double sc = pivot_scale(u);
                if (lane < bs) dinv[lane] = crecip(make_double2(u.x * sc, u.y * sc));
                const bool scaled = __any_sync(FULL_MASK, sc != 1.0);
                if (lane == 0) s_scaled = scaled;
            }
            block_products(LU, n, j0, bs, 0, j0, Y, r);
            __syncthreads();
            for (int c = warp; c < r; c += ADJ_NW) {
                double2 *y = Y + (int64_t)c * n + j0;
                double2 v = lane < bs ? y[lane] : make_double2(0.0, 0.0);
                const double2 di = lane < bs ? dinv[lane] : make_double2(0.0, 0.0);
                // row j is complete in its lane; the others subtract conj(U[j, lane]) y_j
                auto step = [&](int j, double2 num) {
                    const double2 t = tile[min(lane, bs - 1) * ADJ_LDT + j];
                    const double2 m = cfma(num, di, make_double2(0.0, 0.0));
                    const double2 yj = shfl2(m, j);
                    if (lane == j) v = m;
                    if (lane > j) v = cfma(make_double2(-t.x, -t.y), yj, v);
                };
                if (!s_scaled) {
                    for (int j = 0; j < bs; ++j) step(j, v);
                } else {
                    const double sc = lane < bs ? pivot_scale(LU[(j0 + lane) + (int64_t)(j0 + lane) * n]) : 1.0;
                    for (int j = 0; j < bs; ++j) step(j, make_double2(v.x * sc, v.y * sc));
                }
                if (lane < bs) y[lane] = v;
            }
            if (warp == ADJ_NW - 1) {
                const int p = lane < bs ? ipiv[j0 + lane] - 1 : 0;
                for (int j = 0; j < bs; ++j) {
                    const int pj = __shfl_sync(FULL_MASK, p, j);
                    if (lane == 0 && pj != j0 + j) {
                        const int t = perm[j0 + j];
                        perm[j0 + j] = perm[pj];
                        perm[pj] = t;
                    }
                }
            }
            __syncthreads();
        }
        // L^H z = y (unit diagonal), blocks from the last
        for (int j0 = (n - 1) / ADJ_B * ADJ_B; j0 >= 0; j0 -= ADJ_B) {
            const int bs = min(ADJ_B, n - j0);
            load_tile(LU, n, j0, bs, tile);
            block_products(LU, n, j0, bs, j0 + bs, n, Y, r);
            __syncthreads();
            for (int c = warp; c < r; c += ADJ_NW) {
                double2 *y = Y + (int64_t)c * n + j0;
                double2 v = lane < bs ? y[lane] : make_double2(0.0, 0.0);
                for (int j = bs - 1; j > 0; --j) {
                    const double2 t = tile[min(lane, bs - 1) * ADJ_LDT + j];
                    const double2 zj = shfl2(v, j);
                    if (lane < j) v = cfma(make_double2(-t.x, -t.y), zj, v);
                }
                if (lane < bs) y[lane] = v;
            }
            __syncthreads();
        }
        // lambda = P^T z
        if (!TERMS || a.lambda) {
            double2 *lam = a.lambda + (int64_t)f * n * r;
            for (int c = warp; c < r; c += ADJ_NW)
                for (int i = lane; i < n; i += 32) lam[perm[i] + (int64_t)c * n] = Y[i + (int64_t)c * n];
        }
        if constexpr (TERMS) {
            double2 *part = dinv + ADJ_B + ADJ_B * ADJ_LDT + (n + 3) / 4;  // past perm
            for (int c = warp; c < r; c += ADJ_NW)
                for (int i = lane; i < n; i += 32) tile[perm[i] + c * n] = Y[i + c * n];
            __syncthreads();
            for (int e = tid; e < n * r; e += ADJ_NT) Y[e] = R.X[(int64_t)f * n * r + e];
            __syncthreads();
            frequency_terms(a, f, R.omega[f], n, r, tile, Y, part);
        }
        __syncthreads();
    }
}

// The rank terms' columns side by side: Ua, Wa (n x terms) and their scales.
__global__ void adjoint_pack_kernel(const DParamDev *__restrict__ params, const DParamTerm *__restrict__ terms, int n,
                                    double2 *__restrict__ Ua, double2 *__restrict__ Wa, double *__restrict__ sa) {
    const int t = blockIdx.x;
    const DParamTerm T = terms[t];
    const DParamDev &P = params[T.param];
    if (P.kind != 0) return;
    const double2 *u = P.U + (int64_t)T.k * n, *w = (P.W ? P.W : P.U) + (int64_t)T.k * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        Ua[i + (int64_t)t * n] = u[i];
        Wa[i + (int64_t)t * n] = w[i];
    }
    if (threadIdx.x == 0) sa[t] = P.s ? P.s[T.k] : 1.0;
}

// One warp a (frequency, parameter) of the frequencies [f0, f0 + nf).  Low rank: S = sum over the
// parameter's terms t and right-hand sides c of s_t conj(Sa[t, fc]) Sb[t, fc], Sa = Ua^H lambda,
// Sb = Wa^T x.  dense >= 0: that parameter only, S = sum_c lambda_c^H (G x)_c with (G x) in GX.
__global__ void adjoint_combine_kernel(AdjointArgs a, int n, int r, int f0, int nf, int nt, int dense,
                                       const double2 *__restrict__ Sa, const double2 *__restrict__ Sb,
                                       const double *__restrict__ sa, const double2 *__restrict__ GX) {
    const int lane = threadIdx.x & 31;
    const int64_t nwarp = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int np = dense >= 0 ? 1 : a.n_params;
    for (int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < (int64_t)nf * np; e += nwarp) {
        const int f = (int)(e / np), j = dense >= 0 ? dense : (int)(e % np);
        const DParamDev &P = a.params[j];
        double2 S = make_double2(0.0, 0.0);
        if (dense >= 0) {
            const double2 *lam = a.lambda + (int64_t)(f0 + f) * n * r, *gx = GX + (int64_t)f * n * r;
            for (int i = lane; i < n * r; i += 32) S = cfma(conj2(lam[i]), gx[i], S);
        } else {
            if (P.kind != 0) continue;
            for (int k = lane; k < P.nterm * r; k += 32) {
                const int t = P.term0 + k % P.nterm;
                const int64_t at = t + ((int64_t)f * r + k / P.nterm) * nt;
                const double2 u = conj2(Sa[at]), v = Sb[at];
                S = cfma(make_double2(sa[t] * u.x, sa[t] * u.y), v, S);
            }
        }
        S = warp_sum2(S);
        if (lane == 0) a.partial[(int64_t)(f0 + f) * a.n_params + j] = contribution(P, a.rom->omega[f0 + f], S);
    }
}

// out[j] = sum over the frequencies in a fixed order: thread t takes f = t, t + 256, ..., then a tree
__global__ void __launch_bounds__(256) adjoint_reduce_kernel(const double *__restrict__ partial, int F, int P,
                                                             double *__restrict__ out) {
    __shared__ double red[256];
    const int j = blockIdx.x, t = threadIdx.x;
    double s = 0.0;
    for (int f = t; f < F; f += 256) s += partial[(int64_t)f * P + j];
    red[t] = s;
    __syncthreads();
    for (int h = 128; h; h >>= 1) {
        if (t < h) red[t] += red[t + h];
        __syncthreads();
    }
    if (t == 0) out[j] = red[0];
}

// The limit that a call is refused by: two n x r blocks and an entry a term within a CTA's shared memory.  The kernels
// above need less (solve_smem_bytes); the limit is part of the interface and stays.
size_t adjoint_smem_bytes(int n, int r, int n_terms) {
    return sizeof(double2) * ((size_t)2 * n * r + (size_t)n_terms);
}

static size_t solve_smem_bytes(int n, int r) {
    return sizeof(double2) * ((size_t)n * r + ADJ_B + ADJ_B * ADJ_LDT) + sizeof(int) * (size_t)n;
}

// The solve kernel takes the terms too: calls of one wave (four CTAs a multiprocessor) whose terms are a few thousand
// multiply-adds a thread at most.  Apart they are up to nine launches: n = 8, 64 frequencies, one rank term, two dense
// 84 us apart, 42 together (48 with the one-launch kernel before the GEMMs); n = 24, three rank-8 and two dense 99 /
// 56; n = 128, sixteen rank-8 180 / 142, 592 frequencies 221 / 182; but n = 200, r = 3, sixteen rank-8 and two dense
// (3.9e5 multiply-adds) at 592 frequencies 547 / 596.
static bool fused_terms(int n, int r, int n_terms, int n_dense, int F, int sms) {
    const int64_t work = (int64_t)r * n * (2LL * (n_terms - n_dense) + (int64_t)n * n_dense);
    return F <= 4 * sms && (int64_t)n * r <= ADJ_B * ADJ_LDT && n_terms <= 512 && work <= 1LL << 17;
}

static size_t up256(size_t b) { return (b + 255) / 256 * 256; }

// Frequencies a pass of the terms takes: its products (two a term and right-hand side, and n a
// right-hand side for a dense parameter) in about 256 MB.
static int term_chunk(int n, int r, int n_terms, int F) {
    const size_t per = sizeof(double2) * (size_t)r * ((size_t)2 * n_terms + n);
    const size_t cols = (size_t)4 << 20;  // columns of one product (the GEMM's grid takes 65535 tiles of 64)
    return (int)std::max<size_t>(1, std::min<size_t>({(size_t)F, ((size_t)256 << 20) / per, cols / 2 / r}));
}

size_t adjoint_work_bytes(int n, int r, int n_terms, int F, bool own_lambda) {
    const size_t c = (size_t)term_chunk(n, r, n_terms, F) * r;
    return (own_lambda ? up256(sizeof(double2) * (size_t)F * n * r) : 0) + 2 * up256(sizeof(double2) * (size_t)n * n_terms) +
           up256(sizeof(double) * n_terms) + 2 * up256(sizeof(double2) * c * n_terms) + up256(sizeof(double2) * c * n);
}

cudaError_t launch_adjoint(const AdjointArgs &a0, const DParamDev *params, const double2 *X, int n, int r, int F,
                           void *work, int sms, double *dJdp, cudaStream_t st) {
    AdjointArgs a = a0;
    char *w = static_cast<char *>(work);
    auto take = [&](size_t bytes) {
        char *p = w;
        w += up256(bytes);
        return p;
    };
    if (!a.lambda) a.lambda = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)F * n * r));
    const int nt = a.n_terms, fc = term_chunk(n, r, nt, F);
    double2 *Ua = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)n * nt));
    double2 *Wa = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)n * nt));
    double *sa = reinterpret_cast<double *>(take(sizeof(double) * nt));
    double2 *Sa = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)fc * r * nt));
    double2 *Sb = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)fc * r * nt));
    double2 *GX = reinterpret_cast<double2 *>(w);
    bool lowrank = false;
    int n_dense = 0;
    for (int j = 0; j < a.n_params; ++j) {
        lowrank = lowrank || (params[j].kind == 0 && params[j].nterm > 0);
        n_dense += params[j].kind != 0 ? params[j].nterm : 0;
    }

    const bool fused = fused_terms(n, r, nt, n_dense, F, sms);
    if (fused) a.lambda = a0.lambda;
    auto kernel = fused ? adjoint_solve_kernel<true> : adjoint_solve_kernel<false>;
    const size_t smem = solve_smem_bytes(n, r) + (fused ? sizeof(double2) * (size_t)(1 + nt * ADJ_NW) : 0);
    // one value for all sizes: another thread's smaller launch must not lower it between this call and this launch
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, ADJ_NT, smem);
    if (e != cudaSuccess) return e;
    kernel<<<std::min(F, sms * std::max(per_sm, 1)), ADJ_NT, smem, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (fused) {
        adjoint_reduce_kernel<<<a.n_params, 256, 0, st>>>(a.partial, F, a.n_params, dJdp);
        return cudaGetLastError();
    }
    // parameters without a term contribute nothing
    if ((e = cudaMemsetAsync(a.partial, 0, sizeof(double) * (size_t)F * a.n_params, st)) != cudaSuccess) return e;
    if (lowrank) {
        adjoint_pack_kernel<<<nt, 128, 0, st>>>(a.params, a.terms, n, Ua, Wa, sa);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    auto gemm = [&](int opa, int m, int nn, int k, const double2 *A, const double2 *B, double2 *C) {
        Zgemm z;
        z.opa = opa;
        z.opb = ZG_N;
        z.m = m;
        z.n = nn;
        z.k = k;
        z.alpha = make_double2(1.0, 0.0);
        z.beta = make_double2(0.0, 0.0);
        z.A = A;
        z.lda = opa == ZG_N ? m : k;
        z.B = B;
        z.ldb = k;
        z.C = C;
        z.ldc = m;
        z.sms = sms;
        return zgemm(z, st);
    };
    for (int f0 = 0; f0 < F; f0 += fc) {
        const int nf = std::min(fc, F - f0);
        const double2 *lam = a.lambda + (int64_t)f0 * n * r, *x = X + (int64_t)f0 * n * r;
        auto combine = [&](int dense) {
            const int64_t warps = (int64_t)nf * (dense >= 0 ? 1 : a.n_params);
            adjoint_combine_kernel<<<(int)std::min<int64_t>((warps + 7) / 8, 8LL * sms), 256, 0, st>>>(
                a, n, r, f0, nf, nt, dense, Sa, Sb, sa, GX);
            return cudaGetLastError();
        };
        if (lowrank) {
            if ((e = gemm(ZG_C, nt, nf * r, n, Ua, lam, Sa)) != cudaSuccess) return e;
            if ((e = gemm(ZG_T, nt, nf * r, n, Wa, x, Sb)) != cudaSuccess) return e;
            if ((e = combine(-1)) != cudaSuccess) return e;
        }
        for (int j = 0; j < a.n_params; ++j)
            if (params[j].kind != 0) {
                if ((e = gemm(ZG_N, n, nf * r, n, params[j].G, x, GX)) != cudaSuccess) return e;
                if ((e = combine(j)) != cudaSuccess) return e;
            }
    }
    adjoint_reduce_kernel<<<a.n_params, 256, 0, st>>>(a.partial, F, a.n_params, dJdp);
    return cudaGetLastError();
}

}  // namespace srom
