// Host-side entry points of the sweep kernels (used by the C ABI in capi.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace srom {

struct RomDev;
struct Item;

// The kernels read and write complex values as 16-byte vectors (double2), doubles as 8 bytes
// and ints as 4; srom_complex itself only promises 8-byte alignment, so device pointers are
// checked on the host before any launch (a misaligned vector access would fault the kernel).
inline bool misaligned(const void *p, size_t a) { return p && (reinterpret_cast<uintptr_t>(p) % a) != 0; }

// ---- FP64 (bit-identical to the restated zgetrf/zgetrs) ----
// bytes of a whole n x n system with its right-hand sides and pivots: the small orders are those
// whose system fits a CTA's shared memory
size_t fp64_smem_bytes(int n, int r);
// The shared-memory kernel (sweep.cu): the smallest orders and the widest right-hand sides; smem: the largest
// system's bytes
bool fp64_smem_faster(int n, int r, long long systems, int sms);
int fp64_smem_blocks_per_sm(size_t smem);
cudaError_t launch_fp64_smem(const RomDev *roms, const Item *items, int n_items, int *counter,
                             size_t smem, int grid, cudaStream_t st);
size_t fp64_global_smem_bytes(int n_max, int r_max);
// dynamic shared memory of the global kernels; big: the large-order FP64 instances
size_t global_smem_bytes(int n_max, int r_max, bool big = false);
// the shared-memory-panel instances (launch_global) can run (n_max, r_max)
bool global_panel_fits(int n_max, int r_max, int smem_optin);
int global_rpt(int n_max);
constexpr int GLOBAL_MAX_RPT = 3;   // rows per thread of the shared-memory-panel instances
constexpr int BIG_MAX_N = 2560;     // the largest order of all
// large-order FP64 instance: global scratch per CTA (the matrix, then the 16-column panel)
int64_t big_panel_offset(int n_max);
int64_t big_slot_bytes(int n_max);
constexpr int MIXED_MAX_R = 16;
constexpr size_t GLOBAL_STATIC_SMEM = 4096;
constexpr size_t SMEM_OPTIN = 227 * 1024;  // shared memory a CTA may have
// Arguments of the global-storage kernels.
struct GlobalArgs {
    const RomDev *roms;
    const Item *items;
    int n_items;
    const int *n_items_dev;  // when non-null, the item count is read from device memory
    int *counter;            // work counter (zero before the launch)
    unsigned char *scratch;  // one slot of slot_bytes per CTA
    int64_t slot_bytes;
    int ldp, n_max, r_max;
    int max_refine;
    double tol;
    Item *fb_items;  // mixed: non-converged systems are appended here (null: keep the last iterate)
    int *fb_count;
    int steps_value;  // FP64: value stored in steps (0; -1 when re-solving mixed fallbacks)
    int smem_dyn;     // dynamic shared memory of the launch (set by launch_global)
    int *err_flag;    // tensor-core kernel: set to 1 when a bounded device-side wait ran out
    int64_t panel_off;  // large-order FP64 instances: offset of the panel in a slot (set by launch_global_big)
};
// Global-storage kernel, FP64 (mixed = false) or complex-FP32 factors + FP64 refinement.
cudaError_t launch_global(bool mixed, const GlobalArgs &a, int grid, cudaStream_t st);
// The same with the FP64 panel in global scratch (slot_bytes >= big_slot_bytes(n_max)): systems up to
// n = 768 whose panel and right-hand sides do not fit shared memory together
cudaError_t launch_global_big(const GlobalArgs &a, int grid, cudaStream_t st);

// ---- FP64, orders up to LU64_MAX_N (sweep_lu64.cu): one thread a row, Schur updates on the FP64
// tensor cores; threads = 64, 128, 256 or 512, at least n_max ----
constexpr int LU64_MAX_N = 512;
int lu64_blocks_per_sm(int threads, int n_max);
constexpr int lu64_lda(int n) { return (n + 7) / 8 * 8; }
// global scratch per CTA: the matrix and the right-hand sides
constexpr int64_t lu64_slot_bytes(int n_max, int r_max) {
    return ((int64_t)lu64_lda(n_max) * ((int64_t)n_max + r_max) * 16 + 127) / 128 * 128;
}
cudaError_t launch_lu64(int threads, const GlobalArgs &a, int grid, cudaStream_t st);

// ---- FP64, large orders (sweep_large.cu): groups of systems advance panel by panel, several
// multiprocessors a system; a sequence of launches on the stream ----
constexpr int LARGE_MAX_N = BIG_MAX_N;
struct LargeArgs {
    const RomDev *roms;
    const Item *items;
    int n_items;
    int group;               // systems in flight: scratch holds group slots
    unsigned char *scratch;
    int64_t slot_bytes;      // at least large_slot_bytes(n_max, r_max)
    int n_max, r_max, sms;
    bool keep;               // some system keeps its factors
};
int64_t large_slot_bytes(int n_max, int r_max);
cudaError_t launch_large(const LargeArgs &a, cudaStream_t st);

// ---- tensor-core mixed form (sweep_tc.cu): complex-FP32 LU whose Schur updates run as
// tcgen05 MMAs on three-piece bf16 splits, FP64 refinement as in the global kernel ----
constexpr int TC_MAX_N = 512;
size_t tc_slot_bytes(int n_max);                 // global scratch per CTA
size_t tc_smem_bytes(int n_max, int r_max);      // dynamic shared memory of the launch
// Whether the kernel handles systems up to n_max with r_max right-hand sides; why (may be
// null) receives the reason when it does not.
bool tc_supported(int n_max, int r_max, int smem_optin, const char **why);
// a.slot_bytes must be at least tc_slot_bytes(a.n_max); a.fb_items / a.err_flag as for the
// mixed global kernel.
cudaError_t launch_tc(const GlobalArgs &a, int grid, cudaStream_t st);

// Back-projection Y_f = C X_f of one ROM's solutions (F blocks of n x r -> n_out x r).
struct BackProj {
    int n, r, F, n_out, ldc;
    const double2 *C;
    const double2 *X;
    double2 *Y;
};
cudaError_t launch_backproject(const BackProj &p, int sms, cudaStream_t st);

}  // namespace srom
