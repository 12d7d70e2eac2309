// gpufft_internal.h — the plan object shared by the host translation units.
#pragma once
#include <cstdarg>
#include <cstddef>
#include <cstdint>
#include <string>

#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/gpufft_b200.h"
#include "fast_registry.h"
#include "fft_kernels.cuh"

namespace gpufft {

namespace axis {
struct Form;
}

struct Plan {
    int64_t nx = 0, ny = 0, nz = 0;
    int dtype = 0;
    int device = 0;
    void *tw_dev = nullptr;     // x, y, z twiddle tables back to back
    void *stage_dev = nullptr;  // per-stage tables of the specialised kernels
    PassAParams pa{};
    PassBParams pb{};
    size_t smem_a = 0, smem_b = 0;
    int grid_a = 0, grid_b = 0;
    int occ_a = 0, occ_b = 0;
    // compile-time specialised kernels, when the registry has this shape
    const fast::VariantA *fa = nullptr;
    const fast::VariantB *fb = nullptr;
    int grid_fa = 0, grid_fb = 0, k_fa = 1, occ_fa = 0, occ_fb = 0;
    int idx_a = 0, idx_b = 0;  // registry candidate in use per pass (-1 = generic kernels)
    int kfix = 0;              // specialised Pass A cluster size (0: chosen from the L2 size;
                               // -1: split Pass A, z rows and y columns in two launches)
    bool split_a = false;      // specialised Pass A runs as two launches (kfix == -1)
    bool tc_split = false;     // x pass on the tensor-core radix-16 kernels (GPUFFT_PLAN_TC_SPLIT)
    bool tuned = false;
    // queue-scheduled Pass A (kind 2, fft_queue.cuh): counters, the forward and
    // inverse item lists and the full unpack table in one allocation
    void *q_dev = nullptr;
    int q_depth = 0;     // planes between a plane's first and second phase in the lists
    int q_nitems = 0;    // items per launch
    int q_need = 0;      // first-phase items per plane (forward)
    int q_extra = 0;     // test hook: items a plane's second phase waits for beyond those that exist
    const int *q_items_f = nullptr, *q_items_i = nullptr;
    const void *q_unp = nullptr;    // forward unpack factors
    const void *q_unp_i = nullptr;  // inverse pack factors
    const void *q_rtw = nullptr;  // the row FFT's step-1 twiddles
    // one-axis-per-launch kernels (axis.cu), made when a pass has no
    // specialised kernel or they are the faster choice (axis_a, axis_b).  Then fa
    // or fb is null, but for the fa of a plan that also runs the exchange layout.
    axis::Form *axis = nullptr;
    bool axis_a = false, axis_b = false;
    bool exchange = false;
};

// Programmatic dependent launches (fft_kernels.cuh).  R2C + C2R of a
// transform whose launches start while the one before drains, us: 100^3 FP32
// 36.2 -> 26.6, 128^3 47.2 -> 43.0, 200^3 91.6 -> 87.6, 256^3 FP64 312 -> 301.
// Fields above 400 MB gain nothing (500^3 FP32 1185 -> 1195) and go plainly.
inline cudaLaunchAttribute dependent_launch() {
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    return a;
}
inline bool chain_inside(const Plan &P) {
    return (double)P.nx * P.ny * (P.nz / 2 + 1) * (P.dtype == GPUFFT_FLOAT ? 8 : 16) <= 400e6;
}
// Whether a transform's first launch may be one too: whatever kernel is before
// it in the stream has completed when its wait returns.  Not under capture,
// where what comes before may be no kernel.
inline bool chain_first(const Plan &P, cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (!chain_inside(P)) return false;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return st == cudaStreamCaptureStatusNone;
}

namespace axis {
// Makes what P's Pass A (a) or x pass (b) needs, once each, if fft_axis.cuh
// takes its lengths (has_a: the z and y axes, has_b: the x axis).  Only the
// passes that will run: their kernels are loaded here.
int form_create(Plan &P, bool a, bool b);
void form_destroy(Plan &P);
bool has_a(const Plan &P);
bool has_b(const Plan &P);
// (chained: the first launch goes as a programmatic dependent one)
int launch_a(const Plan &P, void *data, cudaStream_t s, bool fwd, bool chained);
int launch_b(const Plan &P, void *data, cudaStream_t s, bool fwd, double scale, int dealias, bool chained);
void form_describe(const Plan &P, std::string &out, bool a, bool b);
}  // namespace axis

int set_error(int code, const char *fmt, ...);
const char *last_error();
// Raises a kernel's dynamic shared memory limit on the current device to at
// least `bytes`.  Never lowers it: plans of different sizes share the generic
// kernels, and a later, smaller plan must not undo an earlier plan's limit.
cudaError_t raise_smem_limit(const void *fn, size_t bytes);
// tensor map of a 2D view in 8-byte elements (gpufft.cu)
bool encode_view(CUtensorMap *m, void *data, long long width, long long lines, long long pitch, int box_w, int box_h);
// slab-decomposed plans (dist.cu), for the reference-shaped process-wide plans
struct DistPlan;
int dist_exec(DistPlan *D, void *data, cudaStream_t s, bool fwd);
void dist_free(DistPlan *D);
// (kPlanExchange among the flags: the plan also runs its Pass A in the exchange layout)
constexpr int kPlanExchange = 1 << 30;
int plan_create(Plan **out, int64_t nx, int64_t ny, int64_t nz, int dtype, int flags);
int plan_destroy(Plan *P);
int plan_exec(const Plan *P, void *data, void *stream, bool forward);
int plan_exec_ex(const Plan *P, void *data, void *stream, bool forward, double scale, int dealias);
int plan_exec_pass(const Plan *P, void *data, void *stream, int pass, bool forward);
int plan_launches(const Plan *P);
// Slab decomposition: whether P's Pass A has exchange-layout kernels, and a
// Pass A whose y columns write (forward) or read (inverse) the all-to-all's
// layout in `xch` -- chunk y / nyl, element (x * nyl + y % nyl) * Nh + kz --
// instead of the field
bool plan_has_xch(const Plan *P);
int plan_exec_pass_a_xch(const Plan *P, void *data, void *xch, int nyl, long long chunk, void *stream, bool forward);
int plan_describe(const Plan *P, char *buf, int len);
int plan_autotune(Plan *P, void *scratch, void *stream);
// P takes Q's kernel choice (same grid, precision and form; Q tuned already)
int plan_adopt(Plan *P, const Plan *Q);
int wisdom_save(const char *path);
int wisdom_load(const char *path);

}  // namespace gpufft
