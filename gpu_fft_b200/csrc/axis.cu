// axis.cu — plans and launches of the one-axis-per-launch kernels
// (fft_axis.cuh): taken by every pass whose lengths they take and that has no
// entry in the registry of specialised kernels or is faster on these (the rule
// of prefer_axis_a and prefer_axis_b in gpufft.cu).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "../../include/gpufft_b200.h"
#include "fft_axis.cuh"
#include "gpufft_internal.h"

namespace gpufft {
namespace axis {

#define GPUFFT_AXIS_PARTS(X) \
    X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) \
    X(16) X(17) X(18) X(19) X(20) X(21) X(22) X(23) X(24) X(25) X(26) X(27) X(28) X(29) X(30) X(31) \
    X(32) X(33) X(34) X(35) X(36) X(37) X(38) X(39) X(40) X(41) X(42) X(43) X(44) X(45) X(46) X(47) \
    X(48) X(49) X(50) X(51) X(52) X(53) X(54) X(55) X(56) X(57) X(58) X(59) X(60) X(61) X(62) X(63)
#define GPUFFT_AXIS_DECLARE(i) extern const KernelTable kKernels_f32_##i, kKernels_f64_##i;
GPUFFT_AXIS_PARTS(GPUFFT_AXIS_DECLARE)
#define GPUFFT_AXIS_F32(i) &kKernels_f32_##i,
#define GPUFFT_AXIS_F64(i) &kKernels_f64_##i,
static const KernelTable *const kKernels_f32[] = {GPUFFT_AXIS_PARTS(GPUFFT_AXIS_F32)};
static const KernelTable *const kKernels_f64[] = {GPUFFT_AXIS_PARTS(GPUFFT_AXIS_F64)};

// the kernels of length n, or null
static const Kernels *kernels_of(int dtype, int n) {
    for (const KernelTable *t : dtype == GPUFFT_FLOAT ? kKernels_f32 : kKernels_f64)
        for (int i = 0; i < t->count; ++i)
            if (t->lengths[i].r[0] * t->lengths[i].r[1] * t->lengths[i].r[2] == n) return &t->lengths[i];
    return nullptr;
}

// Twiddles of the stages of length n, one after the other: stage of radix r
// after radices of product p, exp(-2 pi i j k / (p r)) at (j - 1) p + k; in long
// double, rounded once; n entries (the last unused).
template <typename T>
static void stage_table(std::vector<unsigned char> &out, int n, const int (&radices)[3]) {
    const size_t at = out.size();
    out.resize(at + (size_t)n * 2 * sizeof(T));
    T *t = reinterpret_cast<T *>(out.data() + at);
    const long double two_pi = 6.283185307179586476925286766559005768L;
    int p = 1;
    for (int r : radices) {
        for (int j = 1; j < r; ++j)
            for (int k = 0; k < p; ++k) {
                const long double ang = two_pi * (long double)((long long)j * k % (p * r)) / (long double)(p * r);
                *t++ = (T)cosl(ang);
                *t++ = (T)(-sinl(ang));
            }
        p *= r;
    }
    t[0] = t[1] = (T)0;
}

struct Launch {
    const void *fn[2] = {};  // [forward]
    const Kernels *k = nullptr;
    int n = 0, w = 0, nt = 0, nbuf = 0, ntiles = 0, grid = 0;
    int copy = 0, boxh = 0, nbox = 0, odd = 0, tile = 0;  // columns: ColParams
    size_t smem = 0, table = 0;  // table: byte offset into the part's tables
};

// the launches of one pass, its tables on the device
struct Part {
    bool made = false, has = false;  // made: form_create has been here; has: these lengths have kernels
    void *dev = nullptr;
    size_t bytes = 0;
};

struct Form {
    Part a, b;       // Pass A (z and y), x pass: each made when a plan first needs it
    size_t unp = 0;  // byte offset of the rows' unpack factors, then the pack factors (RowParams)
    Launch x, y, z;
    long long wait_ns = 2000000000LL;  // limit of the wait for a tile's copy: 2 s, far above any launch's length
    int missing_rows = 0, missing_cols = 0;  // RowParams, ColParams::missing
};

// Shared memory and grid of a launch; false where one tile does not fit.
// Columns: one tile buffer, refilled while the last stage computes, where two
// CTAs or more run on an SM (fractions of the copy bandwidth, FP32 x axis:
// 320 points 0.85 against 0.75 with two buffers, 384 0.84 against 0.74), two
// where only one CTA does (500 points 0.83 against 0.62).  Rows have no stage
// that writes global memory while a refill could run: two buffers while two
// CTAs still fit (m = 320: 0.86 against 0.75).
static bool size_launch(Launch &L, bool rows, size_t fixed, size_t tile, int sms, int limit) {
    fixed += 128 + 2 * sizeof(uint64_t);  // alignment of the buffers, a barrier each
    const size_t least = fixed + tile;
    if (least > (size_t)limit) return false;
    const size_t most = fixed + 2 * tile <= (size_t)limit ? fixed + 2 * tile : least;
    for (const void *fn : L.fn)
        if (raise_smem_limit(fn, most) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
    int occ1 = 0, occ2 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ1, L.fn[1], L.nt, least);
    if (most > least) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ2, L.fn[1], L.nt, most);
    if (occ1 < 1) return false;
    L.nbuf = occ2 >= (rows && occ1 >= 2 ? 2 : 1) && (rows || occ1 < 2) ? 2 : 1;
    L.smem = L.nbuf == 2 ? most : least;
    L.grid = std::min(L.ntiles, (L.nbuf == 2 ? occ2 : occ1) * sms);
    return true;
}

template <typename T>
static int build(Plan &P, Form &F, Part &part) {
    using V = cx_t<T>;
    const int nx = (int)P.nx, ny = (int)P.ny, m = (int)(P.nz / 2), nh = m + 1;
    int sms = 1, limit = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, P.device);
    cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, P.device);
    if (limit <= 0) limit = 227 * 1024;
    std::vector<unsigned char> tab;
    const long long nrows = (long long)nx * ny, ycols = (long long)nx * nh, xcols = (long long)ny * nh;
    const long long most = (1LL << 31) - 64;
    // kernels and threads of length n
    auto kernels = [&](Launch &L, int n, bool col) {
        L.k = kernels_of(P.dtype, n);
        if (!L.k || !(col ? L.k->cols : L.k->rows)[0]) return false;
        for (int f = 0; f < 2; ++f) L.fn[f] = (col ? L.k->cols : L.k->rows)[f];
        L.n = n;
        L.w = Width<T>::value;
        L.nt = L.k->nt;
        return true;
    };
    // tiles of `groups` groups of gcols columns (ColParams)
    auto columns = [&](Launch &L, int n, int groups, int gcols, long long pitch) {
        if (n / 2 * pitch >= 1LL << 32 || !kernels(L, n, true)) return false;  // (ColOut's 32-bit step)
        L.ntiles = groups * (gcols / L.w) + (groups * (gcols % L.w) + L.w - 1) / L.w;
        // equal boxes of at most 256 lines that start 128-byte aligned in shared memory (the last one may
        // reach past the tile's lines: the buffer has room for it)
        auto boxes = [&](int lines, int width) {
            const int row = width * (int)sizeof(V), align = 128 / std::min(128, row & -row);
            L.nbox = (lines + 255) / 256;
            L.boxh = (lines + L.nbox - 1) / L.nbox;
            if (L.nbox > 1) L.boxh = (L.boxh + align - 1) / align * align;
        };
        if (sizeof(V) == 8 && pitch % 2) {
            // two rows as one line where rows pair up inside a group
            boxes((n + 1) / 2, L.w + 2);
            L.copy = n % 2 == 0 ? 3 : 2;
            L.odd = (L.nbox * L.boxh * (L.w + 2) + 15) / 16 * 16;
            L.tile = L.odd + L.nbox * L.boxh * (L.w + 2);
        } else {
            boxes(n, L.w);
            L.copy = 1;
            L.tile = L.nbox * L.boxh * L.w;
        }
        L.tile = (std::max(L.tile, n * L.w) + 15) / 16 * 16;
        const size_t fixed = col_table_bytes<V>(n), tile = (size_t)L.tile * sizeof(V);
        if (!size_launch(L, false, fixed, tile, sms, limit)) return false;
        L.table = tab.size();
        stage_table<T>(tab, L.n, L.k->r);
        return true;
    };
    bool has = false;
    if (&part == &F.b)
        has = xcols < most && columns(F.x, nx, 1, (int)xcols, xcols);
    else if (ycols < most && nrows < most && columns(F.y, ny, nx, nh, nh) && kernels(F.z, m, false)) {
        Launch &L = F.z;
        L.ntiles = (int)((nrows + L.w - 1) / L.w);
        const int half = m / 2 + 1;
        if (size_launch(L, true, (size_t)((half + m + 1) / 2 * 2) * sizeof(V),
                        (size_t)row_tile<V>(m, L.w) * sizeof(V), sms, limit)) {
            L.table = tab.size();
            stage_table<T>(tab, L.n, L.k->r);
            F.unp = tab.size();
            tab.resize(F.unp + 2 * (size_t)half * sizeof(V));
            T *u = reinterpret_cast<T *>(tab.data() + F.unp);
            const long double two_pi = 6.283185307179586476925286766559005768L;
            for (int k = 0; k < half; ++k) {
                const long double ang = two_pi * (long double)k / (long double)(2 * m);
                const long double c = cosl(ang), sn = sinl(ang);  // w^k = c - i sn
                u[2 * k] = (T)(-sn / 2);
                u[2 * k + 1] = (T)(-c / 2);
                u[2 * (half + k)] = (T)(-sn);
                u[2 * (half + k) + 1] = (T)c;
            }
            has = true;
        }
    }
    if (!has) return GPUFFT_SUCCESS;
    cudaError_t e = cudaMalloc(&part.dev, tab.size());
    if (e != cudaSuccess) {
        part.dev = nullptr;
        return set_error(GPUFFT_ERR_OOM, "cudaMalloc axis tables: %s", cudaGetErrorString(e));
    }
    e = cudaMemcpy(part.dev, tab.data(), tab.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return set_error(GPUFFT_ERR_CUDA, "upload axis tables: %s", cudaGetErrorString(e));
    part.bytes = tab.size();
    part.has = true;
    return GPUFFT_SUCCESS;
}

int form_create(Plan &P, bool a, bool b) {
    if (P.axis) {
        a = a && !P.axis->a.made;
        b = b && !P.axis->b.made;
    }
    if (!a && !b) return GPUFFT_SUCCESS;
    if (!P.axis) P.axis = new (std::nothrow) Form();
    if (!P.axis) return set_error(GPUFFT_ERR_OOM, "host allocation failed");
    // test hooks of the bounded wait: with GPUFFT_AXIS_UNREACHABLE at plan creation the row tiles (1), the column
    // tiles (2) or both (3) wait for 16 bytes more than their copies bring, so the wait runs out, after
    // GPUFFT_AXIS_WAIT_MS, and gpufft_plan_check reports it
    if (const char *ev = std::getenv("GPUFFT_AXIS_UNREACHABLE")) {
        const int which = std::atoi(ev);
        P.axis->missing_rows = which & 1 ? 16 : 0;
        P.axis->missing_cols = which & 2 ? 16 : 0;
    }
    if (const char *ev = std::getenv("GPUFFT_AXIS_WAIT_MS")) P.axis->wait_ns = 1000000LL * std::max(1, std::atoi(ev));
    int rc = GPUFFT_SUCCESS;
    for (Part *part : {a ? &P.axis->a : nullptr, b ? &P.axis->b : nullptr}) {
        if (!part || rc != GPUFFT_SUCCESS) continue;
        part->made = true;
        rc = P.dtype == GPUFFT_FLOAT ? build<float>(P, *P.axis, *part) : build<double>(P, *P.axis, *part);
    }
    return rc;
}

void form_destroy(Plan &P) {
    if (!P.axis) return;
    for (Part *part : {&P.axis->a, &P.axis->b})
        if (part->dev) cudaFree(part->dev);
    delete P.axis;
    P.axis = nullptr;
}

bool has_a(const Plan &P) { return P.axis && P.axis->a.has; }
bool has_b(const Plan &P) { return P.axis && P.axis->b.has; }

static cudaError_t launch(const Launch &L, bool fwd, void **args, cudaStream_t s, bool chained) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(L.grid);
    cfg.blockDim = dim3(L.nt);
    cfg.dynamicSmemBytes = L.smem;
    cfg.stream = s;
    cfg.attrs = attr;
    if (chained) attr[cfg.numAttrs++] = dependent_launch();
    return cudaLaunchKernelExC(&cfg, L.fn[fwd], args);
}

static int launch_cols(const Plan &P, const Part &part, const Launch &L, void *data, cudaStream_t s, bool fwd, long long pitch,
                       long long gstride, int groups, int gcols, double scale, int dealias, bool chained) {
    ColParams c{};
    c.data = data;
    c.tw = (const char *)part.dev + L.table;
    c.pitch = pitch;
    c.gstride = gstride;
    c.gcols = gcols;
    c.full = gcols / L.w;
    c.rem = gcols % L.w;
    c.fulldiv = make_fastdiv((uint32_t)std::max(c.full, 1));
    c.remdiv = make_fastdiv((uint32_t)std::max(c.rem, 1));
    c.nfull = groups * c.full;
    c.nrem = groups * c.rem;
    c.ntiles = L.ntiles;
    c.nbuf = L.nbuf;
    c.copy = L.copy;
    c.boxh = L.boxh;
    c.nbox = L.nbox;
    c.odd = L.odd;
    c.tile = L.tile;
    c.gpar = L.copy == 2 ? (int)(gstride % 2) : 0;
    c.err = P.pb.err;
    c.wait_ns = P.axis->wait_ns;
    c.missing = P.axis->missing_cols;
    if ((uintptr_t)data % 16) c.copy = 0;
    CUtensorMap tm{};
    if (c.copy == 1) {
        const int e8 = P.dtype == GPUFFT_FLOAT ? 1 : 2;  // 8-byte elements per complex
        if (!encode_view(&tm, data, (long long)gcols * e8, (long long)groups * L.n, pitch * 8 * e8, L.w * e8, L.boxh))
            c.copy = 0;
    } else if (c.copy == 3) {
        if (!encode_view(&tm, data, 2 * pitch, (long long)groups * L.n / 2, 2 * pitch * 8, L.w + 2, L.boxh)) c.copy = 2;
    }
    c.dealias = dealias;
    c.scale = scale;
    c.ny = (int)P.ny;
    c.nz = (int)P.nz;
    c.nh = (int)(P.nz / 2 + 1);
    c.epi = scale != 1.0 || dealias;
    void *args[] = {&c, &tm};
    const cudaError_t e = launch(L, fwd, args, s, chained);
    return e == cudaSuccess ? GPUFFT_SUCCESS : set_error(GPUFFT_ERR_CUDA, "launch axis columns: %s", cudaGetErrorString(e));
}

static int launch_rows(const Plan &P, const Launch &L, void *data, cudaStream_t s, bool fwd, bool chained) {
    const int m = (int)(P.nz / 2);
    RowParams p{};
    p.data = data;
    p.tw = (const char *)P.axis->a.dev + L.table;
    const size_t vs = P.dtype == GPUFFT_FLOAT ? sizeof(float2) : sizeof(double2);
    p.unp = (const char *)P.axis->a.dev + P.axis->unp + (fwd ? 0 : (size_t)(m / 2 + 1) * vs);
    p.nrows = (int)(P.nx * P.ny);
    p.aligned = (uintptr_t)data % 16 == 0;
    p.ntiles = L.ntiles;
    p.nbuf = L.nbuf;
    p.err = P.pb.err;
    p.wait_ns = P.axis->wait_ns;
    p.missing = P.axis->missing_rows;
    void *args[] = {&p};
    const cudaError_t e = launch(L, fwd, args, s, chained);
    return e == cudaSuccess ? GPUFFT_SUCCESS : set_error(GPUFFT_ERR_CUDA, "launch axis rows: %s", cudaGetErrorString(e));
}

int launch_a(const Plan &P, void *data, cudaStream_t s, bool fwd, bool chained) {
    const Form &F = *P.axis;
    const int nh = (int)(P.nz / 2 + 1);
    int rc = GPUFFT_SUCCESS;
    if (fwd) rc = launch_rows(P, F.z, data, s, true, chained);
    if (rc == GPUFFT_SUCCESS)
        rc = launch_cols(P, F.a, F.y, data, s, fwd, nh, P.ny * nh, (int)P.nx, nh, 1.0, 0, fwd ? chain_inside(P) : chained);
    if (!fwd && rc == GPUFFT_SUCCESS) rc = launch_rows(P, F.z, data, s, false, chain_inside(P));
    return rc;
}

int launch_b(const Plan &P, void *data, cudaStream_t s, bool fwd, double scale, int dealias, bool chained) {
    const int ncols = (int)(P.ny * (P.nz / 2 + 1));
    return launch_cols(P, P.axis->b, P.axis->x, data, s, fwd, ncols, 0, 1, ncols, scale, dealias, chained);
}

static void describe(std::string &out, const char *name, const Launch &L) {
    char b[160];
    snprintf(b, sizeof(b), " %s{n=%d[%dx%dx%d] nt=%d grid=%d nbuf=%d smem=%zu}", name, L.n, L.k->r[0], L.k->r[1], L.k->r[2],
             L.nt, L.grid, L.nbuf, L.smem);
    out += b;
}

void form_describe(const Plan &P, std::string &out, bool a, bool b) {
    if (a && has_a(P)) {
        describe(out, "axisZ", P.axis->z);
        describe(out, "axisY", P.axis->y);
    }
    if (b && has_b(P)) describe(out, "axisX", P.axis->x);
    if (has_a(P) || has_b(P)) out += " axisTables=" + std::to_string(P.axis->a.bytes + P.axis->b.bytes);
}

}  // namespace axis
}  // namespace gpufft
