// axis.cu — plans and launches of the one-axis-per-launch kernels
// (fft_axis.cuh): the general path, taken by every pass that has no entry in
// the registry of specialised kernels (gpufft.cu) and whose lengths they take.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "../../include/gpufft_b200.h"
#include "fft_axis.cuh"
#include "gpufft_internal.h"

namespace gpufft {
namespace axis {

#define GPUFFT_AXIS_PARTS(X) X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7)
#define GPUFFT_AXIS_DECLARE(i) extern const FixedTable kFixed_f32_##i, kFixed_f64_##i;
GPUFFT_AXIS_PARTS(GPUFFT_AXIS_DECLARE)
#define GPUFFT_AXIS_F32(i) &kFixed_f32_##i,
#define GPUFFT_AXIS_F64(i) &kFixed_f64_##i,
static const FixedTable *const kFixed_f32[] = {GPUFFT_AXIS_PARTS(GPUFFT_AXIS_F32)};
static const FixedTable *const kFixed_f64[] = {GPUFFT_AXIS_PARTS(GPUFFT_AXIS_F64)};

// the kernels of length n, or null
static const Fixed *fixed_length(int dtype, int n) {
    for (const FixedTable *t : dtype == GPUFFT_FLOAT ? kFixed_f32 : kFixed_f64)
        for (int i = 0; i < t->count; ++i)
            if (t->lengths[i].n == n) return &t->lengths[i];
    return nullptr;
}

static const int kRadices[] = {2,  3,  4,  5,  6,  7,  8,  9,  10, 11, 12, 13, 14,
                               15, 16, 18, 20, 21, 22, 24, 25, 26, 27, 28, 30, 32};
static int hold(int r) { return r <= 12 ? 2 : 1; }  // Hold<R, Stage>

// threads for `radices` of length n on tiles of w sequences
static int threads(int n, int w, const std::vector<int> &radices) {
    int t = 0;
    for (int r : radices) t = std::max(t, (n / r + hold(r) - 1) / hold(r) * w);
    return (t + 31) / 32 * 32;
}

// The radices of a length without kernels of its own (factors of 11 and 13,
// and what needs three stages): two stages, as equal as possible (fewest
// registers and threads), in the first class that has the radices and the
// threads; else three stages of the last class with the fewest threads.
static bool choose(int n, const Kernel *table, std::vector<int> &radices, const Kernel *&k, int &nt) {
    for (int c = 0; c + 1 < kClasses; ++c) {
        int best = 0;
        for (int a : kRadices)
            for (int b : kRadices)
                if (a * b == n && a <= b && b <= table[c].rmax && (!best || b < best)) {
                    const std::vector<int> r = {b, a};
                    const int t = threads(n, table[c].w, r);
                    if (t > table[c].nt) continue;
                    best = b;
                    radices = r;
                    nt = t;
                    k = &table[c];
                }
        if (best) return true;
    }
    const Kernel &last = table[kClasses - 1];
    int best = last.nt + 1;
    for (int a : kRadices)
        for (int b : kRadices)
            for (int c : kRadices)
                if (a <= b && b <= c && c <= last.rmax && a * b * c == n) {
                    const std::vector<int> r = {c, b, a};
                    const int t = threads(n, last.w, r);
                    if (t < best) {
                        best = t;
                        radices = r;
                        nt = t;
                        k = &last;
                    }
                }
    return best <= last.nt;
}

static void fill(Axis &ax, int n, const std::vector<int> &radices) {
    ax.n = n;
    ax.nst = (int)radices.size();
    int p = 1, off = 0;
    for (int s = 0; s < ax.nst; ++s) {
        const int r = radices[s];
        ax.st[s] = {r, p, n / r, off, make_fastdiv((uint32_t)p)};
        off += (r - 1) * p;
        p *= r;
    }
}

// exp(-2 pi i j k / (p r)) at off + (j - 1) p + k, in long double, rounded once
template <typename T>
static void stage_table(std::vector<unsigned char> &out, const Axis &ax) {
    const size_t at = out.size();
    out.resize(at + (size_t)ax.n * 2 * sizeof(T));
    T *t = reinterpret_cast<T *>(out.data() + at);
    const long double two_pi = 6.283185307179586476925286766559005768L;
    for (int s = 0; s < ax.nst; ++s) {
        const Stage &st = ax.st[s];
        for (int j = 1; j < st.r; ++j)
            for (int k = 0; k < st.p; ++k) {
                const long double ang = two_pi * (long double)((long long)j * k % (st.p * st.r)) / (long double)(st.p * st.r);
                const size_t e = 2 * ((size_t)st.off + (size_t)(j - 1) * st.p + k);
                t[e] = (T)cosl(ang);
                t[e + 1] = (T)(-sinl(ang));
            }
    }
    t[2 * (ax.n - 1)] = t[2 * (ax.n - 1) + 1] = (T)0;
}

struct Launch {
    const void *fn[2][2] = {};  // [forward][epilogue]
    Axis ax{};
    int w = 0, nt = 0, nbuf = 0, ntiles = 0, grid = 0;
    size_t smem = 0, table = 0;  // table: byte offset into Form::dev
    bool fixed = false;
};

struct Form {
    void *dev = nullptr;
    size_t unp = 0;  // byte offset of the rows' unpack factors, then the pack factors (RowParams)
    Launch x, y, z;
    bool has_a = false, has_b = false;
};

// Shared memory and grid of a launch; false where one tile does not fit.  Two
// tile buffers, so that one fills while the other is transformed, unless one
// buffer lets more CTAs run: 384^2 x 480 FP32 x axis 99 against 114 us, 320^3
// FP64 x axis 95 against 111; with the same CTAs either way two buffers win
// (512^3 FP32 x axis 200 against 246, 500^3 220 against 244).
static bool size_launch(Launch &L, size_t fixed, size_t tile, int sms, int limit) {
    const size_t least = fixed + tile;
    if (least > (size_t)limit) return false;
    const size_t most = fixed + 2 * tile <= (size_t)limit ? fixed + 2 * tile : least;
    for (const auto &fns : L.fn)
        for (const void *fn : fns)
            if (fn && raise_smem_limit(fn, most) != cudaSuccess) {
                cudaGetLastError();
                return false;
            }
    int occ1 = 0, occ2 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ1, L.fn[1][0], L.nt, least);
    if (most > least) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ2, L.fn[1][0], L.nt, most);
    if (occ1 < 1) return false;
    L.nbuf = occ2 >= occ1 ? 2 : 1;
    L.smem = L.nbuf == 2 ? most : least;
    L.grid = std::min(L.ntiles, (L.nbuf == 2 ? occ2 : occ1) * sms);
    return true;
}

template <typename T>
static int build(Plan &P, Form &F, const Kernel *cols, const Kernel *cols_epi, const Kernel *rows) {
    using V = cx_t<T>;
    const int nx = (int)P.nx, ny = (int)P.ny, m = (int)(P.nz / 2), nh = m + 1;
    int sms = 1, limit = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, P.device);
    cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, P.device);
    if (limit <= 0) limit = 227 * 1024;
    std::vector<unsigned char> tab;
    const long long nrows = (long long)nx * ny, ycols = (long long)nx * nh, xcols = (long long)ny * nh;
    const long long most = (1LL << 31) - 64;
    // tiles of `groups` groups of gcols columns (ColParams)
    // radices, kernels and threads of length n
    auto kernels = [&](Launch &L, int n, bool col) {
        const Fixed *fx = fixed_length(P.dtype, n);
        std::vector<int> r;
        if (fx && (col || fx->rows[0])) {
            for (int f = 0; f < 2; ++f)
                for (int e = 0; e < 2; ++e) L.fn[f][e] = col ? fx->cols[f][e] : e ? nullptr : fx->rows[f];
            L.w = Width<T>::value;
            L.nt = fx->nt;
            r = {fx->r1, fx->r2};
            L.fixed = true;
        } else {
            const Kernel *k;
            if (n < 16 || !choose(n, col ? cols : rows, r, k, L.nt)) return false;
            L.fn[0][0] = k->inv;
            L.fn[1][0] = k->fwd;
            if (col) {
                L.fn[0][1] = cols_epi[k - cols].inv;
                L.fn[1][1] = cols_epi[k - cols].fwd;
            }
            L.w = k->w;
        }
        fill(L.ax, n, r);
        return true;
    };
    // tiles of `groups` groups of gcols columns (ColParams)
    auto columns = [&](Launch &L, int n, int groups, int gcols, long long pitch) {
        if (n / 2 * pitch >= 1LL << 32 || !kernels(L, n, true)) return false;  // (ColOut's 32-bit step)
        L.ntiles = groups * (gcols / L.w) + (groups * (gcols % L.w) + L.w - 1) / L.w;
        const size_t fixed = (size_t)((n + 1) / 2 * 2) * sizeof(V);
        const size_t tile = (size_t)n * (L.w + (sizeof(V) == 8 && pitch % 2 ? 2 : 0)) * sizeof(V);
        if (!size_launch(L, fixed, tile, sms, limit)) return false;
        L.table = tab.size();
        stage_table<T>(tab, L.ax);
        return true;
    };
    if (xcols < most) F.has_b = columns(F.x, nx, 1, (int)xcols, xcols);
    if (ycols < most && nrows < most && columns(F.y, ny, nx, nh, nh) && kernels(F.z, m, false)) {
        Launch &L = F.z;
        L.ntiles = (int)((nrows + L.w - 1) / L.w);
        const int half = m / 2 + 1;
        if (size_launch(L, (size_t)((half + m + 1) / 2 * 2) * sizeof(V),
                        (size_t)((nh * (L.w + 1) + 1) / 2 * 2) * sizeof(V), sms, limit)) {
            L.table = tab.size();
            stage_table<T>(tab, L.ax);
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
            F.has_a = true;
        }
    }
    if (!F.has_a && !F.has_b) return GPUFFT_SUCCESS;
    cudaError_t e = cudaMalloc(&F.dev, tab.size());
    if (e != cudaSuccess) {
        F.dev = nullptr;
        return set_error(GPUFFT_ERR_OOM, "cudaMalloc axis tables: %s", cudaGetErrorString(e));
    }
    e = cudaMemcpy(F.dev, tab.data(), tab.size(), cudaMemcpyHostToDevice);
    return e == cudaSuccess ? GPUFFT_SUCCESS
                            : set_error(GPUFFT_ERR_CUDA, "upload axis tables: %s", cudaGetErrorString(e));
}

int form_create(Plan &P) {
    if (P.axis) return GPUFFT_SUCCESS;
    P.axis = new Form();
    return P.dtype == GPUFFT_FLOAT ? build<float>(P, *P.axis, kCols_f32, kColsEpi_f32, kRows_f32)
                                   : build<double>(P, *P.axis, kCols_f64, kColsEpi_f64, kRows_f64);
}

void form_destroy(Plan &P) {
    if (!P.axis) return;
    if (P.axis->dev) cudaFree(P.axis->dev);
    delete P.axis;
    P.axis = nullptr;
}

bool has_a(const Plan &P) { return P.axis && P.axis->has_a; }
bool has_b(const Plan &P) { return P.axis && P.axis->has_b; }

static int launch_cols(const Plan &P, const Launch &L, void *data, cudaStream_t s, bool fwd, long long pitch,
                       long long gstride, int groups, int gcols, double scale, int dealias) {
    ColParams c{};
    c.data = data;
    c.tw = (const char *)P.axis->dev + L.table;
    c.ax = L.ax;
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
    if (P.dtype == GPUFFT_FLOAT) {
        // rows of a whole tile start at an even element of the field, or every other one at an odd element
        const int base = (uintptr_t)data % 16 ? 1 : 0;
        c.copy = base ? 0 : pitch % 2 ? 2 : gstride % 2 ? 0 : 1;
        c.gpar = (int)(gstride % 2);
    }
    c.dealias = dealias;
    c.scale = scale;
    c.ny = (int)P.ny;
    c.nz = (int)P.nz;
    c.nh = (int)(P.nz / 2 + 1);
    const bool epi = scale != 1.0 || dealias;
    void *args[] = {&c};
    const cudaError_t e = cudaLaunchKernel(L.fn[fwd][epi], dim3(L.grid), dim3(L.nt), args, L.smem, s);
    return e == cudaSuccess ? GPUFFT_SUCCESS : set_error(GPUFFT_ERR_CUDA, "launch axis columns: %s", cudaGetErrorString(e));
}

static int launch_rows(const Plan &P, const Launch &L, void *data, cudaStream_t s, bool fwd) {
    const int m = (int)(P.nz / 2);
    RowParams p{};
    p.data = data;
    p.tw = (const char *)P.axis->dev + L.table;
    const size_t vs = P.dtype == GPUFFT_FLOAT ? sizeof(float2) : sizeof(double2);
    p.unp = (const char *)P.axis->dev + P.axis->unp + (fwd ? 0 : (size_t)(m / 2 + 1) * vs);
    p.ax = L.ax;
    p.nrows = (int)(P.nx * P.ny);
    p.nh = m + 1;
    p.half = m / 2 + 1;
    p.aligned = (uintptr_t)data % 16 == 0;
    p.ntiles = L.ntiles;
    p.nbuf = L.nbuf;
    void *args[] = {&p};
    const cudaError_t e = cudaLaunchKernel(L.fn[fwd][0], dim3(L.grid), dim3(L.nt), args, L.smem, s);
    return e == cudaSuccess ? GPUFFT_SUCCESS : set_error(GPUFFT_ERR_CUDA, "launch axis rows: %s", cudaGetErrorString(e));
}

int launch_a(const Plan &P, void *data, cudaStream_t s, bool fwd) {
    const Form &F = *P.axis;
    const int nh = (int)(P.nz / 2 + 1);
    int rc = GPUFFT_SUCCESS;
    if (fwd) rc = launch_rows(P, F.z, data, s, true);
    if (rc == GPUFFT_SUCCESS)
        rc = launch_cols(P, F.y, data, s, fwd, nh, P.ny * nh, (int)P.nx, nh, 1.0, 0);
    if (!fwd && rc == GPUFFT_SUCCESS) rc = launch_rows(P, F.z, data, s, false);
    return rc;
}

int launch_b(const Plan &P, void *data, cudaStream_t s, bool fwd, double scale, int dealias) {
    const int ncols = (int)(P.ny * (P.nz / 2 + 1));
    return launch_cols(P, P.axis->x, data, s, fwd, ncols, 0, 1, ncols, scale, dealias);
}

static void describe(std::string &out, const char *name, const Launch &L) {
    char b[160];
    int n = snprintf(b, sizeof(b), " %s{n=%d[", name, L.ax.n);
    for (int s = 0; s < L.ax.nst; ++s) n += snprintf(b + n, sizeof(b) - n, "%s%d", s ? "x" : "", L.ax.st[s].r);
    snprintf(b + n, sizeof(b) - n, "] fixed=%d w=%d nt=%d grid=%d nbuf=%d smem=%zu}", L.fixed, L.w, L.nt,
             L.grid, L.nbuf, L.smem);
    out += b;
}

void form_describe(const Plan &P, std::string &out, bool a, bool b) {
    if (a && has_a(P)) {
        describe(out, "axisZ", P.axis->z);
        describe(out, "axisY", P.axis->y);
    }
    if (b && has_b(P)) describe(out, "axisX", P.axis->x);
}

}  // namespace axis
}  // namespace gpufft
