// fft_axis.cuh — one axis of the transform per launch, for any axis length
// from 16 up that is a product of two radices of at most 32 or three of at
// most 16.
//
// The cluster-per-plane kernels of fft_kernels.cuh take any length, but they
// walk it in three to six radix stages with run-time strides, one butterfly
// at a time, and spend 130 (x axis) to 320 (z and y axes) instructions per
// element: at 200 x 378 x 500 FP32 they issue on 54-60% of all cycles and
// move 14% (z and y) and 32% (x) of the copy bandwidth.  Here
//  * a length up to 1024 is in almost every case R1 * R2 with R1, R2 <= 32
//    (every product of 2s, 3s and 5s but 972 and 1000): two passes over
//    shared memory, the rest three;
//  * the lengths of axis_lengths.h have kernels of their own, radices and
//    strides as constants (about 50 instructions per element and axis,
//    against 62 to 112 with them at run time, and registers that fit the
//    radices); the others share kernels with one switch over the radices;
//  * a thread keeps its butterflies in registers, so a stage works in place;
//  * a tile is W sequences, element (i, w) at i * PW + w: a half-warp reads
//    and writes W adjacent elements (128 bytes) whatever the radix, so no
//    stage has bank conflicts.  Rows (z) use PW = W + 1, which makes their
//    turning over conflict-free too;
//  * the next tile is copied in by cp.async while the current one is
//    transformed.
// z and y run as two launches, so the field crosses HBM three times per
// transform instead of twice (from L2 when it fits there); what that costs is
// less than what the instructions saved bring: R2C + C2R of 420 x 378 x 500
// FP32 2.01 -> 0.83 ms, 768^3 12.4 -> 5.0, 225 x 243 x 350 FP64 0.86 -> 0.42.
// Each launch moves 0.65-0.8 of the copy bandwidth; issue slots are 40% used
// and no pipe is over 55%: what is left is waiting at the block barriers
// between a stage's bursts of shared-memory accesses and its arithmetic.
#pragma once
#include "fft_fast.cuh"
#include "fft_radix.cuh"

namespace gpufft {
namespace axis {

constexpr int kMaxStages = 3;

struct Stage {
    int r;       // radix
    int p;       // product of the radices before it
    int nb;      // butterflies, n / r
    int off;     // first entry of its twiddles, exp(-2 pi i j k / (p r)) at off + (j - 1) * p + k
    FastDiv pd;  // division by p
};
struct Axis {
    int n, nst;
    Stage st[kMaxStages];
};
__device__ __forceinline__ int divp(const Stage &s, int i) { return (int)fdiv((uint32_t)i, s.pd); }

// the same as constants: stage 0 or 1 of n = R1 * R2 with NT threads on W sequences
template <int R, int P, int NB, int OFF, int G> struct FixedStage {
    static constexpr int r = R, p = P, nb = NB, off = OFF, c = (NB + G - 1) / G;
};
template <int R, int P, int NB, int OFF, int G>
__device__ __forceinline__ int divp(const FixedStage<R, P, NB, OFF, G> &, int i) {
    return i / P;
}

// Columns: groups of gcols adjacent sequences, group g at data + g * gstride,
// consecutive elements of a sequence `pitch` apart.  A group is cut into
// full = gcols / W whole tiles; the columns left over (rem of each group, 1 of
// 2^k + 1 for the y axis) are gathered from several groups into tiles of their
// own, so that no tile is mostly empty.
struct ColParams {
    void *data;
    const void *tw;
    Axis ax;
    long long pitch, gstride;
    int gcols, full, rem;
    FastDiv fulldiv, remdiv;
    int nfull, nrem;  // whole tiles of all groups, left-over columns of all groups
    int ntiles, nbuf;
    // How whole tiles are copied in.  0: element by element.  1 (FP32, rows
    // 16-byte aligned): column pairs.  2 (FP32, odd pitch: every other row
    // starts 8 bytes off): pairs from the 16-byte boundary at or before the
    // row's first column into rows of W + 2, where that column is at slot 0
    // or 1.  (8-byte cp.async allocates lines in L1: with 25 KB of it left
    // beside the tiles the y axis took 103 us where the x axis took 80.)
    int copy;
    int gpar;  // copy 2: row r of group g is off by 8 bytes where r + gpar * g is odd
    // x-pass epilogue (the EPI kernels; PassBParams): scale, and the 2/3-rule mask of column ky * nh + kz
    int dealias, ny, nh, nz;
    double scale;
};

// rows: nrows sequences of m complex, row r at data + r * nh (nh = m + 1)
struct RowParams {
    void *data;
    const void *tw;
    const void *unp;  // forward -i w^k / 2, inverse i conj(w^k), w = exp(-2 pi i / (2 m)), k <= m / 2
    Axis ax;
    int nrows, nh, half;  // half = m / 2 + 1
    int ntiles, nbuf;
    int aligned;  // data 16-byte aligned
};

// sequences per tile for which a tile row is 128 bytes
template <typename T> struct Width;
template <> struct Width<float> { static constexpr int value = 16; };
template <> struct Width<double> { static constexpr int value = 8; };

// butterflies of radix R that one thread holds: with run-time lengths two of
// the small radices, so that three-stage lengths fit a block
template <int R, class S> struct Hold { static constexpr int value = S::c; };
template <int R> struct Hold<R, Stage> { static constexpr int value = R <= 12 ? 2 : 1; };

// A thread's view of a tile.  The stage's inputs are at in_n * n + in_w * w,
// plus one where (n + par) is odd if `odd` is set (copy 2 above).
template <typename T> struct Ctx {
    using V = cx_t<T>;
    V *sm;
    const V *tw;
    int w, i0, g;  // this thread's sequence, first butterfly and butterfly step
    int in_n, in_w, odd, par;
};

// One stage in place in shared memory, its results in the layout n * PW + w,
// or handed to out.put (the last stage of a column).  `freed` runs once every
// thread has read its inputs.
template <typename T, int R, bool FWD, int PW, bool TO_OUT, class S, class Out, class Freed>
__device__ __forceinline__ void stage(const Ctx<T> &c, const S &s, Out &out, Freed &freed) {
    using V = cx_t<T>;
    constexpr int C = Hold<R, S>::value;
    V v[C][R];
    const int in_step = s.nb * c.in_n;
#pragma unroll
    for (int m = 0; m < C; ++m) {
        const int i = c.i0 + m * c.g;
        if (i < s.nb) {
            const int off = (i + c.par) & c.odd;
            const V *in = c.sm + i * c.in_n + c.w * c.in_w;
            const V *even = in + off, *odd = in + (off ^ (s.nb & c.odd));  // of even and odd j
#pragma unroll
            for (int j = 0; j < R; ++j) v[m][j] = (j & 1 ? odd : even)[j * in_step];
        } else {
            // (left undefined, every radix's registers would stay alive through the tile loop: 4 to 45 KB of spills)
#pragma unroll
            for (int j = 0; j < R; ++j) v[m][j] = V{(T)0, (T)0};
        }
    }
    __syncthreads();
    if constexpr (TO_OUT) freed();
#pragma unroll
    for (int m = 0; m < C; ++m) {
        const int i = c.i0 + m * c.g;
        if (i < s.nb) {
            const int ip = divp(s, i);
            const int k = i - ip * s.p;
            if (s.p > 1) {
                const V *tw = c.tw + s.off + k;
#pragma unroll
                for (int j = 1; j < R; ++j) v[m][j] = c_tw<FWD>(v[m][j], tw[(j - 1) * s.p]);
            }
            Dft<R, FWD, V>::run(v[m]);
            if constexpr (TO_OUT) {
                out.template put<R>(i, s.nb, v[m]);
            } else {
                V *o = c.sm + (ip * s.p * R + k) * PW + c.w;
                const int out_step = s.p * PW;
#pragma unroll
                for (int j = 0; j < R; ++j) o[j * out_step] = v[m][j];
            }
        }
    }
    if constexpr (!TO_OUT) __syncthreads();
}

// RMAX: the largest radix compiled in (16, 22 or 32): the register budget
template <typename T, int RMAX, bool FWD, int PW, bool TO_OUT, class Out, class Freed>
__device__ __forceinline__ void run_stage(const Ctx<T> &c, const Stage &s, Out &out, Freed &freed) {
#define GPUFFT_AXIS_RADIX(R)                                                                    \
    case R:                                                                                     \
        if constexpr (R <= RMAX) stage<T, R, FWD, PW, TO_OUT>(c, s, out, freed);                \
        break;
    switch (s.r) {
        GPUFFT_AXIS_RADIX(2)
        GPUFFT_AXIS_RADIX(3)
        GPUFFT_AXIS_RADIX(4)
        GPUFFT_AXIS_RADIX(5)
        GPUFFT_AXIS_RADIX(6)
        GPUFFT_AXIS_RADIX(7)
        GPUFFT_AXIS_RADIX(8)
        GPUFFT_AXIS_RADIX(9)
        GPUFFT_AXIS_RADIX(10)
        GPUFFT_AXIS_RADIX(11)
        GPUFFT_AXIS_RADIX(12)
        GPUFFT_AXIS_RADIX(13)
        GPUFFT_AXIS_RADIX(14)
        GPUFFT_AXIS_RADIX(15)
        GPUFFT_AXIS_RADIX(16)
        GPUFFT_AXIS_RADIX(18)
        GPUFFT_AXIS_RADIX(20)
        GPUFFT_AXIS_RADIX(21)
        GPUFFT_AXIS_RADIX(22)
        GPUFFT_AXIS_RADIX(24)
        GPUFFT_AXIS_RADIX(25)
        GPUFFT_AXIS_RADIX(26)
        GPUFFT_AXIS_RADIX(27)
        GPUFFT_AXIS_RADIX(28)
        GPUFFT_AXIS_RADIX(30)
        GPUFFT_AXIS_RADIX(32)
        default: break;  // the plan only emits the radices above, up to RMAX
    }
#undef GPUFFT_AXIS_RADIX
}

template <typename T, int RMAX, bool FWD, int PW, bool TO_OUT, int R, int P, int NB, int OFF, int G, class Out, class Freed>
__device__ __forceinline__ void run_stage(const Ctx<T> &c, const FixedStage<R, P, NB, OFF, G> &s, Out &out,
                                          Freed &freed) {
    stage<T, R, FWD, PW, TO_OUT>(c, s, out, freed);
}

// what a kernel knows of its axis: everything at run time, or two radices and
// the number of threads at compile time
template <int W_> struct AnyAxis {
    static constexpr int W = W_;
    static constexpr bool fixed = false;
    const Axis &ax;
    __device__ __forceinline__ int n() const { return ax.n; }
    __device__ __forceinline__ int nt() const { return blockDim.x; }
};
template <int W_, int R1, int R2, int NT> struct FixedAxis {
    static constexpr int W = W_;
    static constexpr bool fixed = true;
    const Axis &ax;
    using S0 = FixedStage<R1, 1, R2, 0, NT / W>;
    using S1 = FixedStage<R2, R1, R1, R1 - 1, NT / W>;
    __device__ __forceinline__ constexpr int n() const { return R1 * R2; }
    __device__ __forceinline__ constexpr int nt() const { return NT; }
};

struct NoOut {};
struct NoFreed {
    __device__ __forceinline__ void operator()() const {}
};

// where the last stage of a column puts its results: straight to global memory
template <typename T, bool EPI> struct ColOut {
    using V = cx_t<T>;
    V *base;  // this thread's column, or null past the last one
    long long pitch;
    bool drop;  // EPI: ky or kz outside the 2/3-rule box
    int nx, dealias;
    T scale;
    template <int R> __device__ __forceinline__ void put(int i, int nb, V *v) const {
        if (!base) return;
        V *o = base + (long long)i * pitch;
        const uint32_t step = (uint32_t)nb * (uint32_t)pitch;  // (fits: the plan checks n / 2 * pitch)
#pragma unroll
        for (int j = 0; j < R; ++j) {
            V x = v[j];
            if constexpr (EPI) {
                const int kx = i + j * nb;
                x = V{x.x * scale, x.y * scale};
                if (dealias && (drop || 3 * min(kx, nx - kx) > nx)) x = V{(T)0, (T)0};
            }
            st_g(o + (size_t)j * step, x);
        }
    }
};

template <typename T, int RMAX, bool FWD, bool EPI, class A>
__device__ __forceinline__ void cols_body(const ColParams &P, const A ax) {
    using V = cx_t<T>;
    constexpr int W = A::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = ax.n(), nt = ax.nt(), tid = threadIdx.x;
    V *tw = reinterpret_cast<V *>(smem_raw);  // n - 1 entries, padded to n rounded up to 16 bytes
    V *buf = tw + (n + 1) / 2 * 2;
    const int tile = n * (P.copy == 2 ? W + 2 : W);
    for (int q = tid; q < n - 1; q += nt) tw[q] = reinterpret_cast<const V *>(P.tw)[q];
    V *data = reinterpret_cast<V *>(P.data);
    // group and column of sequence w of tile t; false past the last one
    auto column = [&](int t, int w, int &g, int &c) -> bool {
        if (t < P.nfull) {
            g = (int)fdiv((uint32_t)t, P.fulldiv);
            c = (t - g * P.full) * W + w;
            return true;
        }
        const int q = (t - P.nfull) * W + w;
        g = (int)fdiv((uint32_t)q, P.remdiv);
        c = P.gcols - P.rem + q - g * P.rem;
        return q < P.nrem;
    };
    auto fetch = [&](int t, V *b) {
        int g, c;
        if (sizeof(V) == 8 && t < P.nfull && P.copy == 1) {
            const int w = (tid % (W / 2)) * 2, r0 = tid / (W / 2), rs = nt / (W / 2);
            column(t, w, g, c);
            const V *src = data + (long long)g * P.gstride + c + (long long)r0 * P.pitch;
            const long long step = (long long)rs * P.pitch;
            V *dst = b + r0 * W + w;
            for (int r = r0; r < n; r += rs, src += step, dst += rs * W) fast::cp_async16(dst, src, 16);
        } else if (sizeof(V) == 8 && t < P.nfull && P.copy == 2) {
            // 16 lanes a row, 8 chunks from the boundary plus one more where the row starts 8 bytes
            // before it; the row step is even, so a thread's rows are all of one kind
            constexpr int CH = W / 2;
            const int ch = tid % W, r0 = tid / W, rs = nt / W;
            column(t, 0, g, c);
            const int s = (r0 + P.gpar * g) & 1;
            if (ch < CH + s) {
                const V *src = data + (long long)g * P.gstride + c + (long long)r0 * P.pitch + (2 * ch - s);
                const long long step = (long long)rs * P.pitch;
                V *dst = b + r0 * (W + 2) + 2 * ch;
                const int bytes = ch < CH ? 16 : 8;  // (the last chunk's second element is another tile's, or past the field)
                for (int r = r0; r < n; r += rs, src += step, dst += rs * (W + 2)) fast::cp_async16(dst, src, bytes);
            }
        } else {
            const int w = tid % W, r0 = tid / W, rs = nt / W;
            if (column(t, w, g, c)) {
                const V *src = data + (long long)g * P.gstride + c + (long long)r0 * P.pitch;
                const long long step = (long long)rs * P.pitch;
                V *dst = b + r0 * W + w;
                for (int r = r0; r < n; r += rs, src += step, dst += rs * W) fast::cp_async_elem(dst, src, true);
            }
        }
    };
    const int grid = gridDim.x;
    for (int b = 0; b < P.nbuf; ++b) {
        const int t = blockIdx.x + b * grid;
        if (t < P.ntiles) fetch(t, buf + b * tile);
        fast::cp_async_commit();
    }
    int b = 0;
    for (int t = blockIdx.x; t < P.ntiles; t += grid) {
        if (P.nbuf == 2)
            fast::cp_async_wait<1>();
        else
            fast::cp_async_wait<0>();
        __syncthreads();
        V *cur = buf + b * tile;
        int g, col;
        const bool valid = column(t, tid % W, g, col);
        const bool shifted = sizeof(V) == 8 && t < P.nfull && P.copy == 2;
        Ctx<T> c{cur, tw, tid % W, tid / W, nt / W, shifted ? W + 2 : W, 1, shifted ? 1 : 0, P.gpar * g};
        if (A::fixed) c.in_n = W;
        NoOut none;
        NoFreed nothing;
        if constexpr (A::fixed) {
            // (both with the strides as constants)
            if (shifted) {
                Ctx<T> cs{cur, tw, tid % W, tid / W, nt / W, W + 2, 1, 1, c.par};
                run_stage<T, RMAX, FWD, W, false>(cs, typename A::S0(), none, nothing);
            } else {
                Ctx<T> cs{cur, tw, tid % W, tid / W, nt / W, W, 1, 0, 0};
                run_stage<T, RMAX, FWD, W, false>(cs, typename A::S0(), none, nothing);
            }
            c.in_n = W;
            c.odd = 0;
        } else {
            for (int s = 0; s + 1 < P.ax.nst; ++s) {
                run_stage<T, RMAX, FWD, W, false>(c, P.ax.st[s], none, nothing);
                c.in_n = W;
                c.odd = 0;
            }
        }
        ColOut<T, EPI> out;
        out.base = valid ? data + (long long)g * P.gstride + col : nullptr;
        out.pitch = P.pitch;
        if constexpr (EPI) {
            const int ky = col / P.nh, kz = col - ky * P.nh;
            out.drop = 3 * min(ky, P.ny - ky) > P.ny || 3 * kz > P.nz;
            out.nx = n;
            out.dealias = P.dealias;
            out.scale = (T)P.scale;
        }
        auto freed = [&]() {
            const int tn = t + P.nbuf * grid;
            if (tn < P.ntiles) fetch(tn, cur);
            fast::cp_async_commit();
        };
        if constexpr (A::fixed)
            run_stage<T, RMAX, FWD, W, true>(c, typename A::S1(), out, freed);
        else
            run_stage<T, RMAX, FWD, W, true>(c, P.ax.st[P.ax.nst - 1], out, freed);
        b = P.nbuf == 2 ? b ^ 1 : 0;
    }
}

template <typename T, int W, int RMAX, bool FWD, bool EPI, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) axis_cols(const __grid_constant__ ColParams P) {
    cols_body<T, RMAX, FWD, EPI>(P, AnyAxis<W>{P.ax});
}

// Rows.  A tile is W whole rows, one contiguous span of the field, copied in
// as it is (row w at w * nh: odd for most grids, so that reading W rows at
// one position is conflict-free); the first stage turns it over to n * PW + w.
template <typename T, int RMAX, bool FWD, class A>
__device__ __forceinline__ void rows_body(const RowParams &P, const A ax) {
    using V = cx_t<T>;
    constexpr int W = A::W, PW = W + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int m = ax.n(), nh = m + 1, half = m / 2 + 1, nt = ax.nt(), tid = threadIdx.x;
    V *unp = reinterpret_cast<V *>(smem_raw);      // half entries
    V *tw = unp + half;                            // m - 1 entries
    V *buf = unp + (half + m + 1) / 2 * 2;
    const int tile = (nh * PW + 1) / 2 * 2;
    for (int q = tid; q < half; q += nt) unp[q] = reinterpret_cast<const V *>(P.unp)[q];
    for (int q = tid; q < m - 1; q += nt) tw[q] = reinterpret_cast<const V *>(P.tw)[q];
    V *data = reinterpret_cast<V *>(P.data);
    auto fetch = [&](int t, V *b) {
        const int total = min(W, P.nrows - t * W) * nh;
        const V *src = data + (long long)t * W * nh;
        if (sizeof(V) == 8 && P.aligned) {
            for (int q = 2 * tid; q + 1 < total; q += 2 * nt) fast::cp_async16(b + q, src + q, 16);
            if (tid == 0 && total % 2) fast::cp_async_elem(b + total - 1, src + total - 1, true);
        } else {
            for (int q = tid; q < total; q += nt) fast::cp_async_elem(b + q, src + q, true);
        }
    };
    // bins k and m - k of one row at a time: `span` adjacent threads take a row
    const int span = min(nt, (half + 31) / 32 * 32), lanes = nt / span, k0 = tid % span, w0 = tid / span;
    const int grid = gridDim.x;
    for (int b = 0; b < P.nbuf; ++b) {
        const int t = blockIdx.x + b * grid;
        if (t < P.ntiles) fetch(t, buf + b * tile);
        fast::cp_async_commit();
    }
    const T hf = (T)0.5;
    int b = 0;
    for (int t = blockIdx.x; t < P.ntiles; t += grid) {
        if (P.nbuf == 2)
            fast::cp_async_wait<1>();
        else
            fast::cp_async_wait<0>();
        __syncthreads();
        V *cur = buf + b * tile;
        NoOut none;
        NoFreed nothing;
        const int rows = min(W, P.nrows - t * W);
        V *dst = data + (long long)t * W * nh;
        if constexpr (!FWD) {
            // Z[k] = S + Q, Z[m-k] = conj(S - Q), S = X[k] + conj X[m-k],
            // Q = i conj(w^k) (X[k] - conj X[m-k]); of bins 0 and m the real parts count
            if (w0 < lanes) {
                for (int k = k0; k < half; k += span) {
                    const V u = unp[k];
                    for (int w = w0; w < rows; w += lanes) {
                        V *row = cur + w * nh;
                        V a = row[k], x = row[m - k];
                        if (k == 0) a.y = x.y = (T)0;
                        const V s = V{a.x + x.x, a.y - x.y}, d = V{a.x - x.x, a.y + x.y};
                        const V q = c_mul(u, d);
                        row[k] = c_add(s, q);
                        if (k != 0 && m - k != k) row[m - k] = V{s.x - q.x, q.y - s.y};
                    }
                }
            }
            __syncthreads();
        }
        Ctx<T> c{cur, tw, tid % W, tid / W, nt / W, 1, nh, 0, 0};
        if constexpr (A::fixed) {
            run_stage<T, RMAX, FWD, PW, false>(c, typename A::S0(), none, nothing);
            c.in_n = PW;
            c.in_w = 1;
            run_stage<T, RMAX, FWD, PW, false>(c, typename A::S1(), none, nothing);
        } else {
            for (int s = 0; s < P.ax.nst; ++s) {
                run_stage<T, RMAX, FWD, PW, false>(c, P.ax.st[s], none, nothing);
                c.in_n = PW;
                c.in_w = 1;
            }
        }
        if constexpr (FWD) {
            // X[k] = E + O, X[m-k] = conj(E - O), E = (Z[k] + conj Z[m-k]) / 2,
            // O = -i w^k (Z[k] - conj Z[m-k]) / 2; Z[m] = Z[0]
            if (w0 < lanes) {
                for (int k = k0; k < half; k += span) {
                    const V u = unp[k];
                    const V *pa = cur + k * PW + w0, *px = cur + (k == 0 ? 0 : m - k) * PW + w0;
                    V *row = dst + w0 * nh;
                    for (int w = w0; w < rows; w += lanes, pa += lanes, px += lanes, row += lanes * nh) {
                        const V a = *pa, x = *px;
                        const V s = V{a.x + x.x, a.y - x.y}, d = V{a.x - x.x, a.y + x.y};
                        const V o = c_mul(u, d);
                        st_g(row + k, c_fma(o, hf, s));
                        if (m - k != k) st_g(row + m - k, V{hf * s.x - o.x, o.y - hf * s.y});
                    }
                }
            }
        } else {
            // the reals, and the two cells of padding as zero
            const int ospan = min(nt, (nh + 31) / 32 * 32), olanes = nt / ospan, oj = tid % ospan, ow = tid / ospan;
            if (ow < olanes) {
                for (int j = oj; j < nh; j += ospan) {
                    const V *in = cur + j * PW + ow;
                    V *out = dst + ow * nh + j;
                    for (int w = ow; w < rows; w += olanes, in += olanes, out += olanes * nh)
                        st_g(out, j < m ? *in : V{(T)0, (T)0});
                }
            }
        }
        __syncthreads();
        const int tn = t + P.nbuf * grid;
        if (tn < P.ntiles) fetch(tn, cur);
        fast::cp_async_commit();
        b = P.nbuf == 2 ? b ^ 1 : 0;
    }
}

// Threads and CTAs per SM of a length R1 * R2 (R1 >= R2).  The second stage
// has R1 butterflies of R2: a thread takes R1 / R2 of them, rounded, so that
// both stages keep the same threads busy (25 x 10 rows: 7 warps instead of 13
// of which 8 idle through the first stage, 63 against 115 us with the
// constants for 200 x 378 x 500).  Registers are estimated from what a thread
// holds; as many CTAs as these and one tile buffer each allow.
template <typename T, int R1, int R2> struct Shape {
    static constexpr int W = Width<T>::value;
    static constexpr int C2 = (R1 + R2 / 2) / R2;
    static constexpr int G = (R1 + C2 - 1) / C2 > R2 ? (R1 + C2 - 1) / C2 : R2;
    static constexpr int NT = (G * W + 31) / 32 * 32;
    static constexpr int HELD = R1 > C2 * R2 ? R1 : C2 * R2;
    static constexpr int REGS = sizeof(T) == 4 ? 2 * HELD + 36 : 4 * HELD + 48;
    static constexpr int SMEM = R1 * R2 * (W + 2) * 2 * (int)sizeof(T) + 1024;
    static constexpr int BY_REGS = 65536 / (NT * REGS), BY_SMEM = 232448 / SMEM, BY_THREADS = 2048 / NT;
    static constexpr int LEAST = BY_REGS < BY_SMEM ? BY_REGS : BY_SMEM;
    static constexpr int MINB = LEAST < 1 ? 1 : LEAST < BY_THREADS ? LEAST : BY_THREADS;
};
template <typename T, int R1, int R2, bool FWD, bool EPI>
__global__ void __launch_bounds__(Shape<T, R1, R2>::NT, Shape<T, R1, R2>::MINB)
    axis_cols_n(const __grid_constant__ ColParams P) {
    using S = Shape<T, R1, R2>;
    cols_body<T, 32, FWD, EPI>(P, FixedAxis<S::W, R1, R2, S::NT>{P.ax});
}
template <typename T, int R1, int R2, bool FWD>
__global__ void __launch_bounds__(Shape<T, R1, R2>::NT, Shape<T, R1, R2>::MINB)
    axis_rows_n(const __grid_constant__ RowParams P) {
    using S = Shape<T, R1, R2>;
    rows_body<T, 32, FWD>(P, FixedAxis<S::W, R1, R2, S::NT>{P.ax});
}

template <typename T, int W, int RMAX, bool FWD, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) axis_rows(const __grid_constant__ RowParams P) {
    rows_body<T, RMAX, FWD>(P, AnyAxis<W>{P.ax});
}

// A length with kernels of its own (rows up to 512: m = Nz / 2)
struct Fixed {
    int n, r1, r2, nt;
    const void *cols[2][2];  // [forward][epilogue]
    const void *rows[2];     // [forward]
};
struct FixedTable {
    const Fixed *lengths;
    int count;
};
template <typename T, int R1, int R2, bool FWD> constexpr const void *rows_of() {
    if constexpr (R1 * R2 <= 512)
        return (const void *)axis_rows_n<T, R1, R2, FWD>;
    else
        return nullptr;
}
#define GPUFFT_AXIS_FIXED(R1, R2)                                                                               \
    {R1 * R2, R1, R2, Shape<Real, R1, R2>::NT,                                                                  \
     {{(const void *)axis_cols_n<Real, R1, R2, false, false>, (const void *)axis_cols_n<Real, R1, R2, false, true>}, \
      {(const void *)axis_cols_n<Real, R1, R2, true, false>, (const void *)axis_cols_n<Real, R1, R2, true, true>}},  \
     {rows_of<Real, R1, R2, false>(), rows_of<Real, R1, R2, true>()}},

// The compiled kernels of one precision, by radix class: the class of a
// length is the first whose largest radix and thread limit it keeps to
// (axis.cu).  The last class is for lengths of three stages.
struct Kernel {
    const void *fwd, *inv;
    int w, rmax, nt;  // sequences per tile, largest radix, most threads
};
constexpr int kClasses = 4;
extern const Kernel kCols_f32[kClasses], kColsEpi_f32[kClasses], kRows_f32[kClasses];
extern const Kernel kCols_f64[kClasses], kColsEpi_f64[kClasses], kRows_f64[kClasses];

#define GPUFFT_AXIS_COLS(T, W, RMAX, EPI, NT, MINB)                                                             \
    {(const void *)axis_cols<T, W, RMAX, true, EPI, NT, MINB>, (const void *)axis_cols<T, W, RMAX, false, EPI, NT, MINB>, \
     W, RMAX, NT}
#define GPUFFT_AXIS_ROWS(T, W, RMAX, NT, MINB)                                                                  \
    {(const void *)axis_rows<T, W, RMAX, true, NT, MINB>, (const void *)axis_rows<T, W, RMAX, false, NT, MINB>, W, RMAX, NT}

}  // namespace axis
}  // namespace gpufft
