// fft_axis.cuh — one axis of the transform per launch, for any axis length
// from 16 to 1024 with no prime factor above 13.
//
// The cluster-per-plane kernels of fft_kernels.cuh take any length, but they
// walk it in three to six radix stages with run-time strides, one butterfly
// at a time, and spend 130 (x axis) to 320 (z and y axes) instructions per
// element: at 200 x 378 x 500 FP32 they issue on 54-60% of all cycles and
// move 14% (z and y) and 32% (x) of the copy bandwidth.  Here
//  * a length up to 1024 is in almost every case R1 * R2 with R1, R2 <= 32
//    (every product of 2s, 3s and 5s but 972 and 1000): two passes over
//    shared memory, the rest three;
//  * every length (axis_lengths.h) has kernels of its own, radices and strides
//    as constants: 40 to 50 instructions per element and axis, against 62 to
//    112 for the same stages with run-time lengths and a switch over the
//    radices, and registers that fit the radices;
//  * a thread keeps its butterflies in registers, so a stage works in place;
//  * a tile is W sequences, element (i, w) at i * PW + w: a half-warp reads
//    and writes W adjacent elements (128 bytes) whatever the radix, without
//    bank conflicts.  Rows (z) use PW = W + 1, so that turning them over has
//    none either (ncu counts 10-13% of all shared wavefronts as conflicts in
//    the column kernels, 12-16% in the rows');
//  * tiles are copied in ahead of use by tensor copies (columns) and one bulk
//    copy (rows): against cp.async 20% fewer instructions and 40% fewer
//    shared-memory wavefronts (500^3 FP32 x axis 215 -> 177 us, z and y axes
//    437 -> 390).
// z and y run as two launches, so the field crosses HBM three times per
// transform instead of twice (from L2 when it fits there); what that costs is
// less than what the instructions saved bring: R2C + C2R of 420 x 378 x 500
// FP32 2.01 -> 0.75 ms, 768^3 12.4 -> 4.2, 225 x 243 x 350 FP64 0.86 -> 0.35.
// Each launch moves 0.7-0.85 of the copy bandwidth; at 252 x 378 x 500 FP32
// 34-43% of the issue slots are used, the FMA pipe 27-37%, the shared-memory
// data pipe 36-37% (rows 60%): what is left is waiting at the block barriers
// between a stage's bursts of shared-memory accesses and its arithmetic.
#pragma once
#include "fft_fast.cuh"
#include "fft_queue.cuh"
#include "fft_radix.cuh"

namespace gpufft {
namespace axis {

// Stage of radix R after radices of product P: NB butterflies, taken by G
// threads per sequence, C each; twiddles exp(-2 pi i j k / (P R)) at OFF +
// (j - 1) * P + k.
template <int R_, int P, int NB, int OFF, int G> struct Stage {
    static constexpr int r = R_, p = P, nb = NB, off = OFF, c = (NB + G - 1) / G;
};

// Columns: groups of gcols adjacent sequences, group g at data + g * gstride,
// consecutive elements of a sequence `pitch` apart.  A group is cut into
// full = gcols / W whole tiles; the columns left over (rem of each group, 1 of
// 2^k + 1 for the y axis) are gathered from several groups into tiles of their
// own, so that no tile is mostly empty.
struct ColParams {
    void *data;
    const void *tw;
    long long pitch, gstride;
    int gcols, full, rem;
    FastDiv fulldiv, remdiv;
    int nfull, nrem;  // whole tiles of all groups, left-over columns of all groups
    int ntiles, nbuf;
    int tile;  // elements of a tile buffer
    // How whole tiles are copied in (left-over tiles: element by element).
    // 0: element by element.
    // 1: tensor copies (rows 16-byte aligned): nbox boxes of boxh rows.
    // 2: FP32 with an odd pitch, every other row 8 bytes off a 16-byte
    //    boundary: column pairs by cp.async, from the boundary at or before the row's
    //    first column into rows of W + 2, even and odd rows apart (Ctx).
    // 3: the same by tensor copies over the view of two rows as one line
    //    (n even): boxes of W + 2 columns at column c of the even rows and at
    //    c - 1 of the odd ones.
    int copy;
    int gpar;  // copy 2: row r of group g is off by 8 bytes where r + gpar * g is odd
    int boxh, nbox;
    int odd;   // copies 2 and 3: where the odd rows of a tile start
    int *err;           // raised when a tile's copy has not arrived within wait_ns
    long long wait_ns;
    int missing;        // bytes expected of a tile's copy beyond those it brings: 0 (a test of the limit: more)
    // x-pass epilogue (PassBParams), on when epi is set: scale, and the 2/3-rule mask of column ky * nh + kz
    int epi, dealias, ny, nh, nz;
    double scale;
};

// rows: nrows sequences of m complex, row r at data + r * nh (nh = m + 1)
struct RowParams {
    void *data;
    const void *tw;
    const void *unp;  // forward -i w^k / 2, inverse i conj(w^k), w = exp(-2 pi i / (2 m)), k <= m / 2
    int nrows;
    int ntiles, nbuf;
    int aligned;  // data 16-byte aligned
    int *err;     // these as in ColParams
    long long wait_ns;
    int missing;
};

template <typename V> __host__ __device__ constexpr int col_table_bytes(int n) {
    return (n * (int)sizeof(V) + 127) / 128 * 128;
}

// elements between the rows of a row tile (rows_body), and of a tile buffer
template <typename V> __host__ __device__ constexpr int row_pitch(int m) {
    const int nh = m + 1;
    return nh % 2 ? nh : sizeof(V) == 16 ? nh + 1 : nh % 4 ? nh : nh + 2;  // (FP32: rows 16-byte aligned)
}
template <typename V> __host__ __device__ constexpr int row_tile(int m, int w) {
    const int a = (m + 1) * (w + 1), b = w * row_pitch<V>(m);
    return ((a > b ? a : b) + 1) / 2 * 2;
}

// sequences per tile for which a tile row is 128 bytes
template <typename T> struct Width;
template <> struct Width<float> { static constexpr int value = 16; };
template <> struct Width<double> { static constexpr int value = 8; };

// How a stage's inputs lie in the tile.
enum Lie {
    TILE,   // n * PW + w, as every stage leaves its results
    FIRST,  // the first stage of a column: n * PW + w, or even and odd rows apart (copies 2 and 3)
    ROW     // the first stage of a row: n + w * in_w
};
// Where a stage's results go: n * PW + w of the tile, n + w * in_w (the last
// stage of an inverse row), or out.put (the last stage of a column).
enum To { IN_PLACE, TO_ROWS, TO_OUT };
// a thread's part of a tile
template <typename T> struct Ctx {
    using V = cx_t<T>;
    V *sm;
    const V *tw;
    int w, i0, g;          // this thread's sequence, first butterfly and butterfly step
    int in_w;              // ROW, TO_ROWS
    bool apart;            // FIRST: input n at n / 2 * (PW + 2) + (n % 2) * in1 + in0 + w
    int in1, in0;
};

// the R inputs i + j NB of butterfly i; element n at (n / 2) * IN2 + (n % 2) * in1 from `at`
template <int R, int NB, int IN2, class V>
__device__ __forceinline__ void load_apart(V (&v)[R], const V *at, int in1, int i) {
    // NB odd: inputs of even and of odd j each step by 2 NB
    const V *even = at + (i >> 1) * IN2 + (i & 1) * in1;
    const V *odd = NB % 2 ? at + ((i + NB) >> 1) * IN2 + ((i + NB) & 1) * in1 : even;
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = NB % 2 ? (j & 1 ? odd : even)[j / 2 * NB * IN2] : even[j * (NB / 2) * IN2];
}

// One stage in place in shared memory, its results in the layout n * PW + w,
// or handed to out.put (the last stage of a column).  `freed` runs once every
// thread has read its inputs.
template <typename T, class S, bool FWD, int PW, Lie LIE, To TO, class Out, class Freed>
__device__ __forceinline__ void stage(const Ctx<T> &c, Out &out, Freed &freed) {
    using V = cx_t<T>;
    constexpr int R = S::r, C = S::c, NB = S::nb, P = S::p;
    V v[C][R];
#pragma unroll
    for (int m = 0; m < C; ++m) {
        const int i = c.i0 + m * c.g;
        if (i < NB) {
            if (LIE == FIRST && sizeof(V) == 8 && c.apart) {
                load_apart<R, NB, PW + 2>(v[m], c.sm + c.in0 + c.w, c.in1, i);
            } else {
                const V *in = LIE == ROW ? c.sm + c.w * c.in_w + i : c.sm + i * PW + c.w;
#pragma unroll
                for (int j = 0; j < R; ++j) v[m][j] = in[j * NB * (LIE == ROW ? 1 : PW)];
            }
        } else {
            // (left undefined, the registers would stay alive through the tile loop)
#pragma unroll
            for (int j = 0; j < R; ++j) v[m][j] = V{(T)0, (T)0};
        }
    }
    __syncthreads();
    if constexpr (TO == TO_OUT) freed();
#pragma unroll
    for (int m = 0; m < C; ++m) {
        const int i = c.i0 + m * c.g;
        if (i < NB) {
            const int ip = i / P;
            const int k = i - ip * P;
            if constexpr (P > 1) {
                const V *tw = c.tw + S::off + k;
#pragma unroll
                for (int j = 1; j < R; ++j) v[m][j] = c_tw<FWD>(v[m][j], tw[(j - 1) * P]);
            }
            Dft<R, FWD, V>::run(v[m]);
            if constexpr (TO == TO_OUT) {
                out.template put<R>(i, NB, v[m]);
            } else if constexpr (TO == TO_ROWS) {
                V *o = c.sm + c.w * c.in_w + ip * P * R + k;
#pragma unroll
                for (int j = 0; j < R; ++j) o[j * P] = v[m][j];
            } else {
                V *o = c.sm + (ip * P * R + k) * PW + c.w;
    #pragma unroll
                for (int j = 0; j < R; ++j) o[j * P * PW] = v[m][j];
            }
        }
    }
    if constexpr (TO != TO_OUT) __syncthreads();
}

// The axis of length R1 * R2 * R3 (R3 = 1: two stages) on tiles of W
// sequences, NT threads.
template <int W_, int R1, int R2, int R3, int NT> struct Axis {
    static constexpr int W = W_, n = R1 * R2 * R3, nt = NT, G = NT / W, nst = R3 > 1 ? 3 : 2;
    using S0 = Stage<R1, 1, n / R1, 0, G>;
    using S1 = Stage<R2, R1, n / R2, R1 - 1, G>;
    using S2 = Stage<R3, R1 * R2, n / R3, R1 * R2 - 1, G>;
};

struct NoOut {};
struct NoFreed {
    __device__ __forceinline__ void operator()() const {}
};

// where the last stage of a column puts its results: straight to global
// memory, with the x-pass epilogue if there is one
template <typename T> struct ColOut {
    using V = cx_t<T>;
    V *base;  // this thread's column, or null past the last one
    long long pitch;
    bool epi;
    int nx;  // with the mask: n, else 0
    bool drop;  // ky or kz outside the 2/3-rule box
    T scale;
    template <int R> __device__ __forceinline__ void put(int i, int nb, V *v) const {
        if (!base) return;
        V *o = base + (long long)i * pitch;
        const uint32_t step = (uint32_t)nb * (uint32_t)pitch;  // (fits: the plan checks n / 2 * pitch)
        if (!epi) {
#pragma unroll
            for (int j = 0; j < R; ++j) st_g(o + (size_t)j * step, v[j]);
        } else if (!nx) {
#pragma unroll
            for (int j = 0; j < R; ++j) st_g(o + (size_t)j * step, V{v[j].x * scale, v[j].y * scale});
        } else {
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const int kx = i + j * nb;
                const bool zero = (drop || 3 * min(kx, nx - kx) > nx);
                st_g(o + (size_t)j * step, zero ? V{(T)0, (T)0} : V{v[j].x * scale, v[j].y * scale});
            }
        }
    }
};

// Waits for a tile's copy to arrive.  False once the limit has passed: the flag is raised, and the copy has been
// given the same time again, so that the CTA, which ends now, leaves none in flight into its shared memory unless
// it takes more than twice the limit.  (The other buffer's copy is the caller's to wait for.)
template <class Params>
__device__ __forceinline__ bool arrived(const Params &P, uint64_t *full, int b, uint32_t parity) {
    if (q::mbar_wait(&full[b], parity, P.wait_ns)) return true;
    atomicExch(P.err, 1);
    q::mbar_wait(&full[b], parity, P.wait_ns);
    return false;
}

template <typename T, bool FWD, class A>
__device__ __forceinline__ void cols_body(const ColParams &P, const CUtensorMap &tm) {
    using V = cx_t<T>;
    constexpr int W = A::W, n = A::n, nt = A::nt;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    // n - 1 twiddles, the tile buffers (128-byte aligned), a barrier per buffer
    unsigned char *smem = smem_raw + ((128u - (q::smem_u32(smem_raw) & 127u)) & 127u);
    V *tw = reinterpret_cast<V *>(smem);
    V *buf = reinterpret_cast<V *>(smem + col_table_bytes<V>(n));
    const int tile = P.tile;
    uint64_t *full = reinterpret_cast<uint64_t *>(buf + P.nbuf * tile);
    const bool tensor = P.copy == 1 || P.copy == 3;
    for (int q = tid; q < n - 1; q += nt) tw[q] = reinterpret_cast<const V *>(P.tw)[q];
    if (tensor) {
        if (tid == 0) {
            for (int b = 0; b < P.nbuf; ++b) q::mbar_init(&full[b], 1);
            q::fence_mbar_init();
        }
        __syncthreads();
    }
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
    auto fetch = [&](int t, int b) {
        V *dst = buf + b * tile;
        int g, c;
        if (t < P.nfull && tensor) {
            if (tid == 0) {
                constexpr int E8 = (int)sizeof(V) / 8;  // the maps count 8-byte elements
                column(t, 0, g, c);
                q::fence_proxy_async_shared();  // (the buffer's last readers are behind a block barrier)
                if (P.copy == 1) {
                    q::mbar_arrive_expect_tx(&full[b], (uint32_t)(P.nbox * P.boxh * W * (int)sizeof(V) + P.missing));
                    for (int x = 0; x < P.nbox; ++x)
                        q::tensor_load_2d(dst + x * P.boxh * W, &tm, c * E8, g * n + x * P.boxh, &full[b]);
                } else {
                    q::mbar_arrive_expect_tx(&full[b],
                                             (uint32_t)(2 * P.nbox * P.boxh * (W + 2) * (int)sizeof(V) + P.missing));
                    for (int x = 0; x < P.nbox; ++x) {
                        const int at = x * P.boxh * (W + 2), line = g * (n / 2) + x * P.boxh;
                        q::tensor_load_2d(dst + at, &tm, c, line, &full[b]);
                        q::tensor_load_2d(dst + P.odd + at, &tm, (int)P.pitch - 1 + c, line, &full[b]);
                    }
                }
            }
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
                dst += (r0 >> 1) * (W + 2) + (r0 & 1) * P.odd + 2 * ch;
                const int bytes = ch < CH ? 16 : 8;  // (the last chunk's second element is another tile's, or past the field)
                for (int r = r0; r < n; r += rs, src += step, dst += (rs / 2) * (W + 2)) fast::cp_async16(dst, src, bytes);
            }
        } else {
            const int w = tid % W, r0 = tid / W, rs = nt / W;
            if (column(t, w, g, c)) {
                const V *src = data + (long long)g * P.gstride + c + (long long)r0 * P.pitch;
                const long long step = (long long)rs * P.pitch;
                dst += r0 * W + w;
                for (int r = r0; r < n; r += rs, src += step, dst += rs * W) fast::cp_async_elem(dst, src, true);
            }
        }
        fast::cp_async_commit();
    };
    const int grid = gridDim.x;
    wait_for_previous_launch();
    for (int b = 0; b < P.nbuf; ++b) {
        const int t = blockIdx.x + b * grid;
        if (t < P.ntiles)
            fetch(t, b);
        else
            fast::cp_async_commit();
    }
    int b = 0;
    uint32_t parity = 0;
    for (int t = blockIdx.x; t < P.ntiles; t += grid) {
        if (t + grid >= P.ntiles) let_next_launch_start();
        if (tensor && t < P.nfull) {
            if (!arrived(P, full, b, parity)) {
                if (P.nbuf == 2 && t + grid < P.nfull) q::mbar_wait(&full[b ^ 1], parity ^ (uint32_t)b, P.wait_ns);
                return;
            }
        } else {
            if (P.nbuf == 2)
                fast::cp_async_wait<1>();
            else
                fast::cp_async_wait<0>();
            __syncthreads();
        }
        V *cur = buf + b * tile;
        int g, col;
        const bool valid = column(t, tid % W, g, col);
        const bool apart = sizeof(V) == 8 && t < P.nfull && P.copy >= 2;
        const int off = P.gpar * g & 1;  // the odd rows are 8 bytes off (0) or the even ones (1)
        const Ctx<T> c{cur, tw, tid % W, tid / W, nt / W, 0, apart, P.odd + 1 - 2 * off, off};
        NoOut none;
        NoFreed nothing;
        stage<T, typename A::S0, FWD, W, FIRST, IN_PLACE>(c, none, nothing);
        if constexpr (A::nst == 3) stage<T, typename A::S1, FWD, W, TILE, IN_PLACE>(c, none, nothing);
        ColOut<T> out;
        out.base = valid ? data + (long long)g * P.gstride + col : nullptr;
        out.pitch = P.pitch;
        out.epi = P.epi;
        if (P.epi) {
            const int ky = col / P.nh, kz = col - ky * P.nh;
            out.drop = 3 * min(ky, P.ny - ky) > P.ny || 3 * kz > P.nz;
            out.nx = P.dealias ? n : 0;
            out.scale = (T)P.scale;
        }
        auto freed = [&]() {
            const int tn = t + P.nbuf * grid;
            if (tn < P.ntiles)
                fetch(tn, b);
            else
                fast::cp_async_commit();
        };
        using Last = std::conditional_t<A::nst == 3, typename A::S2, typename A::S1>;
        stage<T, Last, FWD, W, TILE, TO_OUT>(c, out, freed);
        if (P.nbuf == 2) {
            b ^= 1;
            parity ^= b == 0;
        } else {
            parity ^= 1;
        }
    }
}

// Rows.  A tile is W whole rows, one contiguous span of the field, copied in
// row after row; the first stage turns it over to n * PW + w.  Rows lie PITCH
// apart: nh where that keeps W rows' elements at one position out of each
// other's banks (odd nh: one bulk copy for the tile), else padded (a bulk copy
// a row).  The inverse's last stage turns the tile back, and bulk stores write
// it out as it came.
template <typename T, bool FWD, class A>
__device__ __forceinline__ void rows_body(const RowParams &P) {
    using V = cx_t<T>;
    constexpr int W = A::W, PW = W + 1, m = A::n, nh = m + 1, half = m / 2 + 1, nt = A::nt;
    constexpr int PITCH = row_pitch<V>(m), E = (int)sizeof(V);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    V *unp = reinterpret_cast<V *>(smem_raw);      // half entries
    V *tw = unp + half;                            // m - 1 entries
    V *buf = unp + (half + m + 1) / 2 * 2;
    constexpr int tile = row_tile<V>(m, W);
    uint64_t *full = reinterpret_cast<uint64_t *>(buf + P.nbuf * tile);
    for (int q = tid; q < half; q += nt) unp[q] = reinterpret_cast<const V *>(P.unp)[q];
    for (int q = tid; q < m - 1; q += nt) tw[q] = reinterpret_cast<const V *>(P.tw)[q];
    if (tid == 0) {
        for (int b = 0; b < P.nbuf; ++b) q::mbar_init(&full[b], 1);
        q::fence_mbar_init();
    }
    __syncthreads();
    V *data = reinterpret_cast<V *>(P.data);
    // tiles that go by bulk copies: those whose ends are 16-byte aligned (whole tiles are, of aligned fields)
    const int bulk = P.aligned ? P.nrows / W + (E == 16 || P.nrows % W * nh % 2 == 0) : 0;
    // the threads that issue them: one for the tile, or one a row
    constexpr bool whole = PITCH == nh;
    auto fetch = [&](int t, int b) {
        const int rows = min(W, P.nrows - t * W);
        const V *src = data + (long long)t * W * nh;
        V *dst = buf + b * tile;
        if (t < bulk) {
            // Every thread that stored from the buffer waits until its stores have read it, also those
            // that have no row of this tile (the last one): the stages write over the whole buffer, behind
            // the block barrier that follows the pack.
            if (!FWD && tid < (whole ? 1 : W)) q::bulk_wait_read();
            if (tid < (whole ? 1 : rows)) {
                q::fence_proxy_async_shared();       // (its last readers are behind a block barrier)
                if (tid == 0) q::mbar_arrive_expect_tx(&full[b], (uint32_t)(rows * nh * E + P.missing));
                q::bulk_load(dst + tid * PITCH, src + tid * nh, (uint32_t)((whole ? rows : 1) * nh * E), &full[b]);
            }
        } else {
            if (!FWD) {  // (the buffer's last tile may have gone by bulk stores)
                q::bulk_wait_read();
                __syncthreads();
            }
            for (int q = tid; q < rows * nh; q += nt) {
                const int w = q / nh;
                fast::cp_async_elem(dst + q + w * (PITCH - nh), src + q, true);
            }
        }
        fast::cp_async_commit();
    };
    // bins k and m - k of one row at a time: `span` adjacent threads take a row
    constexpr int span = nt < (half + 31) / 32 * 32 ? nt : (half + 31) / 32 * 32, lanes = nt / span;
    const int k0 = tid % span, w0 = tid / span;
    const int grid = gridDim.x;
    wait_for_previous_launch();
    for (int b = 0; b < P.nbuf; ++b) {
        const int t = blockIdx.x + b * grid;
        if (t < P.ntiles)
            fetch(t, b);
        else
            fast::cp_async_commit();
    }
    const T hf = (T)0.5;
    int b = 0;
    uint32_t parity = 0;
    for (int t = blockIdx.x; t < P.ntiles; t += grid) {
        if (t + grid >= P.ntiles) let_next_launch_start();
        if (t < bulk) {
            if (!arrived(P, full, b, parity)) {
                if (P.nbuf == 2 && t + grid < bulk && (FWD || t == (int)blockIdx.x))
                    q::mbar_wait(&full[b ^ 1], parity ^ (uint32_t)b, P.wait_ns);
                if (!FWD) q::bulk_wait_all();
                return;
            }
        } else {
            if (FWD && P.nbuf == 2)
                fast::cp_async_wait<1>();
            else
                fast::cp_async_wait<0>();
            __syncthreads();
        }
        // (the inverse refills the other buffer here, a tile later than it was read: its bulk store has
        // read it by now)
        if (!FWD && P.nbuf == 2 && t != (int)blockIdx.x && t + grid < P.ntiles) fetch(t + grid, b ^ 1);
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
                        V *row = cur + w * PITCH;
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
        const Ctx<T> c{cur, tw, tid % W, tid / W, nt / W, PITCH, false, 0, 0};
        constexpr To last = FWD ? IN_PLACE : TO_ROWS;
        stage<T, typename A::S0, FWD, PW, ROW, IN_PLACE>(c, none, nothing);
        stage<T, typename A::S1, FWD, PW, TILE, A::nst == 3 ? IN_PLACE : last>(c, none, nothing);
        if constexpr (A::nst == 3) stage<T, typename A::S2, FWD, PW, TILE, last>(c, none, nothing);
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
            __syncthreads();
        } else {
            // the two cells of padding as zero, then the rows as they lie
            if (tid < rows) cur[tid * PITCH + m] = V{(T)0, (T)0};
            if (t < bulk) q::fence_proxy_async_shared();
            __syncthreads();
            if (t < bulk) {
                if (tid < (whole ? 1 : rows))
                    q::bulk_store(dst + tid * nh, cur + tid * PITCH, (uint32_t)((whole ? rows : 1) * nh * E));
            } else {
                for (int q = tid; q < rows * nh; q += nt) st_g(dst + q, cur[q + q / nh * (PITCH - nh)]);
                __syncthreads();
            }
        }
        if (FWD || P.nbuf == 1) {
            const int tn = t + P.nbuf * grid;
            if (tn < P.ntiles)
                fetch(tn, b);
            else
                fast::cp_async_commit();
        }
        if (P.nbuf == 2) {
            b ^= 1;
            parity ^= b == 0;
        } else {
            parity ^= 1;
        }
    }
    if (!FWD) q::bulk_wait_all();
}

// Threads and CTAs per SM of a length R1 * R2 (R1 >= R2).  The second stage
// has R1 butterflies of R2: where R1 > 2 R2 a thread takes several of them, so
// that the first stage, with R2 butterflies, does not leave most threads idle
// (25 x 10 FP64 z axis 0.76 of the copy bandwidth against 0.68 with one each);
// from there down one each is the better (128 = 16 x 8 FP64 x axis 0.82
// against 0.73 with two, 18 x 12 0.80 against 0.72).  Registers are estimated
// from what a thread holds; as many CTAs as these and one tile buffer each
// allow (one CTA more, at fewer registers: 5-30% slower almost everywhere).
// Three stages: a thread holds about 24 elements (FP64: 16).
template <typename T, int R1, int R2, int R3> struct Shape {
    static constexpr int W = Width<T>::value, N = R1 * R2 * R3;
    static constexpr int up(int a, int b) { return (a + b - 1) / b; }
    static constexpr int most(int a, int b) { return a > b ? a : b; }
    static constexpr int C2 = R1 > 2 * R2 ? (R1 - 1) / R2 : 1;
    static constexpr int G0 = R3 == 1 ? most(up(R1, C2), R2) : up(N, sizeof(T) == 4 ? 24 : 16);
    static constexpr int NT = up(G0 * W, 32) * 32, G = NT / W;
    static constexpr int HELD = most(up(N / R1, G) * R1, most(up(N / R2, G) * R2, R3 == 1 ? 0 : up(N / R3, G) * R3));
    static constexpr int REGS = sizeof(T) == 4 ? 2 * HELD + 36 : 4 * HELD + 48;
    static constexpr int SMEM = N * (W + 2) * 2 * (int)sizeof(T) + 1024;
    static constexpr int BY_REGS = 65536 / (NT * REGS), BY_SMEM = 232448 / SMEM, BY_THREADS = 2048 / NT;
    static constexpr int LEAST = BY_REGS < BY_SMEM ? BY_REGS : BY_SMEM;
    static constexpr int MINB = LEAST < 1 ? 1 : LEAST < BY_THREADS ? LEAST : BY_THREADS;
    using A = Axis<W, R1, R2, R3, NT>;
};
template <typename T, int R1, int R2, int R3, bool FWD>
__global__ void __launch_bounds__(Shape<T, R1, R2, R3>::NT, Shape<T, R1, R2, R3>::MINB)
    axis_cols(const __grid_constant__ ColParams P, const __grid_constant__ CUtensorMap tm) {
    cols_body<T, FWD, typename Shape<T, R1, R2, R3>::A>(P, tm);
}
template <typename T, int R1, int R2, int R3, bool FWD>
__global__ void __launch_bounds__(Shape<T, R1, R2, R3>::NT, Shape<T, R1, R2, R3>::MINB)
    axis_rows(const __grid_constant__ RowParams P) {
    rows_body<T, FWD, typename Shape<T, R1, R2, R3>::A>(P);
}

// the kernels of a length (rows up to 512: m = Nz / 2)
struct Kernels {
    int r[3], nt;
    const void *cols[2], *rows[2];  // [forward]
};
struct KernelTable {
    const Kernels *lengths;
    int count;
};
template <typename T, int R1, int R2, int R3, bool FWD> constexpr const void *rows_of() {
    if constexpr (R1 * R2 * R3 <= 512)
        return (const void *)axis_rows<T, R1, R2, R3, FWD>;
    else
        return nullptr;
}
#define GPUFFT_AXIS_KERNELS(R1, R2, R3)                                                                         \
    {{R1, R2, R3},                                                                                              \
     Shape<Real, R1, R2, R3>::NT,                                                                               \
     {(const void *)axis_cols<Real, R1, R2, R3, false>, (const void *)axis_cols<Real, R1, R2, R3, true>},       \
     {rows_of<Real, R1, R2, R3, false>(), rows_of<Real, R1, R2, R3, true>()}},

}  // namespace axis
}  // namespace gpufft
