// The track pass on sm_100a: one CTA per search point computes the ZNCC surface in shared
// memory, its row-major argmax and the 5x5 refinement patch; a second kernel runs the pyrUp
// cascade on the patches. The surface never leaves shared memory.
//
// Reference (AutoRIFT.jl): src/track.jl:103-152, 249-305 (the grid loop), src/points.jl:358-395
// (chip and window bounds), src/correlate.jl:423-453 (prepare_chip!), 575-630 (ZNCC / NCC
// normalisation), 785-848 (numerator), src/integral.jl:141-170, 244-247 (per-window sums),
// src/peak.jl:32-61, 102-106, 196-324, 456-522 (peak and sub-pixel cascade).
//
// Numerics.
//  * Numerator: FP32 products accumulated in FP32 over a few chip columns, then flushed into
//    an FP64 accumulator. For UInt8 imagery the chip and window are staged as raw integers
//    and the flush interval keeps every FP32 partial below 2^24, so the numerator
//    sum(T*W) - mean(T)*sum(W) is exact -- the value the reference's FP32 FFT approximates.
//    Other element types stage the mean-removed chip and a centred window (W - c).
//  * Denominator: window box sums from per-window prefix tables built by warp scans in
//    shared memory -- exact integers (uint32) for UInt8, FP64 otherwise -- and
//    wvar = max(s2 - s1*s1/n, 0), den = cnorm*sqrt(wvar), surface = Float32(num/den), each
//    operation an explicitly rounded FP64 intrinsic, as in src/correlate.jl:591-600.
//  * Cascade: every pyrUp sample is fl(fl(0.75*b) + fl(0.125*fl(a+c))) or
//    fl(0.5*fl(b+c)) with __fmul_rn/__fadd_rn, so no step is fused into an FMA and the result
//    is bit-identical to the reference's Float32 arithmetic on the same patch.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>
#include <type_traits>

#include "ar_internal.cuh"
#include "ar_tc.cuh"

namespace ar {
namespace {

constexpr int kMI = 10;        // surface rows per thread item
constexpr int kUA = 16;        // chip rows per inner step
constexpr int kCorrThreads = 256;
constexpr unsigned kFull = 0xffffffffu;

template <typename T>
struct Traits;
template <>
struct Traits<uint8_t> {
    static constexpr bool raw = true;  // exact integer numerator
    static constexpr bool integer = true;
    typedef uint32_t ph_t;
};
template <>
struct Traits<uint16_t> {
    static constexpr bool raw = false;
    static constexpr bool integer = true;
    typedef double ph_t;
};
template <>
struct Traits<int16_t> {
    static constexpr bool raw = false;
    static constexpr bool integer = true;
    typedef double ph_t;
};
template <>
struct Traits<float> {
    static constexpr bool raw = false;
    static constexpr bool integer = false;
    typedef double ph_t;
};

// ----------------------------------------------------------------------------------------------
// Reductions

// Key for a row-major first strict maximum (src/peak.jl:32-61): the larger value wins, and
// among equal values the smaller row-major index. NaN never wins; -0 equals +0.
__device__ __forceinline__ unsigned long long argmax_key(float v, unsigned rowmajor) {
    if (v != v) return 0ull;
    if (v == 0.0f) v = 0.0f;
    unsigned u = __float_as_uint(v);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return (static_cast<unsigned long long>(u) << 32) | (0xffffffffu - rowmajor);
}

__device__ __forceinline__ float key_value(unsigned long long key) {
    unsigned u = static_cast<unsigned>(key >> 32);
    u = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    return __uint_as_float(u);
}

// Decode to (row-major index, value); the reference returns (1,1) when nothing beats -Inf.
__device__ __forceinline__ bool key_decode(unsigned long long key, unsigned* rowmajor,
                                          float* value) {
    if (key == 0ull) return false;
    const float v = key_value(key);
    if (v == -INFINITY) return false;
    *rowmajor = 0xffffffffu - static_cast<unsigned>(key & 0xffffffffull);
    *value = v;
    return true;
}

__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(kFull, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// Largest value of a warp (no lane NaN): floats as ordered integers, one reduction instruction.
__device__ __forceinline__ float warp_max(float v) {
    int i = __float_as_int(v);
    i ^= (i >> 31) & 0x7fffffff;
    i = __reduce_max_sync(kFull, i);
    return __int_as_float(i ^ ((i >> 31) & 0x7fffffff));
}

// A barrier over the block, or (MAIN) over its first 256 threads (k_corr_tc2's main warps).
template <bool MAIN>
__device__ __forceinline__ void block_sync() {
    if constexpr (MAIN) {
        asm volatile("bar.sync 2, 256;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// Block-wide max; every thread gets the result. `red` holds >= 32 entries.
template <bool MAIN = false>
__device__ unsigned long long block_max_u64(unsigned long long v, unsigned long long* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = MAIN ? 8 : (blockDim.x + 31) >> 5;
    v = warp_max_u64(v);
    block_sync<MAIN>();
    if (lane == 0) red[warp] = v;
    block_sync<MAIN>();
    unsigned long long r = lane < nw ? red[lane] : 0ull;
    r = warp_max_u64(r);
    return r;
}

__device__ __forceinline__ double warp_sum_f64(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(kFull, v, o));
    return v;
}

// Block-wide sum of up to three doubles; every thread gets the results.
template <int N, bool MAIN = false>
__device__ void block_sum_f64(double (&v)[N], double* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = MAIN ? 8 : (blockDim.x + 31) >> 5;
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = warp_sum_f64(v[q]);
    block_sync<MAIN>();
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < N; ++q) red[q * 32 + warp] = v[q];
    }
    block_sync<MAIN>();
#pragma unroll
    for (int q = 0; q < N; ++q) {
        double r = lane < nw ? red[q * 32 + lane] : 0.0;
        v[q] = warp_sum_f64(r);
    }
}

template <typename V>
__device__ __forceinline__ V warp_inclusive_scan(V v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const V w = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v = v + w;
    }
    return v;
}

// ----------------------------------------------------------------------------------------------
// pyrUp arithmetic

// One pyrUp sample in the reference's operation order (src/peak.jl:266-292).
__device__ __forceinline__ float pyr_sample(int nt, float a, float b, float c) {
    return nt == 3 ? __fadd_rn(__fmul_rn(0.75f, b), __fmul_rn(0.125f, __fadd_rn(a, c)))
                   : __fmul_rn(0.5f, __fadd_rn(b, c));
}

// ----------------------------------------------------------------------------------------------
// Correlation kernel

struct CorrArgs {
    const void* ref;
    const void* sec;
    const uint8_t* valid;
    int64_t nrows, ncols;
    DevPoints pts;
    int64_t padx, pady;
    int up, measure;
    int TI, TJ;   // surface tile; TI a multiple of kMI and (TI/kMI)*TJ <= blockDim
    int CHP;      // chip smem stride (rows), >= every point's ch rounded up to 16
    int CWM;      // largest chip width
    int BC;       // chip columns staged at a time (== CWM: the whole chip once per point)
    int WS;       // window smem stride (floats): even, WS/2 odd, >= TI + CHP
    int PHS;      // prefix-table stride (entries), >= TI + largest ch
    int NRS;      // surface smem stride (rows), >= largest nr
    int NCM;      // largest nc
    unsigned off_win, off_ph1, off_ph2, off_surf, off_red;  // byte offsets, chip at 0
    DevOutputs out;
    int* sub_count;
    int64_t* sub_point;
    int32_t* sub_origin;
    float* sub_patch;
    float* surf_out;  // optional: each point's surface, NRS x NCM floats per point
    unsigned long long* flops;  // optional: algorithmic FLOPs of the surfaces computed
    unsigned off_surf2;  // rotation search: the best surface so far (NRS x NCM floats)
    int GTI, GTJ;        // k_corr_fp, Float32: the surface tile k_corr would take
    Rotation rot;        // rotation search angles (k_corr<T, true> only)
};
static_assert(sizeof(CorrArgs) <= 4096, "k_corr's arguments must fit the 4 KB parameter space");

template <typename T>
__device__ __forceinline__ double pixel(const T* img, int64_t nrows, int64_t ncols, int64_t r,
                                        int64_t c) {
    if (r < 0 || r >= nrows || c < 0 || c >= ncols) return 0.0;
    return static_cast<double>(img[r + c * nrows]);
}

template <typename PH>
__device__ __forceinline__ PH ph_of(float w);
template <>
__device__ __forceinline__ uint32_t ph_of<uint32_t>(float w) {
    return static_cast<uint32_t>(w);
}

// _rotate_chip (src/track.jl:377-409) at 0-based chip element (a, b) of a ch x cw chip whose
// first element is image element (chip_r, chip_c): the source point by the inverse rotation
// about the chip centre ((ch + 1) / 2, (cw + 1) / 2, 1-based), FP64 bilinear from its four
// neighbours, zero when one of them falls outside the chip, rounded to Float32. Each
// operation is rounded separately, in the reference's order (no contraction).
template <typename T>
__device__ __forceinline__ float rotated_sample(const T* sec, int64_t nrows, int64_t ncols,
                                                int64_t chip_r, int64_t chip_c, int ch, int cw,
                                                int a, int b, double sn, double cs) {
    const double yc = static_cast<double>(ch + 1) * 0.5, xc = static_cast<double>(cw + 1) * 0.5;
    const double dy = static_cast<double>(a + 1) - yc, dx = static_cast<double>(b + 1) - xc;
    const double sy = __dadd_rn(__dadd_rn(yc, __dmul_rn(cs, dy)), __dmul_rn(sn, dx));
    const double sx = __dadd_rn(__dsub_rn(xc, __dmul_rn(sn, dy)), __dmul_rn(cs, dx));
    const double fi = floor(sy), fj = floor(sx);
    if (!(fi >= 1.0 && fj >= 1.0 && fi + 1.0 <= static_cast<double>(ch) &&
          fj + 1.0 <= static_cast<double>(cw)))
        return 0.0f;
    const int i0 = static_cast<int>(fi), j0 = static_cast<int>(fj);  // 1-based
    const double fy = __dsub_rn(sy, fi), fx = __dsub_rn(sx, fj);
    const double v00 = pixel(sec, nrows, ncols, chip_r + i0 - 1, chip_c + j0 - 1);
    const double v10 = pixel(sec, nrows, ncols, chip_r + i0, chip_c + j0 - 1);
    const double v01 = pixel(sec, nrows, ncols, chip_r + i0 - 1, chip_c + j0);
    const double v11 = pixel(sec, nrows, ncols, chip_r + i0, chip_c + j0);
    const double gx = __dsub_rn(1.0, fx), gy = __dsub_rn(1.0, fy);
    const double top = __dadd_rn(__dmul_rn(gx, v00), __dmul_rn(fx, v01));
    const double bot = __dadd_rn(__dmul_rn(gx, v10), __dmul_rn(fx, v11));
    return __double2float_rn(__dadd_rn(__dmul_rn(gy, top), __dmul_rn(fy, bot)));
}

// ROT: the rotation search. Its chips are Float32 (turned chips are resampled), so the
// numerator takes the FP32/FP64 branch and the box sums are FP64 for every element type.
template <typename T, bool ROT>
__global__ void __launch_bounds__(kCorrThreads, 2) k_corr(const CorrArgs A) {
    typedef Traits<T> Tr;
    constexpr bool RAW = Tr::raw && !ROT;
    typedef typename std::conditional<ROT, double, typename Tr::ph_t>::type PH;
    extern __shared__ __align__(16) unsigned char smem[];
    float* s_chip = reinterpret_cast<float*>(smem);
    float* s_win = reinterpret_cast<float*>(smem + A.off_win);
    PH* s_ph1 = reinterpret_cast<PH*>(smem + A.off_ph1);
    PH* s_ph2 = reinterpret_cast<PH*>(smem + A.off_ph2);
    float* s_surf = reinterpret_cast<float*>(smem + A.off_surf);
    float* s_surf2 = reinterpret_cast<float*>(smem + A.off_surf2);
    double* s_red = reinterpret_cast<double*>(smem + A.off_red);
    __shared__ int s_slot;

    const int tid = threadIdx.x, bd = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = bd >> 5;
    const T* ref = static_cast<const T*>(A.ref);
    const T* sec = static_cast<const T*>(A.sec);
    const int64_t NR = A.nrows + 2 * A.pady, NC = A.ncols + 2 * A.padx;
    const double shx = static_cast<double>(A.padx) + 0.5;
    const double shy = static_cast<double>(A.pady) + 0.5;

    for (int64_t k = blockIdx.x; k < A.pts.n; k += gridDim.x) {
        __syncthreads();  // shared buffers of the previous point are no longer read
        const int64_t prx = A.pts.rx[k], pry = A.pts.ry[k];
        if (!(prx > 0 && pry > 0)) continue;  // issearchable (src/points.jl:116-117)

        // Geometry in padded 1-based coordinates (src/track.jl:207-210, src/points.jl:358-395).
        const double xs = A.pts.x[k] + shx, ys = A.pts.y[k] + shy;
        const int64_t hx = A.pts.csx[k] / 2, hy = A.pts.csy[k] / 2;
        const int64_t ccx = static_cast<int64_t>(floor(__dsub_rn(xs, A.pts.dx0[k])));
        const int64_t ccy = static_cast<int64_t>(floor(__dsub_rn(ys, A.pts.dy0[k])));
        const int64_t wcx = static_cast<int64_t>(floor(xs)), wcy = static_cast<int64_t>(floor(ys));
        const int64_t cr0 = ccy - hy, cr1 = ccy + hy - 1, cc0 = ccx - hx, cc1 = ccx + hx - 1;
        const int64_t wr0 = wcy - hy - pry, wr1 = wcy + hy + pry - 2;
        const int64_t wc0 = wcx - hx - prx, wc1 = wcx + hx + prx - 2;
        // checkbounds (src/track.jl:271-272): an empty range is always in bounds.
        const bool chip_in = (cr1 < cr0 || cc1 < cc0) ||
                             (cr0 >= 1 && cr1 <= NR && cc0 >= 1 && cc1 <= NC);
        const bool win_in = (wr1 < wr0 || wc1 < wc0) ||
                            (wr0 >= 1 && wr1 <= NR && wc0 >= 1 && wc1 <= NC);
        if (!chip_in || !win_in) continue;
        const int ch = static_cast<int>(2 * hy), cw = static_cast<int>(2 * hx);
        const int nr = static_cast<int>(2 * pry), nc = static_cast<int>(2 * prx);
        if (ch <= 0 || cw <= 0) continue;  // an empty chip has no valid pixel
        if (ch > A.CHP || cw > A.CWM || nr > A.NRS || nc > A.NCM) continue;  // not sized for
        const int64_t chip_r = cr0 - 1 - A.pady, chip_c = cc0 - 1 - A.padx;
        const int64_t win_r = wr0 - 1 - A.pady, win_c = wc0 - 1 - A.padx;

        // _any_valid over the chip (src/track.jl:416-421).
        int any = 0;
        for (int e = tid; e < ch * cw; e += bd) {
            const int64_t r = chip_r + e % ch, c = chip_c + e / ch;
            if (r >= 0 && r < A.nrows && c >= 0 && c < A.ncols && A.valid[r + c * A.nrows])
                any = 1;
        }
        if (!__syncthreads_or(any)) continue;
        if (tid == 0) A.out.searched[k] = 1;

        // One correlation, or with the rotation search one per angle with the best surface kept
        // (_correlate_rotations!, src/track.jl:313-350): an angle whose turned chip is
        // degenerate is skipped, and a surface replaces the best so far only if its maximum is
        // strictly larger. s_cur receives each surface; s_best is the best one so far.
        const int nang = ROT ? A.rot.count : 1;
        float* s_cur = s_surf;
        float* s_best = s_surf2;
        float bestpk = -INFINITY;
        unsigned long long best = 0ull;
        bool found = false;
        for (int ia = 0; ia < nang; ++ia) {
            const bool turn = ROT && A.rot.turn[ia];
            const double rsn = ROT ? A.rot.sn[ia] : 0.0, rcs = ROT ? A.rot.cs[ia] : 1.0;

            // prepare_chip! (src/correlate.jl:423-453): FP64 mean, then the mean-removed
            // Float32 copy, its FP64 sum of squares, and the FP64 sum of the rounded copy. With
            // the rotation search the chip (turned, or itself at angle 0) is first staged as
            // Float32 values.
            double st[1] = {0.0};
            for (int e = tid; e < ch * cw; e += bd) {
                const int a = e % ch, b = e / ch;
                double v;
                if (turn) {
                    v = static_cast<double>(rotated_sample(sec, A.nrows, A.ncols, chip_r,
                                                           chip_c, ch, cw, a, b, rsn, rcs));
                } else {
                    v = pixel(sec, A.nrows, A.ncols, chip_r + a, chip_c + b);
                }
                if (ROT) s_chip[b * A.CHP + a] = static_cast<float>(v);
                st[0] = __dadd_rn(st[0], v);
            }
            block_sum_f64<1>(st, s_red);
            const double nn = static_cast<double>(ch * cw);
            const double mean = __ddiv_rn(st[0], nn);
            const int chp = (ch + kUA - 1) & ~(kUA - 1);
            double acc2[2] = {0.0, 0.0};
            for (int e = tid; e < chp * cw; e += bd) {
                const int a = e % chp, b = e / chp;
                float staged = 0.0f;
                if (a < ch) {
                    const double v = ROT ? static_cast<double>(s_chip[b * A.CHP + a])
                                         : pixel(sec, A.nrows, A.ncols, chip_r + a, chip_c + b);
                    const double d = __dsub_rn(v, mean);
                    const float df = __double2float_rn(d);
                    acc2[0] = __dadd_rn(acc2[0], __dmul_rn(d, d));
                    acc2[1] = __dadd_rn(acc2[1], static_cast<double>(df));
                    staged = RAW ? static_cast<float>(v) : df;
                }
                if (A.BC >= cw) s_chip[b * A.CHP + a] = staged;
            }
            block_sum_f64<2>(acc2, s_red);
            const double sq = acc2[0], sumd = acc2[1];
            if (!(sq > __dmul_rn(__dmul_rn(DBL_EPSILON, static_cast<double>(ch)),
                                 static_cast<double>(cw))))
                continue;  // degenerate chip: no surface at this angle (src/track.jl:286, 326)
            const double cnorm = __dsqrt_rn(sq);
            // Centring constant for the window of non-raw element types.
            double cshift = 0.0;
            if (!RAW) cshift = Tr::integer ? rint(mean) : static_cast<double>(__double2float_rn(mean));

            const int F = RAW ? max(1, 16777216 / (chp * 65025)) : 2;
            for (int ti = 0; ti < nr; ti += A.TI) {
                const int trows = min(A.TI, nr - ti);
                const int trows_p = (trows + kMI - 1) / kMI * kMI;
                const int srows = trows_p + chp;  // staged window rows (<= WS)
                const int wrows = trows + ch - 1; // rows the box sums use
                for (int tj = 0; tj < nc; tj += A.TJ) {
                    const int tcols = min(A.TJ, nc - tj);
                    // Numerator item = (row group, column), kMI surface rows per thread; its
                    // partial sums run across the chip-column chunks.
                    const int ig = tid / A.TJ, jl = tid % A.TJ;
                    const bool item = ig * kMI < trows && jl < tcols;
                    const int il = ig * kMI;
                    float acc[kMI];
                    double acc64[kMI];
    #pragma unroll
                    for (int m = 0; m < kMI; ++m) { acc[m] = 0.0f; acc64[m] = 0.0; }
                    int fc = 0;
                    for (int b0 = 0; b0 < cw; b0 += A.BC) {
                        const int bc = min(A.BC, cw - b0);
                        const int xcols = tcols + bc - 1;
                        __syncthreads();
                        if (!ROT && A.BC < cw) {
                            // This chunk of chip columns, staged as in the unchunked case.
                            for (int e = tid; e < chp * bc; e += bd) {
                                const int a = e % chp, bl = e / chp;
                                float staged = 0.0f;
                                if (a < ch) {
                                    const double v = pixel(sec, A.nrows, A.ncols, chip_r + a, chip_c + b0 + bl);
                                    staged = RAW ? static_cast<float>(v)
                                                     : __double2float_rn(__dsub_rn(v, mean));
                                }
                                s_chip[bl * A.CHP + a] = staged;
                            }
                        }
                        // Stage the window block column-major, zero outside the image and below
                        // the window's last row.
                        for (int e = tid; e < xcols * srows; e += bd) {
                            const int r = e % srows, x = e / srows;
                            float v = 0.0f;
                            if (r < wrows) {
                                const double pv =
                                    pixel(ref, A.nrows, A.ncols, win_r + ti + r, win_c + tj + b0 + x);
                                v = RAW ? static_cast<float>(pv)
                                            : __double2float_rn(__dsub_rn(pv, cshift));
                            }
                            s_win[x * A.WS + r] = v;
                        }
                        __syncthreads();
                        // Per-window sums of W and W^2 over the chunk's columns for every row the
                        // tile uses (integral_both!, src/integral.jl:141-170), added at slot r + 1.
                        // They sum the image values themselves: a non-raw staged window is shifted
                        // by cshift for the numerator's FP32 products, and adding the shift back
                        // restores the image value (exactly for zero padding, within one Float32
                        // rounding otherwise). A window without variance -- all zero padding, or
                        // flat integer data -- then sums to exactly zero variance, as the
                        // reference's FP64 integral images do; expanding shifted sums instead
                        // leaves a rounding residue that the numerator's FP32 error turns into
                        // arbitrary correlation values.
                        auto wv = [&](int idx) -> PH {
                            if constexpr (RAW) {
                                return ph_of<PH>(s_win[idx]);
                            } else {
                                return static_cast<PH>(
                                    __dadd_rn(static_cast<double>(s_win[idx]), cshift));
                            }
                        };
                        const int nseg = (tcols + 15) >> 4;
                        for (int task = tid; task < wrows * nseg; task += bd) {
                            const int r = task % wrows, seg = task / wrows;
                            const int j0s = seg << 4, j1s = min(j0s + 16, tcols);
                            PH h1 = 0, h2 = 0;
                            int nz = 0;  // Float32: values other than zero
                            for (int b = 0; b < bc; ++b) {
                                const PH w = wv((j0s + b) * A.WS + r);
                                h1 = h1 + w;
                                h2 = h2 + w * w;
                                if (!Tr::integer) nz += w != PH(0);
                            }
                            for (int jj = j0s; jj < j1s; ++jj) {
                                if (jj > j0s) {
                                    const PH wo = wv((jj - 1) * A.WS + r);
                                    const PH wn = wv((jj - 1 + bc) * A.WS + r);
                                    h1 = h1 + wn - wo;
                                    h2 = h2 + wn * wn - wo * wo;
                                    if (!Tr::integer) nz += (wn != PH(0)) - (wo != PH(0));
                                }
                                // A row of zeros sums to zero: sliding FP64 sums of Float32 values may
                                // miss it by a rounding, which would stand for a variance.
                                if (!Tr::integer && nz == 0 && h2 == h2) h1 = h2 = PH(0);
                                PH* p1 = &s_ph1[jj * A.PHS + r + 1];
                                PH* p2 = &s_ph2[jj * A.PHS + r + 1];
                                *p1 = b0 == 0 ? h1 : *p1 + h1;
                                *p2 = b0 == 0 ? h2 : *p2 + h2;
                            }
                        }
                        // The chunk's share of the numerator.
                        if (item) {
                            const float* wbase = s_win + jl * A.WS + il;
                            for (int b = 0; b < bc; ++b) {
                                const float* wc = wbase + b * A.WS;
                                const float* cc = s_chip + b * A.CHP;
                                for (int a0 = 0; a0 < chp; a0 += kUA) {
                                    float c[kUA];
                                    float w[kUA + kMI];
    #pragma unroll
                                    for (int q = 0; q < kUA / 4; ++q) {
                                        const float4 v = *reinterpret_cast<const float4*>(cc + a0 + 4 * q);
                                        c[4 * q] = v.x; c[4 * q + 1] = v.y; c[4 * q + 2] = v.z; c[4 * q + 3] = v.w;
                                    }
    #pragma unroll
                                    for (int q = 0; q < (kUA + kMI) / 2; ++q) {
                                        const float2 v = *reinterpret_cast<const float2*>(wc + a0 + 2 * q);
                                        w[2 * q] = v.x; w[2 * q + 1] = v.y;
                                    }
    #pragma unroll
                                    for (int a = 0; a < kUA; ++a)
    #pragma unroll
                                        for (int m = 0; m < kMI; ++m) acc[m] = fmaf(c[a], w[m + a], acc[m]);
                                }
                                if (++fc == F) {
    #pragma unroll
                                    for (int m = 0; m < kMI; ++m) {
                                        acc64[m] = __dadd_rn(acc64[m], static_cast<double>(acc[m]));
                                        acc[m] = 0.0f;
                                    }
                                    fc = 0;
                                }
                            }
                        }
                    }
                    __syncthreads();
                    // Exclusive prefix down each column: ph[jl][q] = sum_{r<q} H[r]. Float32: in row
                    // order, a thread a column and table, so that rows of zeros leave it as it was and
                    // windows of zeros keep exactly zero variance (a scan adds each row's sum in an
                    // order of its own). Integer types (exact sums): by warp scans.
                    if constexpr (!Tr::integer) {
                        for (int t = tid; t < 2 * tcols; t += bd) {
                            PH* p = t < tcols ? s_ph1 + t * A.PHS : s_ph2 + (t - tcols) * A.PHS;
                            PH c = 0, v[4];  // four rows loaded ahead of their sums' stores
                            p[0] = PH(0);
                            int q = 1;
                            for (; q + 3 <= wrows; q += 4) {
    #pragma unroll
                                for (int u = 0; u < 4; ++u) v[u] = p[q + u];
    #pragma unroll
                                for (int u = 0; u < 4; ++u) p[q + u] = c = c + v[u];
                            }
                            for (; q <= wrows; ++q) p[q] = c = c + p[q];
                        }
                    } else
                    for (int jw = warp; jw < tcols; jw += nwarps) {
                        PH c1 = 0, c2 = 0;
                        for (int q = 1; q <= wrows; q += 32) {
                            const int idx = q + lane;
                            PH v1 = idx <= wrows ? s_ph1[jw * A.PHS + idx] : PH(0);
                            PH v2 = idx <= wrows ? s_ph2[jw * A.PHS + idx] : PH(0);
                            v1 = warp_inclusive_scan(v1) + c1;
                            v2 = warp_inclusive_scan(v2) + c2;
                            if (idx <= wrows) {
                                s_ph1[jw * A.PHS + idx] = v1;
                                s_ph2[jw * A.PHS + idx] = v2;
                            }
                            c1 = __shfl_sync(kFull, v1, 31);
                            c2 = __shfl_sync(kFull, v2, 31);
                        }
                        if (lane == 0) {
                            s_ph1[jw * A.PHS] = PH(0);
                            s_ph2[jw * A.PHS] = PH(0);
                        }
                    }
                    __syncthreads();

                    if (item) {
    #pragma unroll
                        for (int m = 0; m < kMI; ++m)
                            acc64[m] = __dadd_rn(acc64[m], static_cast<double>(acc[m]));

                        // Normalisation (src/correlate.jl:591-600, 624-628).
    #pragma unroll
                        for (int m = 0; m < kMI; ++m) {
                            const int ir = il + m;
                            if (ir < trows) {
                                const PH p1 = s_ph1[jl * A.PHS + ir + ch] - s_ph1[jl * A.PHS + ir];
                                const PH p2 = s_ph2[jl * A.PHS + ir + ch] - s_ph2[jl * A.PHS + ir];
                                const double s1 = static_cast<double>(p1);
                                const double s2 = static_cast<double>(p2);
                                const double num =
                                    RAW ? __dsub_rn(acc64[m], __dmul_rn(mean, s1))
                                        : __dadd_rn(acc64[m], __dmul_rn(cshift, sumd));
                                double den;
                                if (A.measure == AR_NCC) {
                                    den = __dmul_rn(cnorm, __dsqrt_rn(s2 > 0.0 ? s2 : 0.0));
                                } else {
                                    double wvar = __dsub_rn(s2, __ddiv_rn(__dmul_rn(s1, s1), nn));
                                    if (!(wvar > 0.0)) wvar = 0.0;
                                    den = __dmul_rn(cnorm, __dsqrt_rn(wvar));
                                }
                                const float sv = den > 0.0 ? __double2float_rn(__ddiv_rn(num, den)) : 0.0f;
                                s_cur[(ti + ir) + (tj + jl) * A.NRS] = sv;
                            }
                        }
                    }
                }
            }
            __syncthreads();
            if (A.flops && tid == 0)
                atomicAdd(A.flops, 2ull * static_cast<unsigned long long>(ch) * cw * nr * nc);

            // Integer peak (src/peak.jl:32-61), and the angle's maximum (src/track.jl:327-328).
            unsigned long long key = 0ull;
            for (int e = tid; e < nr * nc; e += bd) {
                const int i = e % nr, j = e / nr;
                const unsigned long long kk =
                    argmax_key(s_cur[i + j * A.NRS], static_cast<unsigned>(i * nc + j));
                key = kk > key ? kk : key;
            }
            key = block_max_u64(key, reinterpret_cast<unsigned long long*>(s_red));
            const float pk = key == 0ull ? NAN : key_value(key);
            if (!ROT || pk > bestpk) {
                bestpk = pk;
                best = key;
                float* t = s_best;
                s_best = s_cur;
                s_cur = t;
                found = true;
            }
        }
        if (!found) continue;  // every angle degenerate: searched, no measurement
        if (A.surf_out) {
            float* so = A.surf_out + k * static_cast<int64_t>(A.NRS) * A.NCM;
            for (int e = tid; e < nr * nc; e += bd) so[e] = s_best[(e % nr) + (e / nr) * A.NRS];
        }

        unsigned rm = 0;
        float pv = 0.0f;
        int pi = 0, pj = 0;
        if (key_decode(best, &rm, &pv)) {
            pi = static_cast<int>(rm / nc);
            pj = static_cast<int>(rm % nc);
        }
        if (A.up == 1 || nr < 5 || nc < 5) {
            // peak_offset (src/peak.jl:102-106) and the output write (src/track.jl:293-295).
            if (tid == 0) {
                const float v = s_best[pi + pj * A.NRS];
                A.out.dx[k] = __double2float_rn(
                    __dadd_rn(static_cast<double>(pj - static_cast<int>(prx)), A.pts.dx0[k]));
                A.out.dy[k] = __double2float_rn(
                    __dadd_rn(static_cast<double>(pi - static_cast<int>(pry)), A.pts.dy0[k]));
                A.out.corr[k] = v;
            }
        } else {
            // The clamped 5x5 patch of subpixel_peak (src/peak.jl:473-482), queued.
            const int pi0 = min(max(pi - 2, 0), max(nr - 5, 0));
            const int pj0 = min(max(pj - 2, 0), max(nc - 5, 0));
            if (tid == 0) s_slot = atomicAdd(A.sub_count, 1);
            __syncthreads();
            const int slot = s_slot;
            if (tid < 25) {
                const int a = tid % 5, b = tid / 5;
                A.sub_patch[static_cast<int64_t>(slot) * 25 + tid] =
                    s_best[(pi0 + a) + (pj0 + b) * A.NRS];
            }
            if (tid == 0) {
                A.sub_point[slot] = k;
                A.sub_origin[2 * slot] = pi0;
                A.sub_origin[2 * slot + 1] = pj0;
            }
        }
    }
}

// Optional phase timer (compiled in with -DAR_TC_PHASES, for profiling builds only): thread 0
// of each CTA accumulates clock64() cycles between the marks below, per phase, and adds them to
// g_tc_phase at exit; entry 15 counts the points that reached the output phase.
#ifdef AR_TC_PHASES
__device__ unsigned long long g_tc_phase[16];
#define TC_PHASE_INIT unsigned long long tcp_t = clock64(), tcp_acc[12] = {}, tcp_n = 0;
#define TC_PHASE(n)                              \
    if (tid == 0) {                              \
        const unsigned long long t_ = clock64(); \
        tcp_acc[n] += t_ - tcp_t;                \
        tcp_t = t_;                              \
    }
#define TC_PHASE_POINT \
    if (tid == 0) ++tcp_n;
#define TC_PHASE_FLUSH                                                           \
    if (tid == 0) {                                                              \
        for (int n_ = 0; n_ < 12; ++n_) atomicAdd(&g_tc_phase[n_], tcp_acc[n_]); \
        atomicAdd(&g_tc_phase[15], tcp_n);                                       \
    }
#else
#define TC_PHASE_INIT
#define TC_PHASE(n)
#define TC_PHASE_POINT
#define TC_PHASE_FLUSH
#endif

// ----------------------------------------------------------------------------------------------
// Direct FP32 correlation of UInt16, Int16 and Float32 imagery and of turned chips of any type,
// surfaces of one tile (k_corr_fp). The numerator of k_corr: the same FP32 sums of two chip columns'
// products, added in FP64 (in the same order, or part by part where the chip's columns are split over
// threads: then within a few FP64 roundings); but
//  * two surface columns per thread as packed FP32 pairs: the window is staged as pairs
//    (W[r, x], W[r, x + 1]), so one 64-bit load feeds a packed FMA whatever the row, and a product
//    pair costs one issue slot;
//  * even and odd window columns lie in separate halves, so that lanes on consecutive column pairs
//    read rows WS pairs apart (WS odd: 16 of them conflict-free), and the lanes take 16 column
//    pairs of a row group at a time as far as these go;
//  * where the column pairs and row groups do not fill the block, the chip's columns are split over
//    the free threads (whole two-column groups; the FP64 sums are added at the end);
//  * box sums from column sums of a few rows at a time, instead of tables of every window row, with
//    counts of non-zero values beside them, so that windows of zeros keep exactly zero variance;
//    each point's variance terms are kept (8 bytes a value), not its sums, and serve every angle of
//    an integer image;
//  * Float32 estimates of the surface, with the FP64 normalisation (src/correlate.jl:591-600) for
//    the candidates of the maximum and the patch only;
//  * NaN and infinite pixels of Float32 imagery show in the column sums, and such windows take a second
//    pass over them (fp_nonfinite).
// Bound: the FMA pipe takes two cycles for a packed warp instruction, 20.5 k cycles a point at chip
// 32 / radius 25 of the 46 k a point takes (30 k of products per CTA without a neighbour; the box
// sums, the window and the estimates around them are FP64 and load latency, which the other of
// the two CTAs per SM covers only in part). Measured, chip 32 / radius 25, against k_corr on the
// same pass: Float32 (14.6 k points) 3.00 -> 2.52 ms, UInt16 2.99 -> 2.50 ms, three angles on UInt8
// 11.84 -> 6.24 ms; chip 16 / radius 10 0.94 -> 0.85 ms; chip 48 / radius 30 5.08 -> 4.54 ms.
// Surfaces of more than one tile stay with k_corr.

// A pixel with zero padding from an address that is always valid, so that loads need no branch and
// several can be in flight.
template <typename T>
__device__ __forceinline__ T pixel_at(const T* img, int64_t nrows, int64_t ncols, int64_t r, int64_t c) {
    const int64_t rr = min(max(r, static_cast<int64_t>(0)), nrows - 1);
    const int64_t cc = min(max(c, static_cast<int64_t>(0)), ncols - 1);
    const T v = img[rr + cc * nrows];
    return r == rr && c == cc ? v : T(0);
}

// rotated_sample from the chip staged in shared memory (column b at raw + b * stride).
__device__ __forceinline__ float rotated_at(const float* raw, int stride, int ch, int cw, int a, int b,
                                            double sn, double cs) {
    const double yc = static_cast<double>(ch + 1) * 0.5, xc = static_cast<double>(cw + 1) * 0.5;
    const double dy = static_cast<double>(a + 1) - yc, dx = static_cast<double>(b + 1) - xc;
    const double sy = __dadd_rn(__dadd_rn(yc, __dmul_rn(cs, dy)), __dmul_rn(sn, dx));
    const double sx = __dadd_rn(__dsub_rn(xc, __dmul_rn(sn, dy)), __dmul_rn(cs, dx));
    const double fi = floor(sy), fj = floor(sx);
    const bool in = fi >= 1.0 && fj >= 1.0 && fi + 1.0 <= static_cast<double>(ch) &&
                    fj + 1.0 <= static_cast<double>(cw);
    const int i0 = in ? static_cast<int>(fi) : 1, j0 = in ? static_cast<int>(fj) : 1;  // 1-based
    // An even chip side has a second row and column, so the clamped indices are in the chip too.
    const float* q = raw + (j0 - 1) * stride + i0 - 1;
    const float p00 = q[0], p10 = q[1], p01 = q[stride], p11 = q[stride + 1];
    const double fy = __dsub_rn(sy, fi), fx = __dsub_rn(sx, fj);
    const double gx = __dsub_rn(1.0, fx), gy = __dsub_rn(1.0, fy);
    const double top = __dadd_rn(__dmul_rn(gx, static_cast<double>(p00)), __dmul_rn(fx, static_cast<double>(p01)));
    const double bot = __dadd_rn(__dmul_rn(gx, static_cast<double>(p10)), __dmul_rn(fx, static_cast<double>(p11)));
    return in ? __double2float_rn(__dadd_rn(__dmul_rn(gy, top), __dmul_rn(fy, bot))) : 0.0f;
}

__device__ __noinline__ float fp_exact(double num, double wvar, double cnorm) {
    const double den = __dmul_rn(cnorm, __dsqrt_rn(wvar));
    return den > 0.0 ? __double2float_rn(__ddiv_rn(num, den)) : 0.0f;
}

// The variance terms of a Float32 window with NaN or infinite pixels, as k_corr's tables have them: an
// FP64 sum that took in a NaN, or let an infinity go, is a NaN from there on. So such a pixel reaches
// every later row of its tile and every later column of its run of sixteen, and a variance that is not
// a number counts as none (the value is 0); the other terms take these pixels as zero. A thread a column, and
// out of line: few windows need it, and a second copy of the kernel's own sums cost the others more (8800 points
// at chip 16, radius 10: 593 us without the check, 603 with a copy, 598 so; over one NaN in 10 000 pixels
// 3.2 and 3.5 ms for 13 924 points of chip 32, radius 25, 4.1 with k_corr). `v` holds the column sums of four rows, then two rows a
// window column: the first with a NaN, the first with an infinity.
__device__ __noinline__ void fp_nonfinite(const float2* win, int XH, int WS, int ch, int cw, int nr, int nc,
                                          double shift, bool zncc, int TI, int TJ, double* v, double* wv, int NRS) {
    const int tid = threadIdx.x, XW = cw + nc - 1;  // at least as many threads as window columns
    const double nn = static_cast<double>(ch * cw);
    double* v2 = v + 4 * kCorrThreads;
    const float2* col = win + ((tid & 1) * XH + (tid >> 1)) * WS;
    auto value = [&](int r) {
        const float w = col[r].x;
        return fabsf(w) <= FLT_MAX ? __dadd_rn(static_cast<double>(w), shift) : 0.0;
    };
    double h1 = 0.0, h2 = 0.0;
    int nz = 0;  // values other than zero
    if (tid < XW)
        for (int r = 0; r < ch; ++r) {
            const double w = value(r);
            h1 += w;
            h2 += w * w;
            nz += w != 0.0;
        }
    for (int i0 = 0; i0 < nr; i0 += 4) {
        const int ni = min(4, nr - i0);
        for (int i = 0; i < ni && tid < XW; ++i) {
            v[i * kCorrThreads + tid] = nz ? h1 : 0.0;
            v2[i * kCorrThreads + tid] = nz ? h2 : 0.0;
            if (i0 + i + 1 == nr) break;  // no row below the window's last
            const double wo = value(i0 + i), wn = value(i0 + i + ch);
            h1 += wn - wo;
            h2 += wn * wn - wo * wo;
            nz += (wn != 0.0) - (wo != 0.0);
        }
        __syncthreads();
        for (int t = tid; t < ni * nc; t += kCorrThreads) {
            const int i = t / nc, j = t - i * nc;
            double s1 = 0.0, s2 = 0.0;
            for (int b = 0; b < cw; ++b) {
                s1 += v[i * kCorrThreads + j + b];
                s2 += v2[i * kCorrThreads + j + b];
            }
            const double var = zncc ? __dsub_rn(s2, __ddiv_rn(__dmul_rn(s1, s1), nn)) : s2;
            wv[j * NRS + i0 + i] = var > 0.0 ? var : 0.0;
        }
        __syncthreads();
    }
    int* first = reinterpret_cast<int*>(v);
    for (int ti = 0; ti < nr; ti += TI) {
        const int te = min(ti + TI, nr), none = te + ch;
        if (tid < XW) {
            int rn = none, ri = none;
            for (int r = ti; r < te + ch - 1 && rn == none; ++r) {
                const float w = fabsf(col[r].x);
                if (isnan(w)) rn = r;
                else if (!(w <= FLT_MAX)) ri = min(ri, r);
            }
            first[2 * tid] = rn;
            first[2 * tid + 1] = ri;
        }
        __syncthreads();
        if (tid < nc) {
            const int run = tid - ((tid % TJ) & 15);  // the sums along a row start afresh here
            int rn = none, ri = none;
            for (int x = run; x < tid + cw; ++x) {
                rn = min(rn, x < tid ? min(first[2 * x], first[2 * x + 1]) : first[2 * x]);
                if (x >= tid) ri = min(ri, first[2 * x + 1]);
            }
            const int rb = min(rn, ri);
            for (int i = max(ti, rb - ch + 1); i < te; ++i)
                wv[tid * NRS + i] = !zncc && i <= rb && i + ch <= rn ? INFINITY : 0.0;
        }
        __syncthreads();
    }
}

template <typename T, bool ROT>
__global__ void __launch_bounds__(kCorrThreads, 2) k_corr_fp(const CorrArgs A) {
    typedef Traits<T> Tr;
    extern __shared__ __align__(16) unsigned char smem[];
    float* s_chip = reinterpret_cast<float*>(smem);
    float2* s_win = reinterpret_cast<float2*>(smem + A.off_win);
    // Partial sums, after the products: in the window's place, or beside it where it stays.
    double* s_ex = reinterpret_cast<double*>(smem + A.off_surf2);
    // Box sums: exact integers for integer types (below 2^32 for UInt8), else FP64.
    typedef typename std::conditional<
        sizeof(T) == 1, uint32_t, typename std::conditional<Tr::integer, long long, double>::type>::type BS;
    BS* s_v1 = reinterpret_cast<BS*>(smem + A.off_ph1);
    BS* s_v2 = s_v1 + kCorrThreads * A.TI;
    float* s_raw = reinterpret_cast<float*>(smem + A.off_surf);  // rotation search: the chip itself
    double* s_wv = reinterpret_cast<double*>(smem + A.off_ph2);
    double* s_red = reinterpret_cast<double*>(smem + A.off_red);
    __shared__ long long s_field[2][8];
    __shared__ float s_top[kCorrThreads / 32], s_sec[kCorrThreads / 32];
    __shared__ int s_at[kCorrThreads / 32];
    __shared__ double s_pn[25], s_pw[25];  // the patch's numerators and variance terms
    __shared__ float s_pp[25], s_best[25];  // its values, and the best angle's

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int nwarps = kCorrThreads / 32;
    const T* ref = static_cast<const T*>(A.ref);
    const T* sec = static_cast<const T*>(A.sec);
    const int64_t NR = A.nrows + 2 * A.pady, NC = A.ncols + 2 * A.padx;
    const double shx = static_cast<double>(A.padx) + 0.5;
    const double shy = static_cast<double>(A.pady) + 0.5;

    // The next point's eight fields, copied into shared memory a point ahead.
    auto prefetch = [&](int64_t k, int b) {
        if (tid < 8 && k < A.pts.n) {
            const void* f[8] = {A.pts.x, A.pts.y, A.pts.rx, A.pts.ry, A.pts.dx0, A.pts.dy0, A.pts.csx, A.pts.csy};
            const void* src = f[0];
#pragma unroll
            for (int q = 1; q < 8; ++q) src = tid == q ? f[q] : src;
            tc::cp_async8(&s_field[b][tid], static_cast<const char*>(src) + 8 * k);
        }
        tc::cp_async_commit();
    };
    prefetch(blockIdx.x, 0);
    int fb = 0;
    TC_PHASE_INIT
    for (int64_t k = blockIdx.x; k < A.pts.n; k += gridDim.x, fb ^= 1) {
        tc::cp_async_wait_all();
        __syncthreads();  // the fields are here; buffers of the previous point are no longer read
        prefetch(k + gridDim.x, fb ^ 1);
        const long long* fld = s_field[fb];
        const int64_t prx = fld[2], pry = fld[3], csx = fld[6], csy = fld[7];
        const double px0 = __longlong_as_double(fld[0]), py0 = __longlong_as_double(fld[1]);
        const double dx0 = __longlong_as_double(fld[4]), dy0 = __longlong_as_double(fld[5]);
        if (!(prx > 0 && pry > 0)) continue;  // issearchable (src/points.jl:116-117)

        // Geometry in padded 1-based coordinates (src/track.jl:207-210, src/points.jl:358-395).
        const double xs = px0 + shx, ys = py0 + shy;
        const int64_t hx = csx / 2, hy = csy / 2;
        const int64_t ccx = static_cast<int64_t>(floor(__dsub_rn(xs, dx0)));
        const int64_t ccy = static_cast<int64_t>(floor(__dsub_rn(ys, dy0)));
        const int64_t wcx = static_cast<int64_t>(floor(xs)), wcy = static_cast<int64_t>(floor(ys));
        const int64_t cr0 = ccy - hy, cr1 = ccy + hy - 1, cc0 = ccx - hx, cc1 = ccx + hx - 1;
        const int64_t wr0 = wcy - hy - pry, wr1 = wcy + hy + pry - 2;
        const int64_t wc0 = wcx - hx - prx, wc1 = wcx + hx + prx - 2;
        // checkbounds (src/track.jl:271-272): an empty range is always in bounds.
        const bool chip_in = (cr1 < cr0 || cc1 < cc0) ||
                             (cr0 >= 1 && cr1 <= NR && cc0 >= 1 && cc1 <= NC);
        const bool win_in = (wr1 < wr0 || wc1 < wc0) ||
                            (wr0 >= 1 && wr1 <= NR && wc0 >= 1 && wc1 <= NC);
        if (!chip_in || !win_in) continue;
        const int ch = static_cast<int>(2 * hy), cw = static_cast<int>(2 * hx);
        const int nr = static_cast<int>(2 * pry), nc = static_cast<int>(2 * prx);
        if (ch <= 0 || cw <= 0) continue;  // an empty chip has no valid pixel
        if (ch > A.CHP || cw > A.CWM || nr > A.NRS || nc > A.NCM) continue;  // not sized for
        const int64_t chip_r = cr0 - 1 - A.pady, chip_c = cc0 - 1 - A.padx;
        const int64_t win_r = wr0 - 1 - A.pady, win_c = wc0 - 1 - A.padx;
        const int chp = (ch + kUA - 1) & ~(kUA - 1);
        const double nn = static_cast<double>(ch * cw);

        // This thread's share of the products: column pair p, row group g, part `part` of the
        // chip's columns.
        const int npair = nc >> 1, ngrp = (nr + kMI - 1) / kMI, items = npair * ngrp;
        int split = 1;
        while (2 * split * items <= kCorrThreads && 4 * split <= cw && split < 8) split *= 2;
        const int part = tid / items, it = tid - part * items;
        const int npf = npair & ~15, itr = it - npf * ngrp, npr = max(npair - npf, 1);
        const int g = itr < 0 ? it / npf : itr / npr;
        const int p = itr < 0 ? it - g * npf : npf + itr - g * npr, il = g * kMI;
        const bool active = part < split;
        const int XW = cw + nc - 1, XH = (A.CWM + A.NCM) >> 1;

        const int nang = ROT ? A.rot.count : 1;
        float bestpk = -INFINITY;
        bool found = false, have_var = false, skip = false, staged = false;
        float staged_cs = 0.0f;
        int pi0 = 0, pj0 = 0;
        const bool single = A.up == 1 || nr < 5 || nc < 5;
        for (int ia = 0; ia < nang; ++ia) {
            const bool turn = ROT && A.rot.turn[ia];
            const double rsn = ROT ? A.rot.sn[ia] : 0.0, rcs = ROT ? A.rot.cs[ia] : 1.0;

            // prepare_chip! (src/correlate.jl:423-453): FP64 mean, then the mean-removed Float32
            // copy, its FP64 sum of squares, and the FP64 sum of the rounded copy. The values are
            // first staged as Float32 (exact for every type).
            // The first angle loads the chip, with _any_valid over it (src/track.jl:416-421); the
            // rotation search keeps it and turns it from shared memory.
            double st[1] = {0.0};
            int any = 0;
            if (ia == 0) {
                float* dst = ROT ? s_raw : s_chip;
                for (int a = lane; a < ch; a += 32)
                    for (int b0 = warp; b0 < cw; b0 += 4 * nwarps) {
                        float v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int64_t r = chip_r + a, c = chip_c + min(b0 + u * nwarps, cw - 1);
                            any |= pixel_at(A.valid, A.nrows, A.ncols, r, c);
                            v[u] = static_cast<float>(pixel_at(sec, A.nrows, A.ncols, r, c));
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (b0 + u * nwarps < cw) {
                                dst[(b0 + u * nwarps) * A.CHP + a] = v[u];
                                if (!ROT) st[0] = __dadd_rn(st[0], static_cast<double>(v[u]));
                            }
                    }
            }
            if (ia == 0) {
                if (!__syncthreads_or(any)) {
                    skip = true;
                    break;
                }
                if (tid == 0) A.out.searched[k] = 1;
            }
            if constexpr (ROT) {
                for (int b = warp; b < cw; b += nwarps)
                    for (int a = lane; a < ch; a += 32) {
                        const float v = turn ? rotated_at(s_raw, A.CHP, ch, cw, a, b, rsn, rcs)
                                             : s_raw[b * A.CHP + a];
                        s_chip[b * A.CHP + a] = v;
                        st[0] = __dadd_rn(st[0], static_cast<double>(v));
                    }
            }
            block_sum_f64<1>(st, s_red);
            TC_PHASE(0)
            const double mean = __ddiv_rn(st[0], nn);
            double acc2[2] = {0.0, 0.0};
            for (int b = warp; b < cw; b += nwarps)
                for (int a = lane; a < chp; a += 32) {
                    float df = 0.0f;
                    if (a < ch) {
                        const double d = __dsub_rn(static_cast<double>(s_chip[b * A.CHP + a]), mean);
                        df = __double2float_rn(d);
                        acc2[0] = __dadd_rn(acc2[0], __dmul_rn(d, d));
                        acc2[1] = __dadd_rn(acc2[1], static_cast<double>(df));
                    }
                    s_chip[b * A.CHP + a] = df;
                }
            block_sum_f64<2>(acc2, s_red);
            const double sq = acc2[0], sumd = acc2[1];
            if (!(sq > __dmul_rn(__dmul_rn(DBL_EPSILON, static_cast<double>(ch)),
                                 static_cast<double>(cw))))
                continue;  // degenerate chip: no surface at this angle (src/track.jl:286, 326)
            const double cnorm = __dsqrt_rn(sq);
            TC_PHASE(1)
            // Centring constant of the window: a Float32 value, so that W - c rounds once (the
            // difference is exact for integer types).
            const float cs = Tr::integer ? static_cast<float>(rint(mean)) : __double2float_rn(mean);
            const double cshift = static_cast<double>(cs);

            // The window of an integer image is staged for the first angle; another angle's shift is
            // then added to it (exactly).
            const bool restage = !Tr::integer || !staged;
            if (!restage && cs != staged_cs) {
                const int wrows = nr + ch - 1;
                const float d = staged_cs - cs;
                for (int x = warp; x < XW; x += nwarps) {
                    float2* col = s_win + ((x & 1) * XH + (x >> 1)) * A.WS;
                    const float dn = x + 1 < XW ? d : 0.0f;
#pragma unroll 4
                    for (int r = lane; r < wrows; r += 32) {
                        const float2 w = col[r];
                        col[r] = make_float2(w.x + d, w.y + dn);
                    }
                }
            }
            staged = true;
            staged_cs = cs;
            // The window, shifted, zero-padded outside the image before the shift and below its last
            // row after it: a warp takes a run of columns, lanes the rows, each lane keeping the
            // column before.
            if (restage) {
                const int wrows = nr + ch - 1, srows = ngrp * kMI + chp;
                const int run = (XW + nwarps - 1) / nwarps;
                const int x0 = warp * run, x1 = min(x0 + run, XW);
                // Three row chunks of twelve columns in flight.
                for (int rb = 0; rb < srows && x0 < x1; rb += 96) {
                    const T* row[3];
                    bool rin[3], live[3];
                    float prev[3];
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        const int r = rb + 32 * q + lane;
                        const int64_t ir = win_r + r;
                        live[q] = r < wrows;
                        rin[q] = live[q] && ir >= 0 && ir < A.nrows;
                        row[q] = ref + (rin[q] ? ir : 0);
                    }
                    // Column x of row chunk q, zero outside the image, before the shift; from an
                    // address that is always valid.
                    auto load = [&](int x, int q) {
                        const int64_t c = win_c + x;
                        const bool in = c >= 0 && c < A.ncols;
                        const T v = row[q][(in ? c : 0) * A.nrows];
                        return in && rin[q] ? static_cast<float>(v) : 0.0f;
                    };
                    auto shifted = [&](float v, int x, int q) {
                        return live[q] && x < XW ? __fsub_rn(v, cs) : 0.0f;
                    };
#pragma unroll
                    for (int q = 0; q < 3; ++q) prev[q] = load(x0, q);
#pragma unroll
                    for (int q = 0; q < 3; ++q) prev[q] = shifted(prev[q], x0, q);
                    for (int x = x0; x < x1; x += 12) {
                        float v[3][12];
#pragma unroll
                        for (int u = 0; u < 12; ++u)
#pragma unroll
                            for (int q = 0; q < 3; ++q) v[q][u] = load(x + u + 1, q);
#pragma unroll
                        for (int u = 0; u < 12; ++u) {
                            const int xx = x + u;
                            float2* dst = s_win + ((xx & 1) * XH + (xx >> 1)) * A.WS + rb + lane;
#pragma unroll
                            for (int q = 0; q < 3; ++q) {
                                const float next = shifted(v[q][u], xx + 1, q);
                                if (xx < x1 && rb + 32 * q + lane < srows) dst[32 * q] = make_float2(prev[q], next);
                                prev[q] = next;
                            }
                        }
                    }
                }
            }
            __syncthreads();
            TC_PHASE(2)

            // Box sums of W and W^2 (integral_both!, boxsum, src/integral.jl:141-170, 244-247) in
            // FP64 from the image values (the staged ones plus the shift: exact for integer types
            // and zero padding) and each value's variance term max(s2 - s1 s1 / n, 0) (NCC: max(s2,
            // 0)). A thread slides a column's sums of ch rows down one of `nseg` segments of the
            // surface rows; A.TI rows of each segment at a time go to shared memory, where a task
            // sums cw columns for five neighbouring values. The counts of non-zero values keep
            // windows of zeros at exactly zero, which sliding FP64 sums would miss by a rounding.
            if (!have_var) {
                const int nseg = max(1, min(8, kCorrThreads / XW));
                const int seglen = (nr + nseg - 1) / nseg;
                const int seg = tid / XW, x = tid - seg * XW;
                const bool sums = seg < nseg;
                const int i0 = seg * seglen, i1 = min(i0 + seglen, nr);
                const float2* col = s_win + ((x & 1) * XH + (x >> 1)) * A.WS;
                // An image value from its staged one; integers by way of 1.5 x 2^23, whose last bits
                // hold them.
                auto value = [&](float v) -> BS {
                    if constexpr (Tr::integer) {
                        return static_cast<BS>(__float_as_int(__fadd_rn(__fadd_rn(v, cs), 12582912.0f)) - 0x4B400000);
                    } else {
                        return __dadd_rn(static_cast<double>(v), cshift);
                    }
                };
                BS h1 = 0, h2 = 0;
                int nz = 1;  // non-zero values (Float32: the others' sums are exact)
                if (sums && i0 < i1) {
                    BS a1[4] = {0, 0, 0, 0}, a2[4] = {0, 0, 0, 0};
                    if (!Tr::integer) nz = 0;
                    int a = 0;
#pragma unroll 2
                    for (; a + 4 <= ch; a += 4)
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const BS w = value(col[i0 + a + u].x);
                            a1[u] += w;
                            a2[u] += w * w;
                            if (!Tr::integer) nz += w != BS(0);
                        }
                    for (; a < ch; ++a) {
                        const BS w = value(col[i0 + a].x);
                        a1[0] += w;
                        a2[0] += w * w;
                        if (!Tr::integer) nz += w != BS(0);
                    }
                    h1 = (a1[0] + a1[1]) + (a1[2] + a1[3]);
                    h2 = (a2[0] + a2[1]) + (a2[2] + a2[3]);
                }
                const bool p2 = ((ch * cw) & (ch * cw - 1)) == 0;
                const double inv = 1.0 / nn;
                const int slots = nseg * A.TI, jtasks = slots * ((nc + 4) / 5);
                for (int t0 = 0; t0 < seglen; t0 += A.TI) {
                    // Four rows at a time, their values loaded before the sums are stored (the stores
                    // may alias the window as far as the compiler knows).
                    for (int t = 0; sums && t < A.TI; t += 4) {
                        const int i = i0 + t0 + t;
                        if (i >= i1) break;
                        float fo[4], fn[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            fo[u] = col[min(i + u, i1 - 1)].x;
                            fn[u] = col[min(i + u, i1 - 1) + ch].x;
                        }
                        BS e1[4], e2[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            e1[u] = nz ? h1 : BS(0);
                            e2[u] = nz ? h2 : BS(0);
                            const BS wo = value(fo[u]), wn = value(fn[u]);
                            h1 += wn - wo;
                            h2 += wn * wn - wo * wo;
                            if (!Tr::integer) nz += (wn != BS(0)) - (wo != BS(0));
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (t + u < A.TI && i + u < i1) {
                                s_v1[(seg * A.TI + t + u) * XW + x] = e1[u];
                                s_v2[(seg * A.TI + t + u) * XW + x] = e2[u];
                            }
                    }
                    __syncthreads();
                    for (int task = tid; task < jtasks; task += kCorrThreads) {
                        const int jg = task / slots, sl = task - jg * slots;
                        const int sg = sl / A.TI, t = t0 + sl - sg * A.TI;
                        const int i = sg * seglen + t, j0 = 5 * jg;
                        if (t >= seglen || i >= nr) continue;
                        const BS* v1 = s_v1 + sl * XW + j0;
                        const BS* v2 = s_v2 + sl * XW + j0;
                        BS a1[4] = {0, 0, 0, 0}, a2[4] = {0, 0, 0, 0};
                        int n = Tr::integer ? 1 : 0, b = 0;
#pragma unroll 2
                        for (; b + 4 <= cw; b += 4)
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const BS w2 = v2[b + u];
                                a1[u] += v1[b + u];
                                a2[u] += w2;
                                if (!Tr::integer) n += w2 != BS(0);
                            }
                        for (; b < cw; ++b) {
                            a1[0] += v1[b];
                            a2[0] += v2[b];
                            if (!Tr::integer) n += v2[b] != BS(0);
                        }
                        BS g1[5], g2[5];
                        int ng[5];
                        g1[0] = (a1[0] + a1[1]) + (a1[2] + a1[3]);
                        g2[0] = (a2[0] + a2[1]) + (a2[2] + a2[3]);
                        ng[0] = n;
                        const int last = nc - 1 - j0;  // columns past the surface repeat its last one
#pragma unroll
                        for (int m = 1; m < 5; ++m) {
                            const int o = max(min(m, last) - 1, 0);
                            const BS o2 = v2[o], n2 = v2[o + cw];
                            g1[m] = g1[m - 1] + (v1[o + cw] - v1[o]);
                            g2[m] = g2[m - 1] + (n2 - o2);
                            ng[m] = ng[m - 1];
                            if (!Tr::integer) ng[m] += (n2 != BS(0)) - (o2 != BS(0));
                        }
#pragma unroll
                        for (int m = 0; m < 5; ++m) {
                            const double s1 = static_cast<double>(g1[m]), s2 = static_cast<double>(g2[m]);
                            double wvar = s2;
                            if (A.measure != AR_NCC) {
                                const double q = __dmul_rn(s1, s1);
                                wvar = __dsub_rn(s2, p2 ? __dmul_rn(q, inv) : __ddiv_rn(q, nn));
                            }
                            if (m <= last) s_wv[(j0 + m) * A.NRS + i] = ng[m] && wvar > 0.0 ? wvar : 0.0;
                        }
                    }
                    __syncthreads();
                }
                // From a pixel that is not finite on, its column's sums are not either.
                if constexpr (!Tr::integer) {
                    if (__syncthreads_or(!(h2 <= DBL_MAX)))
                        fp_nonfinite(s_win, XH, A.WS, ch, cw, nr, nc, cshift, A.measure != AR_NCC, A.GTI, A.GTJ,
                                     s_v1, s_wv, A.NRS);
                }
                have_var = Tr::integer;  // Float32 image values carry the shift's rounding
            }

            TC_PHASE(3)
            // Numerator: kMI rows of two columns per thread over its part of the chip columns.
            double acc64[2 * kMI];
#pragma unroll
            for (int v = 0; v < 2 * kMI; ++v) acc64[v] = 0.0;
            if (active) {
                const int ncg = cw >> 1;  // groups of two chip columns
                const int ge = ncg * (part + 1) / split;
                for (int gc = ncg * part / split; gc < ge; ++gc) {
                    float2 acc[kMI];
#pragma unroll
                    for (int m = 0; m < kMI; ++m) acc[m] = make_float2(0.0f, 0.0f);
#pragma unroll 1
                    for (int bb = 0; bb < 2; ++bb) {
                        const float2* wc = s_win + (bb * XH + p + gc) * A.WS + il;
                        const float4* cc = reinterpret_cast<const float4*>(s_chip + (2 * gc + bb) * A.CHP);
                        float2 w[kMI + 8];
#pragma unroll
                        for (int m = 0; m < kMI; ++m) w[m] = wc[m];
                        wc += kMI;
                        // The chip values of the next step are loaded a step ahead (past the last one
                        // they are the next column's, or the window's, and unused).
                        float4 c0 = cc[0], c1 = cc[1];
#pragma unroll 2
                        for (int a0 = 0; a0 < chp; a0 += 8) {
#pragma unroll
                            for (int m = 0; m < 8; ++m) w[kMI + m] = wc[a0 + m];
                            const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
                            c0 = cc[(a0 >> 2) + 2];
                            c1 = cc[(a0 >> 2) + 3];
#pragma unroll
                            for (int a = 0; a < 8; ++a)
#pragma unroll
                                for (int m = 0; m < kMI; ++m)
                                    acc[m] = __ffma2_rn(make_float2(c[a], c[a]), w[m + a], acc[m]);
#pragma unroll
                            for (int m = 0; m < kMI; ++m) w[m] = w[m + 8];
                        }
                    }
#pragma unroll
                    for (int m = 0; m < kMI; ++m) {
                        acc64[2 * m] = __dadd_rn(acc64[2 * m], static_cast<double>(acc[m].x));
                        acc64[2 * m + 1] = __dadd_rn(acc64[2 * m + 1], static_cast<double>(acc[m].y));
                    }
                }
            }
            TC_PHASE(4)
            // The parts' sums: halves until two are left, which then keep half of the rows each.
            for (int h = split >> 1; h > 1; h >>= 1) {
                __syncthreads();
                if (active && part >= h && part < 2 * h)
#pragma unroll
                    for (int v = 0; v < 2 * kMI; ++v) s_ex[v * (kCorrThreads / 2) + tid - h * items] = acc64[v];
                __syncthreads();
                if (part < h)
#pragma unroll
                    for (int v = 0; v < 2 * kMI; ++v)
                        acc64[v] = __dadd_rn(acc64[v], s_ex[v * (kCorrThreads / 2) + tid]);
            }
            if (split > 1) {
                __syncthreads();
                if (part < 2)
#pragma unroll
                    for (int v = 0; v < 2 * kMI; ++v)
                        if ((v < kMI) != (part == 0)) s_ex[v * (kCorrThreads / 2) + it] = acc64[v];
                __syncthreads();
                if (part < 2)
#pragma unroll
                    for (int v = 0; v < 2 * kMI; ++v)
                        if ((v < kMI) == (part == 0)) acc64[v] = __dadd_rn(acc64[v], s_ex[v * (kCorrThreads / 2) + it]);
            }
            TC_PHASE(5)
            // Value v of this thread is surface row il + v / 2, column 2 p + v % 2.
            auto mine = [&](int v) {
                return (split == 1 ? part == 0 : part < 2 && (v < kMI) == (part == 0)) && il + (v >> 1) < nr;
            };
            const double add = __dmul_rn(cshift, sumd);
#pragma unroll
            for (int v = 0; v < 2 * kMI; ++v) acc64[v] = __dadd_rn(acc64[v], add);

            // Float32 estimates num rsqrt(wvar), within 8 x 2^-24 of cnorm times the value they stand
            // for; 0 where there is no variance (the value is 0). `odd`: a magnitude that Float32
            // cannot be trusted with, or a NaN: then every value is evaluated exactly. The largest
            // and second largest of each thread, then of each warp.
            auto estimate = [&](int v, bool& bad) {
                const double wvar = s_wv[(2 * p + (v & 1)) * A.NRS + il + (v >> 1)];
                const float n = __double2float_rn(acc64[v]), w = __double2float_rn(wvar);
                if (!(wvar > 0.0)) return 0.0f;
                bad |= !(w > 1e-30f && w < 1e30f && fabsf(n) < 1e30f);
                return __fmul_rn(n, rsqrtf(w));
            };
            bool odd = false;
            float own = -INFINITY, own2 = -INFINITY;
            int at = 0;
#pragma unroll
            for (int v = 0; v < 2 * kMI; ++v)
                if (mine(v)) {
                    const float e = estimate(v, odd);
                    own2 = fmaxf(own2, fminf(own, e));
                    at = e > own ? v : at;
                    own = fmaxf(own, e);
                }
            {
                const float top = warp_max(own);
                const unsigned who = __ballot_sync(kFull, own == top && own > -INFINITY);
                const int first = who ? __ffs(who) - 1 : 0;
                const float sec_ = warp_max(odd ? INFINITY : lane == first ? own2 : own);
                if (lane == first) {
                    s_top[warp] = top;
                    s_sec[warp] = sec_;
                    s_at[warp] = ((il + (at >> 1)) << 16) | (2 * p + (at & 1));
                }
            }
            __syncthreads();  // also: s_ex is read
            TC_PHASE(6)
            const float wt = lane < nwarps ? s_top[lane] : -INFINITY;
            const float M = warp_max(wt);
            const float cut = M - 1.9073486e-06f * fabsf(M);  // 32 x 2^-24
            const int mw = __ffs(__ballot_sync(kFull, wt == M)) - 1;
            const bool unique =
                fabsf(M) > 1e-30f && fabsf(M) < 1e37f &&
                !__any_sync(kFull, lane < nwarps && (!(s_sec[lane & 7] < cut) || (lane != mw && !(wt < cut))));
            int pi = 0, pj = 0;
            bool any_peak = true;
            if (unique && !A.surf_out) {
                // Every other value is below this one: it is the strict (so the first) maximum.
                pi = s_at[mw] >> 16;
                pj = s_at[mw] & 0xFFFF;
            } else {
                const bool all = __syncthreads_or(odd) || !(fabsf(M) > 1e-30f && fabsf(M) < 1e37f);
                unsigned long long key = 0ull;
#pragma unroll
                for (int v = 0; v < 2 * kMI; ++v)
                    if (mine(v) && (all || A.surf_out || !(estimate(v, odd) < cut))) {
                        const int i = il + (v >> 1), j = 2 * p + (v & 1);
                        const float x = fp_exact(acc64[v], s_wv[j * A.NRS + i], cnorm);
                        const unsigned long long kk = argmax_key(x, static_cast<unsigned>(i * nc + j));
                        key = kk > key ? kk : key;
                        if (A.surf_out) A.surf_out[k * static_cast<int64_t>(A.NRS) * A.NCM + i + j * nr] = x;
                    }
                key = block_max_u64(key, reinterpret_cast<unsigned long long*>(s_red));
                unsigned rm = 0;
                float pv = 0.0f;
                any_peak = key != 0ull;
                if (key_decode(key, &rm, &pv)) {
                    pi = static_cast<int>(rm / nc);
                    pj = static_cast<int>(rm % nc);
                }
            }
            TC_PHASE(7)
            if (A.flops && tid == 0)
                atomicAdd(A.flops, 2ull * static_cast<unsigned long long>(ch) * cw * nr * nc);

            // The peak's value or the 5x5 patch's (src/peak.jl:473-482), exactly, a thread each; with
            // the rotation search kept if the angle's maximum (src/track.jl:327-328) is the largest.
            const int qi = single ? pi : min(max(pi - 2, 0), max(nr - 5, 0));
            const int qj = single ? pj : min(max(pj - 2, 0), max(nc - 5, 0));
            const unsigned span = single ? 1u : 5u;
            if (qi < il + kMI && qi + static_cast<int>(span) > il && qj <= 2 * p + 1 &&
                qj + static_cast<int>(span) > 2 * p) {
#pragma unroll
                for (int v = 0; v < 2 * kMI; ++v) {
                    const int i = il + (v >> 1), j = 2 * p + (v & 1);
                    const unsigned a = static_cast<unsigned>(i - qi), c = static_cast<unsigned>(j - qj);
                    if (a < span && c < span && mine(v)) {
                        s_pn[c * 5 + a] = acc64[v];
                        s_pw[c * 5 + a] = s_wv[j * A.NRS + i];
                    }
                }
            }
            __syncthreads();
            const int npatch = single ? 1 : 25;
            if constexpr (!ROT) {
                found = true;
                pi0 = qi;
                pj0 = qj;
                if (tid < npatch) s_best[tid] = fp_exact(s_pn[tid], s_pw[tid], cnorm);
            } else {
                if (tid < npatch) s_pp[tid] = fp_exact(s_pn[tid], s_pw[tid], cnorm);
                __syncthreads();
                const float pk = any_peak ? s_pp[(pj - qj) * 5 + (pi - qi)] : NAN;
                if (pk > bestpk) {
                    bestpk = pk;
                    found = true;
                    pi0 = qi;
                    pj0 = qj;
                    if (tid < npatch) s_best[tid] = s_pp[tid];
                }
            }
            TC_PHASE(8)
        }
        if (skip || !found) continue;  // every angle degenerate: searched, no measurement
        // Warp 0 has the values (it computed them).
        if (warp == 0) {
            if (single) {
                // peak_offset (src/peak.jl:102-106) and the output write (src/track.jl:293-295).
                if (lane == 0) {
                    A.out.dx[k] = __double2float_rn(__dadd_rn(static_cast<double>(pj0 - static_cast<int>(prx)), dx0));
                    A.out.dy[k] = __double2float_rn(__dadd_rn(static_cast<double>(pi0 - static_cast<int>(pry)), dy0));
                    A.out.corr[k] = s_best[0];
                }
            } else {
                int slot = 0;
                if (lane == 0) slot = atomicAdd(A.sub_count, 1);
                slot = __shfl_sync(kFull, slot, 0);
                if (lane < 25) A.sub_patch[static_cast<int64_t>(slot) * 25 + lane] = s_best[lane];
                if (lane == 0) {
                    A.sub_point[slot] = k;
                    A.sub_origin[2 * slot] = pi0;
                    A.sub_origin[2 * slot + 1] = pj0;
                }
            }
        }
        TC_PHASE(9)
        TC_PHASE_POINT
    }
    TC_PHASE_FLUSH
}

// ----------------------------------------------------------------------------------------------
// Tensor-core correlation for UInt8 imagery (tcgen05.mma kind::i8, exact 32-bit accumulation).
//
// The numerator S[i, j] = sum_{a,b} C[a, b] W[i + a, j + b] (C the chip, W the window, i the
// surface row, j the surface column) is a sum of products D[j, i] += sum_k A[j, k] B[i, k] over
// K = (16-row block q of the window, chip column b, row r within the block):
//   A[j, (q, b, r)] = W'[16 q + r, j + b]     the window as 16-byte blocks s_W[q][x][r]; row j
//                                             of A starts 16 bytes after row j - 1, so A is
//                                             read in place;
//   B[i, (q, b, r)] = E_b[i - 16 q][r]        with E_b[u][r] = C[r - u - delta, b], the chip as
//                                             16-byte rows per column b, built once per point.
// W' starts at the 16-aligned image row `delta` rows above the window's first row, so each
// 16-byte block of a column-major image with 16-aligned columns is one aligned load. The chip
// rows a block q can meet are surface rows i in [16 q + 16 - NB, 16 q + 16), i.e. the same
// NB = 16 * ceil((ch + 30) / 16) rows u = i - 16 q of E for every q: each block's product
// (M = 64 surface columns, N = NB, K = 32: two chip columns) adds into accumulator columns
// [16 q, 16 q + NB), surface row i living in column i + NB - 16 of a cleared accumulator. The
// products are exact (u8 x u8 summed below 2^31), so the numerator equals the CUDA-core
// kernel's and every surface value, the peak and the patch are bit-identical to it.
//
// Normalising all 2ry x 2rx values in FP64 would cost as much as the products, and only the
// peak and its 5 x 5 patch are read. So each value is first estimated in FP32 with a
// rigorous bound on its distance from the FP32 surface value (a bound a value for surfaces up to
// 64 x 64, one for all of them beyond); only values whose bound reaches
// the largest estimate, and the patch, get the reference's exact FP64 normalisation.
//
// What bounds the larger surfaces: the products' operand reads (6 KB of shared memory a
// 128 x 64 x 32 product, 884 KB a point at chip 32, surface 88 x 88, some 7 k cycles), then the
// latency of every other step at eight warps. So the numerators stay in Tensor Memory, nothing
// but the box sums is kept for each value, and two CTAs share an SM up to 94 x 94 at chip 32 and
// 96 x 96 at chip 16: 14 400 points of chip 32, radius 44 took 1.67 ms and take 1.19 ms, 12 000 of chip 16,
// radius 48 0.93 ms (1.42). One CTA of 512 threads, or four issuing threads, gave nothing.

constexpr int kTcThreads = 256;
constexpr int kTc2Threads = 320;  // k_corr_tc2: eight main warps, a fetch warp, a patch warp
constexpr int kPadL = 32;            // zero bytes before each staged chip column
constexpr uint32_t kTcWaitPolls = 1u << 22;

struct TcArgs {
    const uint8_t* ref;
    const uint8_t* sec;
    const uint8_t* valid;
    int64_t nrows, ncols;
    DevPoints pts;
    int64_t padx, pady;
    int up, measure;
    int NB, QM, QS, PS, PC, XS, NRS, NRM, NCM, CHM, CWM;
    int BC;                          // chip columns per chunk of the chip operand (even)
    int MT;                          // MMA M: 64 or 128 surface columns
    int big;                         // 1: box sums before the products, chunks reuse their space
    int VR;                          // k_corr_tc: surface rows per box-sum stripe
    int roots;                       // k_corr_tc: reciprocal roots kept beside the box sums
    unsigned off_E, off_W, off_P, off_V, off_S1, off_S2, off_R, off_num, off_est, off_red;
    unsigned off_L, off_rawW, off_rawC;  // k_corr_tc2
    int XV;                          // row stride (words) of the column sums V1, V2
    int acc1_col;                    // stride between the accumulators (first column of the
                                     // second one)
    int issuers;                     // k_corr_tc: threads issuing the products, 2 or 4
    uint32_t tmem_cols;
    DevOutputs out;
    int* sub_count;
    int64_t* sub_point;
    int32_t* sub_origin;
    float* sub_patch;
    float* surf_out;
    unsigned long long* flops;
    int* status;                     // set to 1 when a tensor-core wait ran out
};

// The reference's normalisation of one value from its exact integer numerator and box sums
// (the raw-numerator branch of k_corr).
__device__ __forceinline__ float tc_exact(uint32_t D, uint32_t S1, uint32_t S2, double mean,
                                          double nn, double cnorm, int measure) {
    const double s1 = static_cast<double>(S1), s2 = static_cast<double>(S2);
    const double num = __dsub_rn(static_cast<double>(D), __dmul_rn(mean, s1));
    double den;
    if (measure == AR_NCC) {
        den = __dmul_rn(cnorm, __dsqrt_rn(s2 > 0.0 ? s2 : 0.0));
    } else {
        double wvar = __dsub_rn(s2, __ddiv_rn(__dmul_rn(s1, s1), nn));
        if (!(wvar > 0.0)) wvar = 0.0;
        den = __dmul_rn(cnorm, __dsqrt_rn(wvar));
    }
    return den > 0.0 ? __double2float_rn(__ddiv_rn(num, den)) : 0.0f;
}

// FP32 estimate of one surface value and a bound on its distance from the value tc_exact
// returns. With nn, C = sum(chip), s1, s2, D exact integers, the value is
//   ZNCC: (nn D - C s1) / (cnorm sqrt(nn) sqrt(nn s2 - s1^2)),  NCC: (nn D - C s1) / (cnorm nn sqrt(s2)).
// D and s2 are converted with one rounding each (s1 < 2^24 and C are exact). The numerator and
// the variance are then formed with three roundings of relative size u = 2^-24 on terms no
// larger than `tn` and `tv`, so their absolute errors are below 3u tn and 3u tv; rsqrt (2 ulp),
// the scale `k` and two products add < 6u relative, and the final Float32 rounding of the
// reference 1u. 1/vx is taken as r^2 (within 9u of it). The bound returned covers all of it
// with more than 3x slack; NaN marks a value whose variance is too small for the bound
// (evaluated exactly). `k7` is 7u k.
__device__ __forceinline__ float tc_estimate(uint32_t D, uint32_t S1, uint32_t S2, float nnf,
                                             float csum, float k, float k7, int measure,
                                             float* bound) {
    const float d = __uint2float_rn(D), s1 = __uint2float_rn(S1), s2 = __uint2float_rn(S2);
    const float p = __fmul_rn(csum, s1);
    const float nx = __fmaf_rn(nnf, d, -p);
    const float tn = __fmaf_rn(nnf, d, p);  // |nn D| + |C s1| (both non-negative)
    float vx, tv;
    if (measure == AR_NCC) {
        vx = s2;
        tv = s2;
    } else {
        const float q = __fmul_rn(s1, s1);
        vx = __fmaf_rn(nnf, s2, -q);
        tv = __fmaf_rn(nnf, s2, q);
    }
    const float ev = 3.5762786865234375e-07f * tv;  // 6u tv
    if (!(vx > 64.0f * ev)) {
        *bound = 0.0f;
        return __int_as_float(0x7fc00000);
    }
    const float r = rsqrtf(vx);
    const float est = __fmul_rn(__fmul_rn(nx, r), k);
    // |err| <= |est| (8u + ev / vx) + 3.5u tn r k  (u = 2^-24), doubled for slack.
    const float rel = __fmaf_rn(ev, __fmul_rn(r, r), 9.5367431640625e-07f);  // 16u + ev/vx
    *bound = __fmaf_rn(fabsf(est), 2.0f * rel, __fmul_rn(__fmul_rn(tn, r), k7)) + 1e-30f;
    return est;
}

__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// Rows of the chip operand that block q's product needs: operand row e holds offset
// u = e - NB + 16 (surface row i = 16 q + u), and only surface rows 0 <= i < nr are read, so
// e runs over [max(0, NB - 16 - 16 q), min(NB, NB - 16 + nr - 16 q)). Returned as a 16-aligned
// start `elo` and a multiple of 16 `n` (elo + n <= NB); false when the block reaches no
// surface row.
__device__ __forceinline__ bool block_rows(int q, int NB, int nr, int* elo, int* n) {
    const int lo = max(0, NB - 16 - 16 * q);
    const int hi = min(NB, NB - 16 + nr - 16 * q);
    if (hi <= lo) return false;
    *elo = lo & ~15;
    *n = (hi - *elo + 15) & ~15;
    return true;
}

// Sixteen bytes of column `c` from row r0 (zero outside the image), in two steps so that a
// thread can have several in flight: col16_issue starts the loads -- two aligned 16-byte loads
// when they stay inside the image, else byte by byte -- and col16_finish shifts the bytes into
// place.
struct Col16 {
    uint4 lo, hi;
    uint32_t s;  // byte offset of row r0 in `lo` (0: `lo` is the result)
};

__device__ __forceinline__ Col16 col16_issue(const uint8_t* img, const uint8_t* img_end,
                                             int64_t nrows, int64_t ncols, int64_t c, int64_t r0) {
    Col16 L;
    L.s = 0;
    L.lo = L.hi = make_uint4(0, 0, 0, 0);
    if (c < 0 || c >= ncols) return L;
    const uint8_t* p = img + c * nrows + r0;
    if (r0 >= 0 && r0 + 16 <= nrows) {
        const uintptr_t pa = reinterpret_cast<uintptr_t>(p);
        const uint32_t s = static_cast<uint32_t>(pa & 15);
        const uint4* a = reinterpret_cast<const uint4*>(pa - s);
        if (s == 0) {
            L.lo = __ldg(a);
            return L;
        }
        if (reinterpret_cast<const uint8_t*>(a) + 32 <= img_end) {
            L.lo = __ldg(a);
            L.hi = __ldg(a + 1);
            L.s = s;
            return L;
        }
    }
    uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        const int64_t r = r0 + t;
        const uint32_t bb = (r >= 0 && r < nrows) ? p[t] : 0u;
        w[t >> 2] |= bb << (8 * (t & 3));
    }
    L.lo = make_uint4(w[0], w[1], w[2], w[3]);
    return L;
}

__device__ __forceinline__ uint4 col16_finish(const Col16& L) {
    const uint32_t s = L.s;
    if (s == 0) return L.lo;
    const uint32_t w[8] = {L.lo.x, L.lo.y, L.lo.z, L.lo.w, L.hi.x, L.hi.y, L.hi.z, L.hi.w};
    uint32_t u[6], v[5];
#pragma unroll
    for (int k = 0; k < 6; ++k) u[k] = (s & 8) ? w[k + 2] : w[k];
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = (s & 4) ? u[k + 1] : u[k];
    const uint32_t sh = (s & 3) * 8u;
    return make_uint4(__funnelshift_r(v[0], v[1], sh), __funnelshift_r(v[1], v[2], sh),
                      __funnelshift_r(v[2], v[3], sh), __funnelshift_r(v[3], v[4], sh));
}

// prepare_chip! statistics (src/correlate.jl:423-453) of a UInt8 chip staged as zero-padded
// byte columns (row a of column b at s_P[b * PC + kPadL + a]; rows outside the image are 0, as
// `pixel` reads them), with the CUDA-core kernel's FP64 results bit for bit: thread t takes
// elements t, t + bd, ... of the column-major chip (rows padded to a multiple of kUA) and the
// per-thread partial sums go through the same block sum.
//   One pass gives each thread the count m, sum P and sum of squares Q of its elements (exact
// integers; the sum of C is exact in any order). When the area nn is a power of two the mean
// S/nn is exact, so is every deviation d = N/nn (N = nn C - S) and its square, and a thread's
// FP64 running sum of squares is exactly K/nn^2 with K = sum N^2 = nn^2 Q - 2 nn S P + m S^2
// while K stays below 2^53 -- guaranteed when (its terms) x (255 nn)^2 is: then the partial is
// that integer scaled by 1/nn^2, the double the FP64 loop produces. Other areas take the FP64
// loop over the staged chip.
template <bool MAIN = false>
__device__ __forceinline__ void staged_chip_stats(const uint8_t* s_P, int PC, int ch, int cw, int tid,
                                                  int bd, double* s_red, double* csum, double* mean,
                                                  double* sq) {
    const int chp = (ch + kUA - 1) & ~(kUA - 1);
    const int ne = chp * cw;
    const int db = bd / chp, da = bd - db * chp;
    const int b0 = tid / chp, a0 = tid - b0 * chp;
    auto step = [&](int& a, int& b) {
        a += da;
        b += db;
        if (a >= chp) {
            a -= chp;
            ++b;
        }
    };
    uint32_t P = 0u, Q = 0u, m = 0u;
    {
        int a = a0, b = b0;
        for (int e = tid; e < ne; e += 4 * bd) {
            int o[4];
            bool in[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                in[u] = e + u * bd < ne && a < ch;
                o[u] = b * PC + kPadL + a;
                step(a, b);
            }
            uint32_t v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = in[u] ? s_P[o[u]] : 0u;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                P += v[u];
                Q += v[u] * v[u];
                m += in[u] ? 1u : 0u;
            }
        }
    }
    double st[1] = {static_cast<double>(P)};
    block_sum_f64<1, MAIN>(st, s_red);
    *csum = st[0];
    const int nn = ch * cw;
    const double mn = __ddiv_rn(st[0], static_cast<double>(nn));
    *mean = mn;
    const int terms = (ne + bd - 1) / bd;
    const double span = 255.0 * static_cast<double>(nn);
    const bool exact = (nn & (nn - 1)) == 0 && static_cast<double>(terms) * span * span < 9007199254740992.0;
    double acc2[1] = {0.0};
    if (exact) {
        const long long S = static_cast<long long>(st[0]), N2 = static_cast<long long>(nn);
        const long long K = N2 * N2 * static_cast<long long>(Q) - 2 * N2 * S * static_cast<long long>(P) +
                            static_cast<long long>(m) * S * S;
        const double inv = 1.0 / (static_cast<double>(nn) * static_cast<double>(nn));  // 2^-2k
        acc2[0] = static_cast<double>(K) * inv;
    } else {
        int a = a0, b = b0;
        for (int e = tid; e < ne; e += bd) {
            if (a < ch) {
                const double d = __dsub_rn(static_cast<double>(s_P[b * PC + kPadL + a]), mn);
                acc2[0] = __dadd_rn(acc2[0], __dmul_rn(d, d));
            }
            step(a, b);
        }
    }
    block_sum_f64<1, MAIN>(acc2, s_red);
    *sq = acc2[0];
}

// REG: every surface of the pass has at most 64 rows and 64 columns (M = 64), so one 16x256b
// read per warp covers it and each thread keeps its 16 numerators and upper bounds in
// registers through both passes. Otherwise each pass reads the numerators from Tensor Memory.
template <bool REG>
__global__ void __launch_bounds__(kTcThreads, 2) k_corr_tc(const TcArgs A) {
    extern __shared__ __align__(1024) unsigned char smem_tc[];
    __shared__ uint64_t s_mbar;
    __shared__ uint32_t s_taddr;
    __shared__ int s_slot;
    __shared__ int s_ncand;
    __shared__ uint32_t s_pd[25];
    __shared__ float s_fmax[kTcThreads / 32], s_sec[kTcThreads / 32];
    __shared__ int s_at[kTcThreads / 32];
    __shared__ unsigned long long s_isum[2][2];
    uint8_t* s_E = smem_tc + A.off_E;
    uint8_t* s_W = smem_tc + A.off_W;
    uint8_t* s_P = smem_tc + A.off_P;
    uint32_t* s_V1 = reinterpret_cast<uint32_t*>(smem_tc + A.off_V);
    uint2* s_S = reinterpret_cast<uint2*>(smem_tc + A.off_S1);  // box sums of W, of W^2
    float* s_R = reinterpret_cast<float*>(smem_tc + A.off_R);
    uint32_t* s_num = reinterpret_cast<uint32_t*>(smem_tc + A.off_num);
    float* s_est = reinterpret_cast<float*>(smem_tc + A.off_est);
    double* s_red = reinterpret_cast<double*>(smem_tc + A.off_red);

    const int tid = threadIdx.x, bd = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = bd >> 5;
    // Threads issuing the products (four where REG has the SM to itself).
    const int NI = A.issuers;
    const int64_t NR = A.nrows + 2 * A.pady, NC = A.ncols + 2 * A.padx;
    const double shx = static_cast<double>(A.padx) + 0.5;
    const double shy = static_cast<double>(A.pady) + 0.5;
    const uint8_t* ref_end = A.ref + A.nrows * A.ncols;
    const uint8_t* sec_end = A.sec + A.nrows * A.ncols;
    const uint8_t* valid_end = A.valid + A.nrows * A.ncols;

    if (warp == 0) {
        tc::tmem_alloc(&s_taddr, A.tmem_cols);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        tc::mbar_init(&s_mbar, NI);  // one commit per issuing thread
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t taddr = s_taddr;
    const uint32_t acc1 = static_cast<uint32_t>(A.acc1_col);  // second accumulator's first column
    uint32_t phase = 0;
    bool failed = false;
    if (tid < 4) s_isum[tid >> 1][tid & 1] = 0ull;
    for (int e = tid; e < A.CWM * A.PC; e += bd) s_P[e] = 0;
    int iter = 0;
    int dirty_ch = 0;
    TC_PHASE_INIT

    // Each CTA takes a contiguous run of points: consecutive points of a grid column have the
    // same window columns one grid step lower, so most of their box sums carry over. s_S
    // is a ring of NRS rows per column: surface row i of the held point is stored at row
    // (i + rbase) mod NRS, and carrying the sums down by `sh` rows advances rbase.
    const int64_t per = (A.pts.n + gridDim.x - 1) / gridDim.x;
    const int64_t kbeg = static_cast<int64_t>(blockIdx.x) * per;
    const int64_t kend = min(A.pts.n, kbeg + per);
    bool held = false;  // s_S holds the sums of the geometry h_*
    int64_t h_wr = 0, h_wc = 0;
    int h_ch = 0, h_cw = 0, h_nr = 0, h_nc = 0;
    int rbase = 0;
    auto ring = [&](int i) {
        const int r = i + rbase;
        return r >= A.NRS ? r - A.NRS : r;
    };

    for (int64_t k = kbeg; k < kend; ++k, ++iter) {
        tc::fence_before_sync();
        __syncthreads();  // the previous point's buffers and accumulator are no longer read
        tc::fence_after_sync();
        TC_PHASE(0)
        // The chip sums of this iteration go to s_isum[ib]; the other buffer, last read
        // before the barrier above, is cleared for the next iteration.
        const int ib = iter & 1;
        if (tid < 2) s_isum[ib ^ 1][tid] = 0ull;
        const int64_t prx = A.pts.rx[k], pry = A.pts.ry[k];
        if (!(prx > 0 && pry > 0)) continue;
        const double xs = A.pts.x[k] + shx, ys = A.pts.y[k] + shy;
        const int64_t hx = A.pts.csx[k] / 2, hy = A.pts.csy[k] / 2;
        const int64_t ccx = static_cast<int64_t>(floor(__dsub_rn(xs, A.pts.dx0[k])));
        const int64_t ccy = static_cast<int64_t>(floor(__dsub_rn(ys, A.pts.dy0[k])));
        const int64_t wcx = static_cast<int64_t>(floor(xs)), wcy = static_cast<int64_t>(floor(ys));
        const int64_t cr0 = ccy - hy, cr1 = ccy + hy - 1, cc0 = ccx - hx, cc1 = ccx + hx - 1;
        const int64_t wr0 = wcy - hy - pry, wr1 = wcy + hy + pry - 2;
        const int64_t wc0 = wcx - hx - prx, wc1 = wcx + hx + prx - 2;
        const bool chip_in = (cr1 < cr0 || cc1 < cc0) ||
                             (cr0 >= 1 && cr1 <= NR && cc0 >= 1 && cc1 <= NC);
        const bool win_in = (wr1 < wr0 || wc1 < wc0) ||
                            (wr0 >= 1 && wr1 <= NR && wc0 >= 1 && wc1 <= NC);
        if (!chip_in || !win_in) continue;
        const int ch = static_cast<int>(2 * hy), cw = static_cast<int>(2 * hx);
        const int nr = static_cast<int>(2 * pry), nc = static_cast<int>(2 * prx);
        if (ch <= 0 || cw <= 0) continue;
        if (ch > A.CHM || cw > A.CWM || nr > A.NRM || nc > A.NCM || nc > A.MT) continue;
        TC_PHASE(1)
        const int64_t chip_r = cr0 - 1 - A.pady, chip_c = cc0 - 1 - A.padx;
        const int64_t win_r = wr0 - 1 - A.pady, win_c = wc0 - 1 - A.padx;
        const long long nnl = static_cast<long long>(ch) * cw;
        // Power-of-two areas up to 4096: every term of the reference's FP64 chip sums is exact.
        const bool pow2 = (nnl & (nnl - 1)) == 0 && nnl <= 4096;

        // The chip as zero-padded byte columns, _any_valid over it (src/track.jl:416-421) and,
        // for power-of-two areas, its exact integer sums: warps over chip columns, lanes over
        // rows, all loads of a lane issued before their uses. Rows a taller chip left behind
        // are cleared (the padding itself is never written).
        // Invariant: chip rows at or beyond `dirty_ch` are zero in every column.
        if (ch < dirty_ch)
            for (int b = warp; b < A.CWM; b += nwarps)
                for (int a = ch + lane; a < dirty_ch; a += 32) s_P[b * A.PC + kPadL + a] = 0;
        dirty_ch = ch;
        // A task is 16 rows of one chip column: a 16-byte block of the image and of its mask
        // (col16_issue: aligned loads and a byte shift, zero outside the image), rows beyond ch
        // zeroed. Each thread starts the loads of two tasks before using them.
        int any = 0;
        unsigned long long isum = 0ull, isq = 0ull;
        {
            const int nb16 = (ch + 15) >> 4, ntask = nb16 * cw;
            uint32_t s1 = 0u, s2 = 0u;
            for (int t0 = tid; t0 < ntask; t0 += 2 * bd) {
                Col16 Lv[2], Lm[2];
                int tb[2], tj[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int t = t0 + u * bd;
                    tb[u] = t / nb16;
                    tj[u] = t - tb[u] * nb16;
                    const int64_t c = t < ntask ? chip_c + tb[u] : -1;
                    Lv[u] = col16_issue(A.sec, sec_end, A.nrows, A.ncols, c, chip_r + 16 * tj[u]);
                    Lm[u] = col16_issue(A.valid, valid_end, A.nrows, A.ncols, c, chip_r + 16 * tj[u]);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (t0 + u * bd >= ntask) continue;
                    const uint4 v = col16_finish(Lv[u]), mk = col16_finish(Lm[u]);
                    const int keep = ch - 16 * tj[u];
                    uint32_t w[4] = {v.x, v.y, v.z, v.w}, mw[4] = {mk.x, mk.y, mk.z, mk.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int kb = keep - 4 * i;
                        const uint32_t m = kb >= 4 ? 0xffffffffu : kb <= 0 ? 0u : (1u << (8 * kb)) - 1u;
                        w[i] &= m;
                        any |= (mw[i] & m) != 0u;
                        s1 = __dp4a(w[i], 0x01010101u, s1);
                        s2 = __dp4a(w[i], w[i], s2);
                    }
                    *reinterpret_cast<uint4*>(s_P + tb[u] * A.PC + kPadL + 16 * tj[u]) =
                        make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            isum = s1;
            isq = s2;
        }
        if (pow2) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                isum += __shfl_xor_sync(kFull, isum, o);
                isq += __shfl_xor_sync(kFull, isq, o);
            }
            if (lane == 0) {
                atomicAdd(&s_isum[ib][0], isum);
                atomicAdd(&s_isum[ib][1], isq);
            }
        }
        if (!__syncthreads_or(any)) continue;
        TC_PHASE(2)
        if (tid == 0) A.out.searched[k] = 1;

        // prepare_chip! statistics. Power-of-two areas: every term of the reference's FP64
        // sums is exact, so mean = sum/nn and sq = (nn sum(C^2) - sum(C)^2)/nn exactly;
        // otherwise the CUDA-core kernel's FP64 loops, in its order (bit-identical sums).
        double mean, sq, csum_d;
        if (pow2) {
            const long long cs = static_cast<long long>(s_isum[ib][0]);
            const long long c2 = static_cast<long long>(s_isum[ib][1]);
            csum_d = static_cast<double>(cs);
            mean = __ddiv_rn(csum_d, static_cast<double>(nnl));
            sq = __ddiv_rn(static_cast<double>(nnl * c2 - cs * cs), static_cast<double>(nnl));
        } else {
            staged_chip_stats(s_P, A.PC, ch, cw, tid, bd, s_red, &csum_d, &mean, &sq);
        }
        if (!(sq > __dmul_rn(__dmul_rn(DBL_EPSILON, static_cast<double>(ch)), static_cast<double>(cw))))
            continue;  // degenerate chip: searched, no measurement (src/track.jl:286)
        TC_PHASE(3)
        const double cnorm = __dsqrt_rn(sq);
        const double nn = static_cast<double>(nnl);

        // Box sums carried from the held point: same window columns and shape, `sh` rows
        // higher; only surface rows iA .. nr - 1 are computed (iA = 0: all of them).
        const int64_t sh64 = win_r - h_wr;
        const bool carry = held && win_c == h_wc && ch == h_ch && cw == h_cw && nr == h_nr &&
                           nc == h_nc && sh64 > 0 && sh64 < nr;
        int iA = 0;
        if (carry) {
            iA = nr - static_cast<int>(sh64);
            rbase += static_cast<int>(sh64);
            if (rbase >= A.NRS) rbase -= A.NRS;
        } else {
            rbase = 0;
        }
        held = true;
        h_wr = win_r;
        h_wc = win_c;
        h_ch = ch;
        h_cw = cw;
        h_nr = nr;
        h_nc = nc;
#ifdef AR_TC_PHASES
        if (tid == 0 && carry) atomicAdd(&g_tc_phase[14], 1ull);
#endif

        // Window blocks W'[16 q + r][x] (x < XS) from 16 image rows at base_r + 16 q.
        const int64_t delta = ((win_r % 16) + 16) % 16;
        const int64_t base_r = win_r - delta;
        const int Q = static_cast<int>((delta + ch + nr - 1 + 15) / 16);
        const int XW = cw + nc - 1;
        // A block is one aligned 16-byte load when the image's columns are 16-byte aligned (row
        // counts divisible by 16), otherwise two aligned loads and a byte shift.
        // A task is block q of column x (consecutive threads on consecutive columns); each thread
        // starts the loads of three tasks before using them.
        {
            const int ntask = Q * A.XS;
            for (int t0 = tid; t0 < ntask; t0 += 3 * bd) {
                Col16 L[3];
                int tq[3], tx[3];
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    const int t = t0 + u * bd;
                    tq[u] = t / A.XS;
                    tx[u] = t - tq[u] * A.XS;
                    const int64_t c = t < ntask ? win_c + tx[u] : -1;
                    L[u] = col16_issue(A.ref, ref_end, A.nrows, A.ncols, c, base_r + 16 * tq[u]);
                }
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    if (t0 + u * bd >= ntask) continue;
                    const int q = tq[u], x = tx[u];
                    const uint4 v = col16_finish(L[u]);
                    *reinterpret_cast<uint4*>(s_W + q * A.QS + x * 16) = v;
                }
            }
        }
        __syncthreads();  // s_P, s_W complete
        TC_PHASE(4)

        // The reciprocal roots of two values' variance terms (pass 1).
        const float nnf = static_cast<float>(nnl);
        auto recip2 = [&](uint2 a, uint2 b) {
            const float2 s1 = make_float2(__uint2float_rn(a.x), __uint2float_rn(b.x));
            const float2 s2 = make_float2(__uint2float_rn(a.y), __uint2float_rn(b.y));
            float2 vx = s2;
            if (A.measure != AR_NCC) {
                const float2 q = __fmul2_rn(s1, s1), n2 = make_float2(nnf, nnf);
                vx = __ffma2_rn(n2, s2, neg2(q));
                const float2 tv = __ffma2_rn(n2, s2, q);
                vx.x = tv.x > 2048.0f * vx.x ? -1.0f : vx.x;  // its root is NaN
                vx.y = tv.y > 2048.0f * vx.y ? -1.0f : vx.y;
            }
            return make_float2(a.y == 0u ? 0.0f : rsqrtf(vx.x), b.y == 0u ? 0.0f : rsqrtf(vx.y));
        };
        const bool roots = !REG && A.roots;  // s_R holds them, carried like the box sums

        // Box sums of W and W^2 (integral_both!, boxsum, src/integral.jl:141-170, 244-247) as
        // exact integers, in stripes of A.VR surface rows, by the threads below kBT (named barrier
        // 1). They run while the tensor core works on the chip operand, or, when that comes in
        // chunks that share the stripe's space, before it. Only surface rows iA .. nr - 1 are
        // computed (the others carried over), into ring rows. Column sums of a stripe straight
        // from the 16-byte window blocks (no transposed
        // copy): a thread per column, dp4a over the chip's rows for the stripe's first row, then a
        // slide of four rows at a time. Row sums of a stripe as prefix sums, a warp per row: a
        // difference of two prefixes is exact modulo 2^32 and the sums are below 2^32.
        auto box_sums = [&](const int kBT) {
            auto bar_box = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(kBT) : "memory"); };
            uint32_t* s_V2 = s_V1 + A.VR * A.XV;
            for (int is = iA; is < nr; is += A.VR) {
                const int ie = min(is + A.VR, nr);
                for (int x = tid; x < XW; x += kBT) {
                    const uint8_t* col = s_W + x * 16;
                    const int R0 = static_cast<int>(delta) + is, R1 = R0 + ch;
                    uint32_t h1 = 0u, h2 = 0u;
                    for (int q = R0 >> 4; 16 * q < R1; ++q) {
                        const uint4 v = *reinterpret_cast<const uint4*>(col + q * A.QS);
                        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                        const int lo = R0 - 16 * q, hi = R1 - 16 * q;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int l = lo - 4 * u, h = hi - 4 * u;
                            uint32_t m = l <= 0 ? 0xffffffffu : l >= 4 ? 0u : 0xffffffffu << (8 * l);
                            m &= h >= 4 ? 0xffffffffu : h <= 0 ? 0u : (1u << (8 * h)) - 1u;
                            const uint32_t wm = w[u] & m;
                            h1 = __dp4a(wm, 0x01010101u, h1);
                            h2 = __dp4a(wm, wm, h2);
                        }
                    }
                    // The word of rows a .. a + 3 (a a multiple of 4, held to the staged blocks).
                    auto word = [&](int a) {
                        const int q = min(a >> 4, Q - 1);
                        return *reinterpret_cast<const uint32_t*>(col + q * A.QS + (a & 12));
                    };
                    const uint32_t so = static_cast<uint32_t>(R0 & 3) * 8u;
                    const uint32_t sn = static_cast<uint32_t>(R1 & 3) * 8u;
                    int ao = R0 & ~3, an = R1 & ~3;
                    uint32_t lo_o = word(ao), lo_n = word(an);
                    uint32_t* v1 = s_V1 + x;
                    uint32_t* v2 = s_V2 + x;
                    for (int i = is; i < ie; i += 4) {
                        ao += 4;
                        an += 4;
                        const uint32_t hi_o = word(ao), hi_n = word(an);
                        const uint32_t wo = __funnelshift_r(lo_o, hi_o, so);
                        const uint32_t wn = __funnelshift_r(lo_n, hi_n, sn);
                        lo_o = hi_o;
                        lo_n = hi_n;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (i + u < ie) {
                                *v1 = h1;
                                *v2 = h2;
                            }
                            v1 += A.XV;
                            v2 += A.XV;
                            const uint32_t bo = (wo >> (8 * u)) & 255u, bn = (wn >> (8 * u)) & 255u;
                            h1 += bn - bo;
                            h2 += bn * bn - bo * bo;
                        }
                    }
                }
                bar_box();
                // Two rows at a time, as a row's loads, scans and stores are one chain (one with REG, whose
                // registers are all in use: 342 -> 348 us over 1024 points at chip 128, radius 25). 16 points at
                // chip 32, radius 44, refined: 78.3 -> 76.3 us a call; 14 400: 1993 -> 1978.
                constexpr int kRows = REG ? 1 : 2;
                const int bw = kBT >> 5;
                for (int i = is + warp; i < ie; i += kRows * bw) {
                    uint32_t* v1 = s_V1 + (i - is) * A.XV;
                    uint32_t* v2 = s_V2 + (i - is) * A.XV;
                    const int rows = i + bw < ie ? kRows : 1;
                    uint32_t c1[kRows] = {}, c2[kRows] = {};
                    for (int x0 = 0; x0 < XW; x0 += 128) {
                        const int x = x0 + 4 * lane;
                        uint4 a[kRows], b[kRows];
                        uint32_t t1[kRows], t2[kRows];
#pragma unroll
                        for (int r = 0; r < kRows; ++r) {
                            a[r] = b[r] = make_uint4(0, 0, 0, 0);
                            if (x < XW && r < rows) {
                                a[r] = *reinterpret_cast<const uint4*>(v1 + r * bw * A.XV + x);
                                b[r] = *reinterpret_cast<const uint4*>(v2 + r * bw * A.XV + x);
                            }
                        }
#pragma unroll
                        for (int r = 0; r < kRows; ++r) {
                            a[r].y += a[r].x;
                            a[r].z += a[r].y;
                            a[r].w += a[r].z;
                            b[r].y += b[r].x;
                            b[r].z += b[r].y;
                            b[r].w += b[r].z;
                            t1[r] = warp_inclusive_scan(a[r].w);
                            t2[r] = warp_inclusive_scan(b[r].w);
                        }
#pragma unroll
                        for (int r = 0; r < kRows; ++r) {
                            const uint32_t p1 = t1[r] - a[r].w + c1[r], p2 = t2[r] - b[r].w + c2[r];
                            if (x < XW && r < rows) {
                                *reinterpret_cast<uint4*>(v1 + r * bw * A.XV + x) =
                                    make_uint4(a[r].x + p1, a[r].y + p1, a[r].z + p1, a[r].w + p1);
                                *reinterpret_cast<uint4*>(v2 + r * bw * A.XV + x) =
                                    make_uint4(b[r].x + p2, b[r].y + p2, b[r].z + p2, b[r].w + p2);
                            }
                            c1[r] += __shfl_sync(kFull, t1[r], 31);
                            c2[r] += __shfl_sync(kFull, t2[r], 31);
                        }
                    }
                    __syncwarp();
                    for (int r = 0; r < rows; ++r) {
                        const int ri = ring(i + r * bw);
                        const uint32_t* w1 = v1 + r * bw * A.XV;
                        const uint32_t* w2 = v2 + r * bw * A.XV;
                        for (int j = lane; j < nc; j += 32) {
                            const uint32_t s1 = w1[j + cw - 1] - (j > 0 ? w1[j - 1] : 0u);
                            const uint32_t s2 = w2[j + cw - 1] - (j > 0 ? w2[j - 1] : 0u);
                            s_S[j * A.NRS + ri] = make_uint2(s1, s2);
                            if (roots) s_R[j * A.NRS + ri] = recip2(make_uint2(s1, s2), make_uint2(s1, s2)).x;
                        }
                    }
                }
                if (ie < nr) bar_box();  // the next stripe overwrites the sums
            }
        };
        if (A.big) {
            box_sums(kTcThreads);
            __syncthreads();  // the chip chunks overwrite the stripe
        }

        const int nchunk = (cw + A.BC - 1) / A.BC;
        bool ok = true;
        for (int cc = 0; cc < nchunk; ++cc) {
            const int b0 = cc * A.BC, b1 = min(cw, b0 + A.BC);
            if (cc > 0) {
                // The previous chunk's products must be done before its rows are replaced.
                ok = tc::mbar_wait(&s_mbar, phase, kTcWaitPolls);
                phase ^= 1u;
                ok = !__syncthreads_or(!ok);
                if (!ok) break;
                tc::fence_after_sync();
            }
            // E: NB rows u = 16 - NB ... 15 per chip column, row u at e = u - 16 + NB: 16 bytes
            // from chip row -u - delta. Consecutive threads take consecutive rows.
            {
                const int nrow = (b1 - b0) * A.NB;
                int bl = tid / A.NB, e = tid - bl * A.NB;
                const int sbl = bd / A.NB, se = bd - sbl * A.NB;
                for (int t = tid; t < nrow; t += bd) {
                    const int src = (b0 + bl) * A.PC + kPadL - 16 + A.NB - static_cast<int>(delta) - e;
                    const uint32_t* w = reinterpret_cast<const uint32_t*>(s_P + (src & ~3));
                    const uint32_t sh = static_cast<uint32_t>(src & 3) * 8u;
                    uint4 o;
                    o.x = __funnelshift_r(w[0], w[1], sh);
                    o.y = __funnelshift_r(w[1], w[2], sh);
                    o.z = __funnelshift_r(w[2], w[3], sh);
                    o.w = __funnelshift_r(w[3], w[4], sh);
                    *reinterpret_cast<uint4*>(s_E + bl * A.PS + e * 16) = o;
                    bl += sbl;
                    e += se;
                    if (e >= A.NB) {
                        e -= A.NB;
                        ++bl;
                    }
                }
            }
            if (cc == 0 && warp < 4) {
                // Clear the accumulator columns the products add into (one lane quarter each).
                uint32_t z[16];
#pragma unroll
                for (int t = 0; t < 16; ++t) z[t] = 0u;
                // Products land in columns [NB - 16, NB + nr) of block coordinates (their rows are
                // trimmed to the surface rows), stored from column 0 of each accumulator.
                const int zc = (nr + 16 + 15) & ~15;
                const uint32_t lq = taddr + (static_cast<uint32_t>(32 * warp) << 16);
                for (int s = 0; s < NI; ++s)
                    for (int c = 0; c < zc; c += 16)
                        tc::tmem_st16(lq + static_cast<uint32_t>(s) * acc1 + static_cast<uint32_t>(c), z);
                tc::tmem_wait_st();
            }
            tc::fence_proxy_async_smem();
            tc::fence_before_sync();
            __syncthreads();
            TC_PHASE(5)
            // Lane 0 of each of the last NI warps issues the products of a share of the
            // chunk's chip column pairs into its own accumulator (one thread's MMAs run one after
            // another, so the products of one point are spread over two or four threads).
            if (lane == 0 && warp >= nwarps - NI) {
                const int stream = nwarps - 1 - warp;
                tc::fence_after_sync();
                const uint32_t sW = tc::smem_u32(s_W), sE = tc::smem_u32(s_E);
                const int p0 = b0 / 2, p1 = b1 / 2;
                const int tb = p0 + (p1 - p0) * stream / NI;
                const int te = p0 + (p1 - p0) * (stream + 1) / NI;
                const uint32_t dacc = taddr + static_cast<uint32_t>(stream) * acc1;
                for (int q = 0; q < Q; ++q) {
                    // Only the operand rows e in [elo, elo + n) of block q reach surface rows;
                    // their accumulator columns start at NB - 16 in block coordinates.
                    int elo, n;
                    if (!block_rows(q, A.NB, nr, &elo, &n)) continue;
                    const uint32_t idesc = tc::idesc_u8_s32(A.MT, n);
                    const uint32_t dcol = static_cast<uint32_t>(16 * q + elo - (A.NB - 16));
                    for (int t = tb; t < te; ++t) {
                        const uint64_t da = tc::smem_desc(sW + q * A.QS + 32 * t, 16, 128);
                        const uint64_t db =
                            tc::smem_desc(sE + (2 * t - b0) * A.PS + 16 * elo, A.PS, 128);
                        tc::mma_u8(dacc + dcol, da, db, idesc, true);
                    }
                }
                tc::mma_commit(&s_mbar);
            }
            if (cc == 0 && !A.big && warp < nwarps - NI) box_sums(kTcThreads - 32 * NI);
            TC_PHASE(6)
        }
        if (ok) {
            // Wait for the last chunk's products (bounded; every thread polls the same phase).
            ok = tc::mbar_wait(&s_mbar, phase, kTcWaitPolls);
            phase ^= 1u;
        }
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicExch(A.status, 1);
            failed = true;
            break;
        }
        tc::fence_after_sync();
        TC_PHASE(7)

        // Pass 1: numerators out of Tensor Memory, estimates and bounds, the largest lower bound.
        // Surface column j is accumulator row j (lane (j % 16) + 32 (j / 16) of the M = 64
        // layout); surface row i is column i of each accumulator (their sum). Warp w reads its quarter's
        // 16 lanes (16x256b: thread t gets rows 16 q + t/4 and + 8, columns 2 (t % 4) + {0, 1}
        // + 8 k), columns from 32 (w / 4) in steps of 64.
        const float kk = __double2float_rn(
            A.measure == AR_NCC ? __drcp_rn(__dmul_rn(cnorm, nn))
                                : __drcp_rn(__dmul_rn(cnorm, __dsqrt_rn(nn))));
        const float kk7 = 4.172325134277344e-07f * kk;  // 7u k
        const float csf = static_cast<float>(csum_d);
        const int quarter = warp & 3, half = warp >> 2;
        unsigned long long best = 0ull;
        int pi = 0, pj = 0;  // the peak
        // The peak or its 5 x 5 patch (all inside the surface): the numerators of the output.
        const bool single = A.up == 1 || nr < 5 || nc < 5;
        const int span = single ? 1 : 5;
        // The products are here and nothing below gives up, so the patch of this slot of the
        // refinement queue will be written (k_refine trusts the count). Read after later barriers.
        if (tid == 0 && !single) s_slot = atomicAdd(A.sub_count, 1);
        int pi0 = 0, pj0 = 0;
        auto patch_at = [&](int i, int j) {
            pi = i;
            pj = j;
            pi0 = single ? pi : min(max(pi - 2, 0), max(nr - 5, 0));
            pj0 = single ? pj : min(max(pj - 2, 0), max(nc - 5, 0));
        };
        auto patch_of = [&](unsigned long long key) {
            unsigned rm = 0;
            float pv = 0.0f;
            if (key_decode(key, &rm, &pv)) patch_at(static_cast<int>(rm / nc), static_cast<int>(rm % nc));
            else patch_at(0, 0);
        };
        if constexpr (REG) {
            float lmax = -INFINITY;
            // One read per warp: value v of this thread is surface row
            // i = 32 half + 8 (v / 4) + 2 (lane % 4) + v % 2, column j = 16 quarter + lane / 4
            // (+ 8 when v % 4 >= 2). Registers keep its numerator and its upper bound.
            const int ib0 = 32 * half + 2 * (lane & 3);
            const int jb0 = 16 * quarter + (lane >> 2);
            uint32_t dv[16];
            float upb[16];
            uint32_t vm = 0u;  // values of this thread inside the surface
            if (32 * half < nr) {
                const uint32_t base = taddr + (static_cast<uint32_t>(32 * quarter) << 16) +
                                      static_cast<uint32_t>(32 * half);
                uint32_t dv1[16];
                tc::tmem_ld16dp(base, dv);
                tc::tmem_ld16dp(base + acc1, dv1);
                tc::tmem_wait_ld();
#pragma unroll
                for (int v = 0; v < 16; ++v) dv[v] += dv1[v];
                for (int s = 2; s < NI; ++s) {
                    tc::tmem_ld16dp(base + static_cast<uint32_t>(s) * acc1, dv1);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int v = 0; v < 16; ++v) dv[v] += dv1[v];
                }
#pragma unroll
                for (int v = 0; v < 16; ++v) {
                    const int i = ib0 + 8 * (v >> 2) + (v & 1), j = jb0 + ((v & 2) ? 8 : 0);
                    upb[v] = -INFINITY;
                    if (i < nr && j < nc) {
                        vm |= 1u << v;
                        const int o = j * A.NRS + ring(i);
                        float bnd;
                        const float est = tc_estimate(dv[v], s_S[o].x, s_S[o].y, nnf, csf, kk, kk7,
                                                      A.measure, &bnd);
                        upb[v] = est + bnd;
                        lmax = fmaxf(lmax, est - bnd);
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(kFull, lmax, o));
            if (lane == 0) s_fmax[warp] = lmax;
            if (tid == 0) s_ncand = 0;
            __syncthreads();
            TC_PHASE(8)
            float M = s_fmax[0];
            for (int w = 1; w < kTcThreads / 32; ++w) M = fmaxf(M, s_fmax[w]);
            // Pass 2: values whose upper bound reaches M (or whose estimate was not made) go to a
            // list -- numerator and (row, column) -- and are normalised exactly, one per thread.
            uint32_t* s_cD = s_num;
            uint32_t* s_cI = reinterpret_cast<uint32_t*>(s_est);
#pragma unroll
            for (int v = 0; v < 16; ++v) {
                if (((vm >> v) & 1u) && (upb[v] >= M || isnan(upb[v]))) {
                    const int c = atomicAdd(&s_ncand, 1);
                    s_cD[c] = dv[v];
                    s_cI[c] = (static_cast<uint32_t>(ib0 + 8 * (v >> 2) + (v & 1)) << 16) |
                              static_cast<uint32_t>(jb0 + ((v & 2) ? 8 : 0));
                }
            }
            __syncthreads();
            const int ncand = s_ncand;
            for (int c = tid; c < ncand; c += bd) {
                const int i = static_cast<int>(s_cI[c] >> 16), j = static_cast<int>(s_cI[c] & 0xFFFFu);
                const int o = j * A.NRS + ring(i);
                const float x = tc_exact(s_cD[c], s_S[o].x, s_S[o].y, mean, nn, cnorm, A.measure);
                const unsigned long long key = argmax_key(x, static_cast<unsigned>(i * nc + j));
                best = key > best ? key : best;
            }
            best = block_max_u64(best, reinterpret_cast<unsigned long long*>(s_red));
            TC_PHASE(9)
            if (A.flops && tid == 0)
                atomicAdd(A.flops, 2ull * static_cast<unsigned long long>(ch) * cw * nr * nc);
            if (A.surf_out) {
                // Every value exactly (diagnostic surfaces): numerators to shared memory first.
#pragma unroll
                for (int v = 0; v < 16; ++v)
                    if ((vm >> v) & 1u)
                        s_num[(jb0 + ((v & 2) ? 8 : 0)) * A.NRS + ib0 + 8 * (v >> 2) + (v & 1)] = dv[v];
                __syncthreads();
                float* so = A.surf_out + k * static_cast<int64_t>(A.NRM) * A.NCM;
                for (int e = tid; e < nr * nc; e += bd) {
                    const int o = (e / nr) * A.NRS + (e % nr);
                    const int os = (e / nr) * A.NRS + ring(e % nr);
                    so[e] = tc_exact(s_num[o], s_S[os].x, s_S[os].y, mean, nn, cnorm, A.measure);
                }
            }
            patch_of(best);
#pragma unroll
            for (int v = 0; v < 16; ++v) {
                const int a = ib0 + 8 * (v >> 2) + (v & 1) - pi0, b = jb0 + ((v & 2) ? 8 : 0) - pj0;
                if (a >= 0 && a < span && b >= 0 && b < span && ((vm >> v) & 1u)) s_pd[b * 5 + a] = dv[v];
            }
        } else {
            // Numerators out of Tensor Memory, of surface rows ilo .. ihi - 1 and columns
            // jlo .. jhi - 1 and more beside them: fn(two numerators, the even row of the first, column),
            // rows (an even number) and columns beyond the surface included. M = 128: accumulator row j is lane j, a thread reads 16
            // columns; M = 64 as above.
            auto visit = [&](int ilo, int ihi, int jlo, int jhi, auto&& fn) {
                uint32_t r[16], r1[16];
                if (A.MT == 64) {
                    if (16 * quarter >= jhi || 16 * quarter + 16 <= jlo) return;
                    for (int i0 = 32 * half; i0 < nr; i0 += 64) {
                        if (i0 >= ihi || i0 + 32 <= ilo) continue;
                        const uint32_t base = taddr + (static_cast<uint32_t>(32 * quarter) << 16) +
                                              static_cast<uint32_t>(i0);
                        tc::tmem_ld16dp(base, r);
                        for (int s = 1; s < NI; ++s) {
                            tc::tmem_ld16dp(base + static_cast<uint32_t>(s) * acc1, r1);
                            tc::tmem_wait_ld();
#pragma unroll
                            for (int v = 0; v < 16; ++v) r[v] += r1[v];
                        }
#pragma unroll
                        for (int v = 0; v < 16; v += 2)
                            fn(r[v], r[v + 1], i0 + 8 * (v >> 2) + 2 * (lane & 3),
                               16 * quarter + (lane >> 2) + ((v & 2) ? 8 : 0));
                    }
                } else {
                    if (32 * quarter >= jhi || 32 * quarter + 32 <= jlo) return;
                    for (int i0 = 16 * half; i0 < nr; i0 += 32) {
                        if (i0 >= ihi || i0 + 16 <= ilo) continue;
                        const uint32_t base = taddr + (static_cast<uint32_t>(32 * quarter) << 16) +
                                              static_cast<uint32_t>(i0);
                        tc::tmem_ld16(base, r);
                        for (int s = 1; s < NI; ++s) {
                            tc::tmem_ld16(base + static_cast<uint32_t>(s) * acc1, r1);
                            tc::tmem_wait_ld();
#pragma unroll
                            for (int v = 0; v < 16; ++v) r[v] += r1[v];
                        }
#pragma unroll
                        for (int v = 0; v < 16; v += 2) fn(r[v], r[v + 1], i0 + v, 32 * quarter + lane);
                    }
                }
            };
            // The estimate of a value, times kz, and the error bound `bu` of all of them as in
            // k_corr_tc2 (its pass 1): reciprocal roots carried with the box sums, no bound a value,
            // no surface in shared memory. With a bound for each value, numerators and upper bounds
            // staged for a second pass over all of them, these two passes took 11 k of a point's
            // 31.7 k cycles at chip 32, surface 88 x 88.
            auto estimate = [&](uint32_t d0, uint32_t d1, int o0, int o1) {
                const uint2 a = s_S[o0], b = s_S[o1];
                const float2 s1 = make_float2(__uint2float_rn(a.x), __uint2float_rn(b.x));
                const float2 nx = __ffma2_rn(make_float2(nnf, nnf),
                                             make_float2(__uint2float_rn(d0), __uint2float_rn(d1)),
                                             neg2(__fmul2_rn(make_float2(csf, csf), s1)));
                return __fmul2_rn(nx, roots ? make_float2(s_R[o0], s_R[o1]) : recip2(a, b));
            };
            const float u24 = 6.0200e-08f;  // 1.01 x 2^-24
            const float kz = sqrtf(static_cast<float>(sq) * nnf);
            const float kc = sqrtf(nnf * static_cast<float>(sq + csum_d * mean));
            const float bu = A.measure == AR_NCC ? u24 * sqrtf(nnf) * (20.0f * kz + 5.0f * kc)
                                                 : u24 * (3400.0f * kz + 160.0f * kc);
            float sum = 0.0f;                          // NaN when an estimate was not made
            float own = -INFINITY, own2 = -INFINITY;  // this thread's two largest estimates
            int at = 0;                               // where the largest is
            // The ring places of rows i and i + 1 (of the last two for rows beyond the surface).
            auto places = [&](int i, int j, int* o0, int* o1) {
                const unsigned r = static_cast<unsigned>(min(i, nr - 2) + rbase);
                const unsigned n = static_cast<unsigned>(A.NRS), base = min(j, nc - 1) * n;
                *o0 = static_cast<int>(base + min(r, r - n));
                *o1 = static_cast<int>(base + min(r + 1u, r + 1u - n));
            };
            visit(0, nr, 0, nc, [&](uint32_t d0, uint32_t d1, int i, int j) {
                const bool in = i < nr && j < nc;
                int o0, o1;
                places(i, j, &o0, &o1);
                const float2 e = estimate(d0, d1, o0, o1);
                sum += in ? e.x + e.y : 0.0f;
                const float hi = in ? fmaxf(e.x, e.y) : -INFINITY, lo = in ? fminf(e.x, e.y) : -INFINITY;
                own2 = fmaxf(own2, fmaxf(lo, fminf(own, hi)));
                at = hi > own ? ((e.y > e.x ? i + 1 : i) << 16) | j : at;
                own = fmaxf(own, hi);
            });
            {
                const float top = warp_max(own);
                const unsigned who = __ballot_sync(kFull, own == top && own > -INFINITY);
                const int first = who ? __ffs(who) - 1 : 0;
                const float sec = warp_max(isnan(sum) ? INFINITY : lane == first ? own2 : own);
                if (lane == first) {
                    s_fmax[warp] = top;
                    s_sec[warp] = sec;
                    s_at[warp] = at;
                }
            }
            __syncthreads();
            TC_PHASE(8)
            // Is the largest estimate more than the bound above every other?
            constexpr int kW = kTcThreads / 32;
            const float wt = lane < kW ? s_fmax[lane] : -INFINITY;
            const float M = warp_max(wt);
            const float cut = M - 2.0f * bu;
            const int mw = __ffs(__ballot_sync(kFull, wt == M)) - 1;
            const bool unique =
                M > -INFINITY && !__any_sync(kFull, lane < kW && (!(s_sec[lane & (kW - 1)] < cut) ||
                                                                  (lane != mw && !(wt < cut))));
            if (unique) {
                // Every other value is below this one: it is the strict (so the first) maximum.
                patch_at(s_at[mw] >> 16, s_at[mw] & 0xFFFF);
            } else {
                // The values whose estimate is within the bounds of the largest (or was not made),
                // exactly.
                visit(0, nr, 0, nc, [&](uint32_t d0, uint32_t d1, int i, int j) {
                    if (i >= nr || j >= nc) return;
                    int o[2];
                    places(i, j, &o[0], &o[1]);
                    const float2 e = estimate(d0, d1, o[0], o[1]);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if ((u ? e.y : e.x) < cut) continue;
                        const float x = tc_exact(u ? d1 : d0, s_S[o[u]].x, s_S[o[u]].y, mean, nn, cnorm, A.measure);
                        const unsigned long long key = argmax_key(x, static_cast<unsigned>((i + u) * nc + j));
                        best = key > best ? key : best;
                    }
                });
                best = block_max_u64(best, reinterpret_cast<unsigned long long*>(s_red));
                patch_of(best);
            }
            TC_PHASE(9)
            if (A.flops && tid == 0)
                atomicAdd(A.flops, 2ull * static_cast<unsigned long long>(ch) * cw * nr * nc);
            if (A.surf_out) {
                float* so = A.surf_out + k * static_cast<int64_t>(A.NRM) * A.NCM;
                visit(0, nr, 0, nc, [&](uint32_t d0, uint32_t d1, int i, int j) {
                    if (i >= nr || j >= nc) return;
                    int o0, o1;
                    places(i, j, &o0, &o1);
                    so[j * nr + i] = tc_exact(d0, s_S[o0].x, s_S[o0].y, mean, nn, cnorm, A.measure);
                    so[j * nr + i + 1] = tc_exact(d1, s_S[o1].x, s_S[o1].y, mean, nn, cnorm, A.measure);
                });
            }
            visit(pi0, pi0 + span, pj0, pj0 + span, [&](uint32_t d0, uint32_t d1, int i, int j) {
                const int a = i - pi0, b = j - pj0;
                if (i < nr && b >= 0 && b < span) {
                    if (a >= 0 && a < span) s_pd[b * 5 + a] = d0;
                    if (a + 1 >= 0 && a + 1 < span) s_pd[b * 5 + a + 1] = d1;
                }
            });
        }
        __syncthreads();
        if (single) {
            if (tid == 0) {
                const int o = pj * A.NRS + ring(pi);
                A.out.dx[k] = __double2float_rn(
                    __dadd_rn(static_cast<double>(pj - static_cast<int>(prx)), A.pts.dx0[k]));
                A.out.dy[k] = __double2float_rn(
                    __dadd_rn(static_cast<double>(pi - static_cast<int>(pry)), A.pts.dy0[k]));
                A.out.corr[k] = tc_exact(s_pd[0], s_S[o].x, s_S[o].y, mean, nn, cnorm, A.measure);
            }
        } else {
            const int slot = s_slot;
            if (tid < 25) {
                const int a = tid % 5, b = tid / 5;
                const int o = (pj0 + b) * A.NRS + ring(pi0 + a);
                A.sub_patch[static_cast<int64_t>(slot) * 25 + tid] =
                    tc_exact(s_pd[tid], s_S[o].x, s_S[o].y, mean, nn, cnorm, A.measure);
            }
            if (tid == 0) {
                A.sub_point[slot] = k;
                A.sub_origin[2 * slot] = pi0;
                A.sub_origin[2 * slot + 1] = pj0;
            }
        }
        TC_PHASE(10)
        TC_PHASE_POINT
    }
    TC_PHASE_FLUSH
    if (failed) {
        // Products may still be in flight: give them a bounded time before freeing the
        // accumulator.
        tc::mbar_wait(&s_mbar, phase ^ 1u, kTcWaitPolls);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(taddr, A.tmem_cols);
}

// ----------------------------------------------------------------------------------------------
// Tensor-core correlation, surfaces up to 64 x 64 with the chip operand whole (k_corr_tc2).
//
// The window is staged from its first row (no alignment offset; each 16-byte block of a column
// is realigned from the aligned 16-byte chunks cp.async copied into shared memory, or from two
// aligned global loads), so block q of 16 rows meets surface rows i in [16 q - ch + 1,
// 16 q + 15]: NB = 16 * ceil((ch + 15) / 16) rows of the chip operand E_b[u][r] = C[r - u, b]
// (u = 16 - NB ... 15). A block's product lands at accumulator column 16 q + e - (NB - 16) for
// its operand row e, so surface row i is column i and the products of four issuing threads
// (lane 0 of the last four of eight main warps) write four accumulators. The box sums come from
// the 16-byte window blocks: column sums V down ch rows (dp4a for the first row, a sliding update
// for the rest), then row sums. A fetch warp stages the next point's window and chip and a patch
// warp writes the last point's patch while the main warps work on this one. Estimates stay in
// registers; the patch, and the values the bound does not separate from the largest, get the
// reference's FP64 normalisation.

// A point's chip and window placement (src/points.jl:358-395 with the pass's padding and the
// +0.5 shift, src/track.jl:128-138, 207-220) and whether it is searched at all.
struct PtGeo {
    long long k, chip_r, chip_c, win_r, win_c;
    int ch, cw, nr, nc, prx, pry, ok;
};

__device__ __forceinline__ void pt_geometry(const TcArgs& A, int64_t k, PtGeo& g) {
    // All eight fields are loaded before any is used.
    const int64_t prx = A.pts.rx[k], pry = A.pts.ry[k];
    const double x = A.pts.x[k], y = A.pts.y[k], dx0 = A.pts.dx0[k], dy0 = A.pts.dy0[k];
    const int64_t csx = A.pts.csx[k], csy = A.pts.csy[k];
    const int64_t NR = A.nrows + 2 * A.pady, NC = A.ncols + 2 * A.padx;
    g.k = k;
    g.ok = 0;
    if (!(prx > 0 && pry > 0)) return;
    const double xs = x + (static_cast<double>(A.padx) + 0.5);
    const double ys = y + (static_cast<double>(A.pady) + 0.5);
    const int64_t hx = csx / 2, hy = csy / 2;
    const int64_t ccx = static_cast<int64_t>(floor(__dsub_rn(xs, dx0)));
    const int64_t ccy = static_cast<int64_t>(floor(__dsub_rn(ys, dy0)));
    const int64_t wcx = static_cast<int64_t>(floor(xs)), wcy = static_cast<int64_t>(floor(ys));
    const int64_t cr0 = ccy - hy, cr1 = ccy + hy - 1, cc0 = ccx - hx, cc1 = ccx + hx - 1;
    const int64_t wr0 = wcy - hy - pry, wr1 = wcy + hy + pry - 2;
    const int64_t wc0 = wcx - hx - prx, wc1 = wcx + hx + prx - 2;
    const bool chip_in = (cr1 < cr0 || cc1 < cc0) ||
                         (cr0 >= 1 && cr1 <= NR && cc0 >= 1 && cc1 <= NC);
    const bool win_in = (wr1 < wr0 || wc1 < wc0) ||
                        (wr0 >= 1 && wr1 <= NR && wc0 >= 1 && wc1 <= NC);
    if (!chip_in || !win_in) return;
    g.ch = static_cast<int>(2 * hy);
    g.cw = static_cast<int>(2 * hx);
    g.nr = static_cast<int>(2 * pry);
    g.nc = static_cast<int>(2 * prx);
    g.prx = static_cast<int>(prx);
    g.pry = static_cast<int>(pry);
    if (g.ch <= 0 || g.cw <= 0) return;
    if (g.ch > A.CHM || g.cw > A.CWM || g.nr > A.NRM || g.nc > A.NCM) return;
    g.chip_r = cr0 - 1 - A.pady;
    g.chip_c = cc0 - 1 - A.padx;
    g.win_r = wr0 - 1 - A.pady;
    g.win_c = wc0 - 1 - A.padx;
    g.ok = 1;
}

// One CTA is eight main warps, a fetch warp and a patch warp, two CTAs to an SM. The fetch warp reads the points ahead (geometry of 32 points at a time, one per lane)
// and copies the next point's window, chip and mask chunks into shared memory with cp.async
// while the current point's peak is found. The patch warp turns the 5 x 5 numerators of a finished
// point into the exact FP64 patch. So the main warps see neither global latency nor the FP64
// chains: they stage the operands, issue the products (lane 0 of the last A.issuers warps, each
// into its own accumulator), sum the boxes beside them, and find the peak. They meet the fetch warp
// at two mbarriers (`full`: a point's geometry and chunks are in place, `free`: the chunks and the
// column sums that share their space are read) and the patch warp at a barrier before the
// products and at `out` (the patch is handed over); the waits on mbarriers are bounded, and
// whoever gives up still takes the others to their next barrier.
//
// Bound: instruction issue of the CUDA-core work around the products (15 k warp instructions a point
// at chip 32 / radius 25; 51 % issue utilisation with two CTAs of 96 registers a thread, tensor
// pipe 20 %). Measured on that pass, 251 001 points: 9.96 ms before the extra warps, with three
// issuing warps that also made the chip's FP64 statistics and the next geometry, patches in a main
// warp, a bound computed with every estimate and column sums started afresh for every point; 6.99 ms
// now. Three CTAs of 64 registers (two accumulators, no ring of reciprocal roots) measured 7.83 ms,
// products issued by four lanes of the patch warp 7.60 ms, by two lanes each of the fetch and patch
// warps 8 % above this.
struct Tc2Pt {
    long long k;  // point, or -1: no more points
    long long chip_r, chip_c, win_r, win_c;
    int ch, cw, nr, nc;
    int raw;       // bit 0: the window's chunks are in s_rawW, bit 1: the chip's and mask's in s_rawC
};

// A finished point, for the patch warp.
struct Tc2Out {
    long long k;
    int nr, nc, nn;
    int kind;      // 1: the peak alone, 2: the patch
    int pi, pj;    // the peak (kind 1) or the patch's first row and column
    uint32_t cs, c2;      // chip sums (power-of-two areas)
    double mean, sq, csum;  // chip statistics (other areas)
    uint32_t D[25], s2[25];
    float s1[25];
};

__device__ __forceinline__ const uint8_t* align16(const uint8_t* p) {
    return reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(p) & ~uintptr_t(15));
}
__device__ __forceinline__ uint32_t tc2_low(const uint8_t* p) {
    return static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p));
}

// Power-of-two chip areas up to 4096 pixels: every term of the reference's FP64 chip sums is exact,
// so mean = sum / nn and sq = (nn sum(C^2) - sum(C)^2) / nn.
__device__ __forceinline__ bool tc2_exact_sums(int nn) { return (nn & (nn - 1)) == 0 && nn <= 4096; }
__device__ __forceinline__ void tc2_chip_stats(int nn, uint32_t cs, uint32_t c2, double* mean, double* sq) {
    const unsigned long long d =
        static_cast<unsigned long long>(nn) * c2 - static_cast<unsigned long long>(cs) * cs;
    *mean = __ddiv_rn(static_cast<double>(cs), static_cast<double>(nn));
    *sq = __ddiv_rn(static_cast<double>(d), static_cast<double>(nn));
}

__device__ __forceinline__ void bar_main() { block_sync<true>(); }
// The main warps and the patch warp.
__device__ __forceinline__ void bar_products() { asm volatile("bar.sync 3, 288;" ::: "memory"); }
__device__ __forceinline__ bool bar_main_or(bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, 2, 256, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t"
        "}\n"
        : "=r"(r)
        : "r"(static_cast<uint32_t>(v))
        : "memory");
    return r != 0u;
}

// The rare paths as calls, so that their code stays out of the point loop: sixteen image rows at
// the image's border, and an exact value.
__device__ __noinline__ uint4 tc2_border(const uint8_t* img, const uint8_t* img_end, int64_t nrows,
                                         int64_t ncols, int64_t c, int64_t r0) {
    return col16_finish(col16_issue(img, img_end, nrows, ncols, c, r0));
}
__device__ __noinline__ float tc2_exact(uint32_t D, float s1, uint32_t s2, double mean, double nn,
                                        double cnorm, int measure) {
    return tc_exact(D, __float2uint_rn(s1), s2, mean, nn, cnorm, measure);
}

__global__ void __launch_bounds__(kTc2Threads, 2) k_corr_tc2(const TcArgs A) {
    extern __shared__ __align__(1024) unsigned char smem_tc[];
    __shared__ uint64_t s_mbar, s_full, s_free, s_outb[2];
    __shared__ uint32_t s_taddr;
    __shared__ int s_fail, s_more[2];  // s_more, by result slot: a measured point, or the end
    __shared__ int s_lost;             // the patch warp gave up on a point
    __shared__ float s_bu;
    __shared__ float s_top[8], s_sec[8];
    __shared__ int s_at[8];
    __shared__ uint32_t s_isum[2][2];
    __shared__ Tc2Pt s_pt[2];   // by the parity of the point's number in this CTA
    __shared__ Tc2Out s_out[2];
    uint8_t* s_E = smem_tc + A.off_E;
    uint8_t* s_W = smem_tc + A.off_W;
    uint8_t* s_P = smem_tc + A.off_P;
    uint32_t* s_V1 = reinterpret_cast<uint32_t*>(smem_tc + A.off_V);
    uint32_t* s_V2 = s_V1 + A.VR * A.XV + 16;
    uint32_t* s_L1 = reinterpret_cast<uint32_t*>(smem_tc + A.off_L);
    uint32_t* s_L2 = s_L1 + A.XV;
    uint4* s_rawW = reinterpret_cast<uint4*>(smem_tc + A.off_rawW);
    uint4* s_rawC = reinterpret_cast<uint4*>(smem_tc + A.off_rawC);
    float* s_S1 = reinterpret_cast<float*>(smem_tc + A.off_S1);
    uint32_t* s_S2 = reinterpret_cast<uint32_t*>(smem_tc + A.off_S2);
    float* s_R = reinterpret_cast<float*>(smem_tc + A.off_est);
    uint32_t* s_num = reinterpret_cast<uint32_t*>(smem_tc + A.off_num);
    double* s_red = reinterpret_cast<double*>(smem_tc + A.off_red);

    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const uint8_t* ref_end = A.ref + A.nrows * A.ncols;
    const uint8_t* sec_end = A.sec + A.nrows * A.ncols;
    const uint8_t* valid_end = A.valid + A.nrows * A.ncols;

    if (warp == 0) {
        tc::tmem_alloc(&s_taddr, A.tmem_cols);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        tc::mbar_init(&s_mbar, A.issuers);  // one commit per issuing thread
        tc::mbar_init(&s_full, 1);
        tc::mbar_init(&s_free, 1);
        // One arrival per main warp. One per slot: a point's arrivals may come before the product
        // warp has seen its predecessor's.
        tc::mbar_init(&s_outb[0], 8);
        tc::mbar_init(&s_outb[1], 8);
        tc::fence_mbar_init();
        s_fail = s_lost = 0;
    }
    if (tid < 4) s_isum[tid >> 1][tid & 1] = 0u;
    for (int e = tid; e < A.CWM * A.PC; e += kTc2Threads) s_P[e] = 0;
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t taddr = s_taddr;
    const uint32_t acc1 = static_cast<uint32_t>(A.acc1_col);  // stride between accumulators
    // Clears the accumulator columns [32 half, 32 half + 32) of this warp's lane quarter.
    auto clear_acc = [&]() {
        uint32_t zero[16];
#pragma unroll
        for (int v = 0; v < 16; ++v) zero[v] = 0u;
        const uint32_t lq = taddr + (static_cast<uint32_t>(32 * (warp & 3)) << 16) +
                            static_cast<uint32_t>(32 * (warp >> 2));
        if (32u * static_cast<uint32_t>(warp >> 2) < acc1) {
            for (int v = 0; v < A.issuers; ++v) {
                tc::tmem_st16(lq + static_cast<uint32_t>(v) * acc1, zero);
                tc::tmem_st16(lq + static_cast<uint32_t>(v) * acc1 + 16u, zero);
            }
        }
    };

    // Each CTA takes a contiguous run of points: consecutive points of a grid column have the
    // same window columns one grid step lower, so most of their box sums carry over.
    const int64_t per = (A.pts.n + gridDim.x - 1) / gridDim.x;
    const int64_t kbeg = static_cast<int64_t>(blockIdx.x) * per;
    const int64_t kend = min(A.pts.n, kbeg + per);

    if (warp == 8) {
        // ------------------------------------------------------------------------------ helper
        int64_t kb = kbeg - 32;   // the lanes hold the geometry of points kb .. kb + 31
        unsigned okm = 0u;        // of those, the ones still to be correlated
        PtGeo mine{};
        // The next point to correlate and its chunks' copies, into slot `b`.
        auto fetch = [&](int b) {
            while (okm == 0u && kb + 32 < kend) {
                kb += 32;
                mine.ok = 0;
                if (kb + lane < kend) pt_geometry(A, kb + lane, mine);
                okm = __ballot_sync(kFull, mine.ok);
            }
            if (okm == 0u) {
                if (lane == 0) s_pt[b].k = -1;
                return false;
            }
            const int src = __ffs(okm) - 1;
            okm &= okm - 1u;
            const long long chip_r = __shfl_sync(kFull, mine.chip_r, src);
            const long long chip_c = __shfl_sync(kFull, mine.chip_c, src);
            const long long win_r = __shfl_sync(kFull, mine.win_r, src);
            const long long win_c = __shfl_sync(kFull, mine.win_c, src);
            const int ch = __shfl_sync(kFull, mine.ch, src), cw = __shfl_sync(kFull, mine.cw, src);
            const int nr = __shfl_sync(kFull, mine.nr, src), nc = __shfl_sync(kFull, mine.nc, src);
            const int XW = cw + nc - 1, RQ = (ch + nr - 1 + 15) / 16 + 1, RC = (ch + 15) / 16 + 1;
            // Chunks: the aligned 16-byte blocks that hold a column's rows, when every row lies in
            // the image and every block in the array.
            const uint8_t* w0 = A.ref + win_c * A.nrows + win_r;
            const uint8_t* w1 = w0 + static_cast<int64_t>(XW - 1) * A.nrows;
            const bool rw = win_r >= 0 && win_r + 16 * (RQ - 1) <= A.nrows && win_c >= 0 &&
                            win_c + XW <= A.ncols && align16(w0) >= A.ref &&
                            align16(w1) + 16 * RQ <= ref_end;
            const int64_t co = chip_c * A.nrows + chip_r, ce = co + static_cast<int64_t>(cw - 1) * A.nrows;
            const bool rc = chip_r >= 0 && chip_r + ch <= A.nrows && chip_c >= 0 &&
                            chip_c + cw <= A.ncols && align16(A.sec + co) >= A.sec &&
                            align16(A.sec + ce) + 16 * RC <= sec_end &&
                            align16(A.valid + co) >= A.valid &&
                            align16(A.valid + ce) + 16 * RC <= valid_end;
            if (lane == 0) {
                Tc2Pt& p = s_pt[b];
                p.k = kb + src;
                p.chip_r = chip_r;
                p.chip_c = chip_c;
                p.win_r = win_r;
                p.win_c = win_c;
                p.ch = ch;
                p.cw = cw;
                p.nr = nr;
                p.nc = nc;
                p.raw = (rw ? 1 : 0) | (rc ? 2 : 0);
            }
            if (rc) {
                const uint32_t inv = (65536u + static_cast<uint32_t>(RC) - 1u) / static_cast<uint32_t>(RC);
                for (int t = lane; t < cw * RC; t += 32) {
                    const int b2 = static_cast<int>((static_cast<uint32_t>(t) * inv) >> 16), kc = t - b2 * RC;
                    const int64_t o = co + static_cast<int64_t>(b2) * A.nrows;
                    tc::cp_async16(s_rawC + kc * cw + b2, align16(A.sec + o) + 16 * kc);
                    tc::cp_async16(s_rawC + (RC + kc) * cw + b2, align16(A.valid + o) + 16 * kc);
                }
            }
            if (rw) {
                const uint32_t inv = (65536u + static_cast<uint32_t>(RQ) - 1u) / static_cast<uint32_t>(RQ);
                for (int t = lane; t < XW * RQ; t += 32) {
                    const int x = static_cast<int>((static_cast<uint32_t>(t) * inv) >> 16), kq = t - x * RQ;
                    tc::cp_async16(s_rawW + kq * XW + x,
                                   align16(w0 + static_cast<int64_t>(x) * A.nrows) + 16 * kq);
                }
            }
            tc::cp_async_commit();
            return true;
        };
        auto publish = [&]() {
            tc::cp_async_wait_all();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&s_full);
        };
        bool more = fetch(0);
        publish();
        for (uint32_t b = 1, ph = 0; more; b ^= 1u, ph ^= 1u) {
            if (!__all_sync(kFull, tc::mbar_wait(&s_free, ph, kTcWaitPolls))) break;
            more = fetch(static_cast<int>(b));
            publish();
        }
    } else if (warp == 9) {
        // ----------------------------------------------------------------------------- patches
        uint32_t ph = 0;  // the phase of `out`: each slot's own, the same for two points
        for (int b = 0;; b ^= 1) {
            bar_products();
            if (!s_more[b]) break;
            const Tc2Out& o = s_out[b];
            const int nnl = o.nn;
            const bool pow2 = tc2_exact_sums(nnl);
            const double nn = static_cast<double>(nnl);
            double mean = o.mean, sq = o.sq;
            if (pow2) tc2_chip_stats(nnl, o.cs, o.c2, &mean, &sq);
            const double cnorm = __dsqrt_rn(sq);
            if (!__all_sync(kFull, tc::mbar_wait(&s_outb[b], ph, kTcWaitPolls))) {
                // The main warps left, or are late: this point's output is lost, which the status
                // says in the end whatever they do. They are not told, as a flag set here could come
                // between two main threads' reads of it: some would leave and the others wait for them.
                if (lane == 0) s_lost = 1;
                __syncwarp();
                ph ^= static_cast<uint32_t>(b);
                continue;
            }
            ph ^= static_cast<uint32_t>(b);
            const bool patch = o.kind == 2;
            int slot = 0;
            if (patch && lane == 0) slot = atomicAdd(A.sub_count, 1);
            float v = 0.0f;
            if (lane < (patch ? 25 : 1)) v = tc2_exact(o.D[lane], o.s1[lane], o.s2[lane], mean, nn, cnorm, A.measure);
            if (patch) {
                slot = __shfl_sync(kFull, slot, 0);
                if (lane < 25) A.sub_patch[static_cast<int64_t>(slot) * 25 + lane] = v;
                if (lane == 0) {
                    A.sub_point[slot] = o.k;
                    A.sub_origin[2 * slot] = o.pi;
                    A.sub_origin[2 * slot + 1] = o.pj;
                }
            } else if (lane == 0) {
                A.out.dx[o.k] = __double2float_rn(__dadd_rn(static_cast<double>(o.pj - o.nc / 2), A.pts.dx0[o.k]));
                A.out.dy[o.k] = __double2float_rn(__dadd_rn(static_cast<double>(o.pi - o.nr / 2), A.pts.dy0[o.k]));
                A.out.corr[o.k] = v;
            }
            __syncwarp();
        }
    } else {
    // ------------------------------------------------------------------------------------ main
    uint32_t phase = 0, ph = 0;
    bool failed = false;
    int mb = 0;  // the slot of the next measured point's result
    clear_acc();
    int dirty_ch = 0;
    // This thread's row of the chip operand and its first chip column (the same for every point).
    const int e_groups = kTcThreads / A.NB;  // at least one: the plan holds NB to 256
    const int e_row = tid % A.NB, e_grp = tid / A.NB;
    TC_PHASE_INIT
    // Whether s_S1, s_S2 and s_R hold the previous point's box sums, as rings of NRS rows per
    // column: surface row i of that point is at row (i + rbase) mod NRS, so carrying the sums
    // down by `sh` rows advances rbase instead of moving them. s_L1, s_L2: its column sums of the
    // last surface row.
    bool held = false;
    int rbase = 0;
    auto ring = [&](int i) {
        const int r = i + rbase;
        return r >= A.NRS ? r - A.NRS : r;
    };
    for (int b = 0;; b ^= 1, ph ^= 1u) {
        // A wait that runs out leaves this thread with an empty point until the next barrier, where
        // all of them leave. Only main threads write s_fail, before that barrier, and each reads it
        // once after it and before another, so that they all see the same value.
        const bool got = tc::mbar_wait(&s_full, ph, kTcWaitPolls);
        if (!got) s_fail = 1;
        TC_PHASE(0)
        const Tc2Pt& g = s_pt[b];
        const int64_t k = got ? g.k : 0;
        if (k < 0) {
            bar_main_or(false);
            break;
        }
        const int ch = got ? g.ch : 0, cw = got ? g.cw : 0, nr = got ? g.nr : 0, nc = got ? g.nc : 0;
        const int64_t chip_r = g.chip_r, chip_c = g.chip_c, win_r = g.win_r, win_c = g.win_c;
        const int raw = g.raw;
        const int nnl = ch * cw;
        const bool pow2 = tc2_exact_sums(nnl);
        const int Q = (ch + nr - 1 + 15) / 16, XW = cw + nc - 1;
        Tc2Out& out = s_out[mb];
        // Carried box sums: the previous point (its slot is still in place) has the same window
        // columns and shape `sh` rows higher; only surface rows iA .. nr - 1 are new.
        int iA = 0;
        {
            const Tc2Pt& h = s_pt[b ^ 1];
            const int64_t sh = win_r - h.win_r;
            if (held && win_c == h.win_c && ch == h.ch && cw == h.cw && nr == h.nr && nc == h.nc &&
                sh > 0 && sh < nr)
                iA = nr - static_cast<int>(sh);
            held = false;
        }

        // The chip as zero-padded byte columns, _any_valid over it (src/track.jl:416-421) and its
        // exact integer sums; the window as blocks W[16 q + r][x] of 16 rows. A task is 16 rows of
        // one column, from the two chunks that hold them (or from global memory at the image's
        // border) shifted into place.
        int any = 0;
        uint32_t isum = 0u, isq = 0u;
        if (ch < dirty_ch)
            for (int c = warp; c < A.CWM; c += 8)
                for (int a = ch + lane; a < dirty_ch; a += 32) s_P[c * A.PC + kPadL + a] = 0;
        dirty_ch = ch;
        {
            const int nb16 = (ch + 15) >> 4, nct = nb16 * cw;
            const uint32_t ld = static_cast<uint32_t>(A.nrows);
            const uint32_t co = static_cast<uint32_t>(chip_c) * ld + static_cast<uint32_t>(chip_r);
            const uint32_t cbase = tc2_low(A.sec) + co, mbase = tc2_low(A.valid) + co;
            const uint32_t wbase = tc2_low(A.ref) + static_cast<uint32_t>(win_c) * ld + static_cast<uint32_t>(win_r);
            // Window tasks: a column and half of its blocks (the chunk between two blocks is read
            // once); chip tasks from the block's other end.
            const int qh = (Q + 1) >> 1;
            for (int w = tid; w < 2 * XW; w += kTcThreads) {
                const int up = w >= XW ? 1 : 0, x = w - up * XW;
                const int q0 = up * qh, q1 = min(q0 + qh, Q);
                uint8_t* dst = s_W + q0 * A.QS + x * 16;
                if (raw & 1) {
                    Col16 L;
                    L.s = (wbase + static_cast<uint32_t>(x) * ld) & 15u;
                    const uint4* src = s_rawW + q0 * XW + x;
                    L.lo = src[0];
                    for (int q = q0; q < q1; ++q) {
                        src += XW;
                        L.hi = src[0];
                        *reinterpret_cast<uint4*>(dst) = col16_finish(L);
                        L.lo = L.hi;
                        dst += A.QS;
                    }
                } else {
                    for (int q = q0; q < q1; ++q) {
                        *reinterpret_cast<uint4*>(dst) =
                            tc2_border(A.ref, ref_end, A.nrows, A.ncols, win_c + x, win_r + 16 * q);
                        dst += A.QS;
                    }
                }
            }
            for (int t = kTcThreads - 1 - tid; t < nct; t += kTcThreads) {
                const int kb = t / cw, c = t - kb * cw;
                uint4 v, mk;
                if (raw & 2) {
                    const uint4* rc = s_rawC + kb * cw + c;
                    const uint4* rm = rc + (nb16 + 1) * cw;
                    Col16 L;
                    L.lo = rc[0];
                    L.hi = rc[cw];
                    L.s = (cbase + static_cast<uint32_t>(c) * ld) & 15u;
                    v = col16_finish(L);
                    L.lo = rm[0];
                    L.hi = rm[cw];
                    L.s = (mbase + static_cast<uint32_t>(c) * ld) & 15u;
                    mk = col16_finish(L);
                } else {
                    v = tc2_border(A.sec, sec_end, A.nrows, A.ncols, chip_c + c, chip_r + 16 * kb);
                    mk = tc2_border(A.valid, valid_end, A.nrows, A.ncols, chip_c + c, chip_r + 16 * kb);
                }
                const int keep = ch - 16 * kb;
                uint32_t w[4] = {v.x, v.y, v.z, v.w}, mw[4] = {mk.x, mk.y, mk.z, mk.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = keep - 4 * i;
                    const uint32_t m = n >= 4 ? 0xffffffffu : n <= 0 ? 0u : (1u << (8 * n)) - 1u;
                    w[i] &= m;
                    any |= (mw[i] & m) != 0u;
                    isum = __dp4a(w[i], 0x01010101u, isum);
                    isq = __dp4a(w[i], w[i], isq);
                }
                *reinterpret_cast<uint4*>(s_P + c * A.PC + kPadL + 16 * kb) =
                    make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        if (pow2) {  // at most 4096 pixels: sums below 2^20 and 2^28
            isum = __reduce_add_sync(kFull, isum);
            isq = __reduce_add_sync(kFull, isq);
            if (lane == 0 && isq != 0u) {
                atomicAdd(&s_isum[b][0], isum);
                atomicAdd(&s_isum[b][1], isq);
            }
        }
        const bool seen = bar_main_or(any);
        if (s_fail) {
            failed = true;
            break;
        }
        TC_PHASE(1)
        const uint32_t cs = s_isum[b][0], c2 = s_isum[b][1];
        if (tid == 0) {
            if (seen) A.out.searched[k] = 1;
            s_isum[b ^ 1][0] = s_isum[b ^ 1][1] = 0u;  // for the next point
        }
        // prepare_chip! statistics. Power-of-two areas: the sum of squared deviations is
        // (nn sum(C^2) - sum(C)^2) / nn exactly, degenerate only when that integer is 0 (1 / nn is
        // above the threshold); the helper makes mean and norm. Other areas: the CUDA-core
        // kernel's FP64 sums.
        const unsigned long long nsq =
            static_cast<unsigned long long>(nnl) * c2 - static_cast<unsigned long long>(cs) * cs;
        bool measured = seen;
        if (seen) {
            if (pow2) {
                measured = nsq != 0ull;
            } else {
                double mean, sq, csum_d;
                staged_chip_stats<true>(s_P, A.PC, ch, cw, tid, kTcThreads, s_red, &csum_d, &mean, &sq);
                measured = sq > __dmul_rn(__dmul_rn(DBL_EPSILON, static_cast<double>(ch)), static_cast<double>(cw));
                if (measured && tid == 0) {
                    out.mean = mean;
                    out.sq = sq;
                    out.csum = csum_d;
                }
            }
        }
        if (!measured) {  // not searched, or degenerate: no measurement (src/track.jl:286)
            bar_main();
            if (tid == 0) tc::mbar_arrive(&s_free);
            continue;
        }
        TC_PHASE(2)

        // E: NB rows per chip column, row e (u = e - NB + 16) = 16 bytes from chip row -u. A thread
        // keeps its row, so its byte shift is fixed.
        auto build_row = [&](int e, int c) {
            const int src = c * A.PC + kPadL - 16 + A.NB - e;
            const uint32_t* w = reinterpret_cast<const uint32_t*>(s_P + (src & ~3));
            const uint32_t sh = static_cast<uint32_t>(src & 3) * 8u;
            uint4 o;
            o.x = __funnelshift_r(w[0], w[1], sh);
            o.y = __funnelshift_r(w[1], w[2], sh);
            o.z = __funnelshift_r(w[2], w[3], sh);
            o.w = __funnelshift_r(w[3], w[4], sh);
            *reinterpret_cast<uint4*>(s_E + c * A.PS + e * 16) = o;
        };
        if (e_grp < e_groups)
            for (int c = e_grp; c < cw; c += e_groups) build_row(e_row, c);
        if (tid == 0) {
            out.k = k;
            out.nr = nr;
            out.nc = nc;
            out.nn = nnl;
            out.cs = cs;
            out.c2 = c2;
            s_more[mb] = 1;
        }
        // The products add into accumulator columns [0, round16(nr)): surface row i is column i. The
        // accumulators were cleared when the previous point's were read.
        tc::tmem_wait_st();
        tc::fence_proxy_async_smem();
        tc::fence_before_sync();
        bar_products();  // s_P, s_W, s_E complete; accumulators clear; the chunks are read
        TC_PHASE(3)
        // The reciprocal root of a value's variance term (below).
        const float nnf = static_cast<float>(nnl);
        auto recip = [&](float s1, uint32_t s2u) {
            const float s2 = __uint2float_rn(s2u);
            float vx = s2;
            if (A.measure != AR_NCC) {
                const float q = __fmul_rn(s1, s1);
                vx = __fmaf_rn(nnf, s2, -q);
                if (__fmaf_rn(nnf, s2, q) > 2048.0f * vx) vx = -1.0f;  // its root is NaN
            }
            return s2u == 0u ? 0.0f : rsqrtf(vx);
        };
        const bool carry = iA > 0;
        if (carry) {
            rbase += nr - iA;
            if (rbase >= A.NRS) rbase -= A.NRS;
        } else {
            rbase = 0;
        }
#ifdef AR_TC_PHASES
        if (tid == 0 && carry) atomicAdd(&g_tc_phase[14], 1ull);
#endif
        const int nbox = kTcThreads - 32 * A.issuers;  // the threads that sum the boxes
        if (tid >= nbox) {
            // Each issuing thread takes a share of the chip column pairs (one thread issues an MMA
            // about every 120 cycles; several issuers, and other CTAs, interleave theirs).
            if (lane == 0) {
                const int stream = 7 - warp;
                tc::fence_after_sync();
#ifdef AR_TC_PHASES
                const unsigned long long tmi0 = clock64();
#endif
                // Descriptors advance by adding to their start-address field, the low bits of the
                // low word (16-byte units; shared addresses stay below 2^18, so nothing carries):
                // a product costs the issuing thread two 32-bit adds and the MMA itself.
                const uint64_t da0 = tc::smem_desc(tc::smem_u32(s_W), 16, 128);
                const uint64_t db0 = tc::smem_desc(tc::smem_u32(s_E), A.PS, 128);
                const uint32_t a_hi = static_cast<uint32_t>(da0 >> 32);
                const uint32_t b_hi = static_cast<uint32_t>(db0 >> 32);
                const uint32_t bstep = static_cast<uint32_t>(2 * A.PS) >> 4;
                const int pairs = cw / 2;
                const int t_begin = pairs * stream / A.issuers;
                const int npairs = pairs * (stream + 1) / A.issuers - t_begin;
                for (int q = 0; q < Q; ++q) {
                    // Only the operand rows e in [elo, elo + n) of block q reach surface rows.
                    int elo, n;
                    if (!block_rows(q, A.NB, nr, &elo, &n)) continue;
                    const uint32_t idesc = tc::idesc_u8_s32(64, n);
                    uint32_t a_lo = static_cast<uint32_t>(da0) +
                                    static_cast<uint32_t>(q * A.QS >> 4) + 2u * static_cast<uint32_t>(t_begin);
                    uint32_t b_lo = static_cast<uint32_t>(db0) + static_cast<uint32_t>(elo) +
                                    bstep * static_cast<uint32_t>(t_begin);
                    const uint32_t dn = taddr + static_cast<uint32_t>(stream) * acc1 +
                                        static_cast<uint32_t>(16 * q + elo - (A.NB - 16));
                    for (int t = 0; t < npairs; ++t) {
                        tc::mma_u8_halves(dn, a_lo, a_hi, b_lo, b_hi, idesc);
                        a_lo += 2;
                        b_lo += bstep;
                    }
                }
                tc::mma_commit(&s_mbar);
#ifdef AR_TC_PHASES
                if (stream == 0) atomicAdd(&g_tc_phase[12], clock64() - tmi0);
#endif
            }
            __syncwarp();
        } else {
            // Box sums of W and W^2 (integral_both!, boxsum, src/integral.jl:141-170, 244-247) as
            // exact integers, beside the products: column sums V of ch rows, then sums of cw
            // columns of V, s1 kept as Float32 (exact: below 2^24) and s2. VR surface rows at a
            // time.
            const int kBT = nbox;
            auto bar_box = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(kBT) : "memory"); };
            if (carry) {
                // The held sums belong to the same window geometry `sh` rows higher: only the last
                // `sh` rows are new. Their column sums slide on from the held last row (s_L).
                for (int i0 = iA; i0 < nr; i0 += A.VR) {
                    const int ni = min(A.VR, nr - i0);
                    for (int x = tid; x < XW; x += kBT) {
                        const uint8_t* colx = s_W + x * 16;
                        auto word = [&](int a) {  // rows a .. a + 3, a a multiple of 4
                            const int q = min(a >> 4, Q - 1);
                            return *reinterpret_cast<const uint32_t*>(colx + q * A.QS + (a & 12));
                        };
                        // Row i's sum drops window row i - 1 and takes row i - 1 + ch.
                        const int R0 = i0 - 1, R1 = i0 - 1 + ch;
                        const uint32_t so = static_cast<uint32_t>(R0 & 3) * 8u;
                        const uint32_t sn = static_cast<uint32_t>(R1 & 3) * 8u;
                        int ao = R0 & ~3, an = R1 & ~3;
                        uint32_t lo_o = word(ao), lo_n = word(an);
                        uint32_t h1 = s_L1[x], h2 = s_L2[x];
                        uint32_t* v1 = s_V1 + x;
                        uint32_t* v2 = s_V2 + x;
                        for (int i = 0; i < ni; i += 4) {
                            ao += 4;
                            an += 4;
                            const uint32_t hi_o = word(ao), hi_n = word(an);
                            const uint32_t wo = __funnelshift_r(lo_o, hi_o, so);
                            const uint32_t wn = __funnelshift_r(lo_n, hi_n, sn);
                            lo_o = hi_o;
                            lo_n = hi_n;
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                if (i + u < ni) {
                                    const uint32_t bo = (wo >> (8 * u)) & 255u, bn = (wn >> (8 * u)) & 255u;
                                    h1 += bn - bo;
                                    h2 += bn * bn - bo * bo;
                                    *v1 = h1;
                                    *v2 = h2;
                                }
                                v1 += A.XV;
                                v2 += A.XV;
                            }
                        }
                        s_L1[x] = h1;
                        s_L2[x] = h2;
                    }
                    bar_box();
                    // Sums of cw columns as differences of prefix sums (exact modulo 2^32), a warp
                    // per row.
                    for (int il = warp; il < ni; il += kBT >> 5) {
                        uint32_t* v1 = s_V1 + il * A.XV;
                        uint32_t* v2 = s_V2 + il * A.XV;
                        uint32_t c1 = 0u, c2_ = 0u;
                        for (int x0 = 0; x0 < XW; x0 += 128) {
                            const int x = x0 + 4 * lane;
                            uint4 a = make_uint4(0, 0, 0, 0), d = a;
                            if (x < XW) {
                                a = *reinterpret_cast<const uint4*>(v1 + x);
                                d = *reinterpret_cast<const uint4*>(v2 + x);
                            }
                            a.y += a.x;
                            a.z += a.y;
                            a.w += a.z;
                            d.y += d.x;
                            d.z += d.y;
                            d.w += d.z;
                            const uint32_t t1 = warp_inclusive_scan(a.w), t2 = warp_inclusive_scan(d.w);
                            const uint32_t p1 = t1 - a.w + c1, p2 = t2 - d.w + c2_;
                            if (x < XW) {
                                *reinterpret_cast<uint4*>(v1 + x) = make_uint4(a.x + p1, a.y + p1, a.z + p1, a.w + p1);
                                *reinterpret_cast<uint4*>(v2 + x) = make_uint4(d.x + p2, d.y + p2, d.z + p2, d.w + p2);
                            }
                            c1 += __shfl_sync(kFull, t1, 31);
                            c2_ += __shfl_sync(kFull, t2, 31);
                        }
                        __syncwarp();
                        const int ri = ring(i0 + il);
                        for (int j = lane; j < nc; j += 32) {
                            const float s1 = __uint2float_rn(v1[j + cw - 1] - (j > 0 ? v1[j - 1] : 0u));
                            const uint32_t s2 = v2[j + cw - 1] - (j > 0 ? v2[j - 1] : 0u);
                            const int o = j * A.NRS + ri;
                            s_S1[o] = s1;
                            s_S2[o] = s2;
                            s_R[o] = recip(s1, s2);
                        }
                    }
                    if (i0 + ni < nr) bar_box();
                }
            } else {
                // V[i][x] = sums over rows i .. i + ch - 1 of column x: a task is a column and the 16
                // rows i of one block; its outgoing rows are that block, its incoming rows start ch
                // rows lower.
                const int chb = ch >> 4, chr = ch & 15;
                for (int is = 0; is < nr; is += A.VR) {
                    const int ni = min(A.VR, nr - is);
                    const int nseg = (ni + 15) >> 4;
                    for (int task = tid; task < XW * nseg; task += kBT) {
                        const int sgl = task / XW, x = task - sgl * XW;
                        const int sgi = (is >> 4) + sgl, i0 = 16 * sgi;
                        const uint8_t* colx = s_W + x * 16;
                        const uint4 bo = *reinterpret_cast<const uint4*>(colx + sgi * A.QS);
                        uint32_t h1 = 0, h2 = 0;
                        for (int bb = 0; bb < chb; ++bb) {
                            const uint4 w = *reinterpret_cast<const uint4*>(colx + (sgi + bb) * A.QS);
                            h1 = __dp4a(w.x, 0x01010101u, h1);
                            h1 = __dp4a(w.y, 0x01010101u, h1);
                            h1 = __dp4a(w.z, 0x01010101u, h1);
                            h1 = __dp4a(w.w, 0x01010101u, h1);
                            h2 = __dp4a(w.x, w.x, h2);
                            h2 = __dp4a(w.y, w.y, h2);
                            h2 = __dp4a(w.z, w.z, h2);
                            h2 = __dp4a(w.w, w.w, h2);
                        }
                        const uint4 bi = *reinterpret_cast<const uint4*>(colx + (sgi + chb) * A.QS);
                        if (chr) {
                            const uint32_t wv[4] = {bi.x, bi.y, bi.z, bi.w};
#pragma unroll
                            for (int m = 0; m < 4; ++m) {
                                const int keep = min(max(chr - 4 * m, 0), 4);
                                const uint32_t mk = keep == 4 ? 0xffffffffu : ((1u << (8 * keep)) - 1u);
                                h1 = __dp4a(wv[m] & mk, 0x01010101u, h1);
                                h2 = __dp4a(wv[m] & mk, wv[m], h2);
                            }
                        }
                        const uint32_t wo[4] = {bo.x, bo.y, bo.z, bo.w};
                        const uint32_t wi[4] = {bi.x, bi.y, bi.z, bi.w};
                        uint32_t* v1o = s_V1 + 16 * sgl * A.XV + x;
                        uint32_t* v2o = s_V2 + 16 * sgl * A.XV + x;
#pragma unroll
                        for (int u = 0; u < 16; ++u) {
                            if (i0 + u < nr) {
                                v1o[u * A.XV] = h1;
                                v2o[u * A.XV] = h2;
                                if (i0 + u + 1 == nr) {
                                    s_L1[x] = h1;
                                    s_L2[x] = h2;
                                }
                                const uint32_t o = (wo[u >> 2] >> (8 * (u & 3))) & 0xffu;
                                uint32_t in;
                                if (chr == 0) {
                                    in = (wi[u >> 2] >> (8 * (u & 3))) & 0xffu;
                                } else {
                                    const int R = i0 + u + ch;
                                    in = colx[(R >> 4) * A.QS + (R & 15)];
                                }
                                h1 = h1 + in - o;
                                h2 = h2 + in * in - o * o;
                            }
                        }
                    }
                    bar_box();
                    // S[j][i] = sums of V[i][j .. j + cw - 1]: a task is a row i and 16 columns j.
                    const int jseg = (nc + 15) >> 4;
                    const bool vec = (cw & 3) == 0;
                    for (int task = tid; task < ni * jseg; task += kBT) {
                        const int sg = task / ni, il = task - sg * ni, i = is + il;
                        const int j0 = 16 * sg;
                        const uint32_t* r1 = s_V1 + il * A.XV;
                        const uint32_t* r2 = s_V2 + il * A.XV;
                        uint32_t g1 = 0, g2 = 0;
                        int bb = 0;
                        for (; bb + 4 <= cw; bb += 4) {
                            const uint4 v = *reinterpret_cast<const uint4*>(r1 + j0 + bb);
                            const uint4 w = *reinterpret_cast<const uint4*>(r2 + j0 + bb);
                            g1 += (v.x + v.y) + (v.z + v.w);
                            g2 += (w.x + w.y) + (w.z + w.w);
                        }
                        for (; bb < cw; ++bb) {
                            g1 += r1[j0 + bb];
                            g2 += r2[j0 + bb];
                        }
#pragma unroll
                        for (int u4 = 0; u4 < 16; u4 += 4) {
                            const uint4 o1 = *reinterpret_cast<const uint4*>(r1 + j0 + u4);
                            const uint4 o2 = *reinterpret_cast<const uint4*>(r2 + j0 + u4);
                            uint4 i1, i2;
                            if (vec) {
                                i1 = *reinterpret_cast<const uint4*>(r1 + j0 + u4 + cw);
                                i2 = *reinterpret_cast<const uint4*>(r2 + j0 + u4 + cw);
                            } else {
                                const uint32_t* p1 = r1 + j0 + u4 + cw;
                                const uint32_t* p2 = r2 + j0 + u4 + cw;
                                i1 = make_uint4(p1[0], p1[1], p1[2], p1[3]);
                                i2 = make_uint4(p2[0], p2[1], p2[2], p2[3]);
                            }
                            const uint32_t oo1[4] = {o1.x, o1.y, o1.z, o1.w}, ii1[4] = {i1.x, i1.y, i1.z, i1.w};
                            const uint32_t oo2[4] = {o2.x, o2.y, o2.z, o2.w}, ii2[4] = {i2.x, i2.y, i2.z, i2.w};
#pragma unroll
                            for (int m = 0; m < 4; ++m) {
                                const int j = j0 + u4 + m;
                                if (j < nc) {
                                    s_S1[j * A.NRS + i] = __uint2float_rn(g1);
                                    s_S2[j * A.NRS + i] = g2;
                                    g1 = g1 + ii1[m] - oo1[m];
                                    g2 = g2 + ii2[m] - oo2[m];
                                }
                            }
                        }
                    }
                    if (is + ni < nr) bar_box();
                }
            }
        }
        held = true;
        TC_PHASE(4)
        // One warp polls for the products, the others wait for it at the barrier. It first makes the
        // bound of the estimates' error (below).
        bool ok = true;
        if (warp == 7) {
            const float u24 = 6.0200e-08f;  // 1.01 x 2^-24
            const float kz = sqrtf(pow2 ? __ull2float_rn(nsq) : static_cast<float>(out.sq) * nnf);
            const float kc = sqrtf(nnf * (pow2 ? __uint2float_rn(c2)
                                               : static_cast<float>(out.sq + out.csum * out.mean)));
            if (lane == 0)
                s_bu = A.measure == AR_NCC ? u24 * sqrtf(nnf) * (20.0f * kz + 5.0f * kc)
                                           : u24 * (3400.0f * kz + 160.0f * kc);
            ok = tc::mbar_wait(&s_mbar, phase, kTcWaitPolls);
        }
        phase ^= 1u;
        if (bar_main_or(!ok)) {
            failed = true;
            mb ^= 1;  // this point's barrier with the patch warp is past
            break;
        }
        tc::fence_after_sync();
        if (tid == 0) tc::mbar_arrive(&s_free);
        TC_PHASE(5)

        // Pass 1: numerators out of Tensor Memory (one 16x256b read per warp and accumulator), box
        // sums from shared memory. Value v of a thread is surface row
        // i = 32 half + 8 (v / 4) + 2 (lane % 4) + v % 2, column j = 16 quarter + lane / 4 (+ 8
        // when v % 4 >= 2).
        // The estimate of a value is nx r, with nx = nn D - sum(C) s1 and r the reciprocal root of
        // its variance term vx = nn s2 - s1^2 (s2 for NCC), all in Float32: the value times
        // kz = cnorm sqrt(nn) (NCC: cnorm nn). r depends on the window alone, so it is kept in a
        // ring beside s1 and s2 and made for new rows only; it is 0 where s2 is 0 (the value is
        // 0) and NaN where tv = nn s2 + s1^2 is above 2^11 vx, whose value is always evaluated
        // exactly. Errors (u = 2^-24): vx is within 3u tv of exact, so r is within 3080u of exact;
        // D, sum(C) s1, nx and the product round once each. So an estimate is within
        // 3100u |value| + 1.05u (nn D + sum(C) s1) r / kz of the value, and by Cauchy-Schwarz the
        // second term is at most 2.1u T_c T with T_c = |C| / cnorm and T = sqrt(nn s2 / vx) <= 32 (1
        // for NCC). `bu` is (3400u + 5u T_c T) kz, above that (with kc = sqrt(nn sum(C^2))): a value
        // whose estimate is more than 2 bu below the largest one is below that one.
        const float csf = pow2 ? __uint2float_rn(cs) : static_cast<float>(out.csum);
        const int quarter = warp & 3, half = warp >> 2;
        const int ib0 = 32 * half + 2 * (lane & 3);
        const int jb0 = 16 * quarter + (lane >> 2);
        uint32_t dv[16];
        float sum = 0.0f;
        float own = -INFINITY, own2 = -INFINITY;  // this thread's two largest estimates
        int at = 0;                               // the value of the largest
        bool odd = false;                         // an estimate was not made
        if (32 * half < nr && 16 * quarter < nc) {
            const uint32_t base = taddr + (static_cast<uint32_t>(32 * quarter) << 16) +
                                  static_cast<uint32_t>(32 * half);
            {
                // The issuers' shares.
                uint32_t d1[16];
                tc::tmem_ld16dp(base, dv);
                tc::tmem_ld16dp(base + acc1, d1);
                tc::tmem_wait_ld();
#pragma unroll
                for (int v = 0; v < 16; ++v) dv[v] += d1[v];
                for (int s = 2; s < A.issuers; ++s) {
                    tc::tmem_ld16dp(base + static_cast<uint32_t>(s) * acc1, d1);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int v = 0; v < 16; ++v) dv[v] += d1[v];
                }
            }
            clear_acc();  // for the next point (waited for before its products)
            // Values v and v + 1 are surface rows i and i + 1 of one column (nr is even): estimated
            // as a packed pair, from clamped indices so that all loads can be in flight.
            int r0[4], r1[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                r0[m] = ring(min(ib0 + 8 * m, nr - 2));
                r1[m] = r0[m] + 1 == A.NRS ? 0 : r0[m] + 1;
            }
            auto pair = [&](int m, int c, float2 s1, float2 r) {
                const int v = 4 * m + 2 * c;
                const float2 nx = __ffma2_rn(
                    make_float2(nnf, nnf),
                    make_float2(__uint2float_rn(dv[v]), __uint2float_rn(dv[v + 1])),
                    neg2(__fmul2_rn(make_float2(csf, csf), s1)));
                float2 e = __fmul2_rn(nx, r);
                const bool in = jb0 + 8 * c < nc && ib0 + 8 * m < nr;
                sum += in ? e.x + e.y : 0.0f;
                e.x = in ? e.x : -INFINITY;
                e.y = in ? e.y : -INFINITY;
                own2 = fmaxf(own2, fminf(own, e.x));
                at = e.x > own ? v : at;
                own = fmaxf(own, e.x);
                own2 = fmaxf(own2, fminf(own, e.y));
                at = e.y > own ? v + 1 : at;
                own = fmaxf(own, e.y);
            };
            if (carry) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float* S = s_S1 + min(jb0 + 8 * c, nc - 1) * A.NRS;
                    const float* R = s_R + min(jb0 + 8 * c, nc - 1) * A.NRS;
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        pair(m, c, make_float2(S[r0[m]], S[r1[m]]), make_float2(R[r0[m]], R[r1[m]]));
                }
            } else {
                // Every row is new: the reciprocal roots are made here, by all warps.
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int o = min(jb0 + 8 * c, nc - 1) * A.NRS;
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        const float2 s1 = make_float2(s_S1[o + r0[m]], s_S1[o + r1[m]]);
                        const float2 r = make_float2(recip(s1.x, s_S2[o + r0[m]]), recip(s1.y, s_S2[o + r1[m]]));
                        s_R[o + r0[m]] = r.x;
                        s_R[o + r1[m]] = r.y;
                        pair(m, c, s1, r);
                    }
                }
            }
            odd = isnan(sum);
        } else {
            clear_acc();
#pragma unroll
            for (int v = 0; v < 16; ++v) dv[v] = 0u;
        }
        // The warp's largest estimate, where it is, and the largest of its others (+inf when some
        // estimate was not made).
        {
            const float top = warp_max(own);
            const unsigned who = __ballot_sync(kFull, own == top && own > -INFINITY);
            const int first = who ? __ffs(who) - 1 : 0;
            const float sec = warp_max(odd ? INFINITY : lane == first ? own2 : own);
            if (lane == first) {
                s_top[warp] = top;
                s_sec[warp] = sec;
                s_at[warp] = ((ib0 + 8 * (at >> 2) + (at & 1)) << 16) | (jb0 + ((at & 2) ? 8 : 0));
            }
        }
        tc::fence_before_sync();
        bar_main();  // also: the accumulators are read
        tc::fence_after_sync();
        TC_PHASE(6)
        // Lane w looks at warp w's: is the largest estimate more than the bound above every other?
        int pi = 0, pj = 0;
        const float wt = lane < 8 ? s_top[lane] : -INFINITY;
        const float M = warp_max(wt);
        const float cut = M - 2.0f * s_bu;
        const int mw = __ffs(__ballot_sync(kFull, wt == M)) - 1;
        const bool unique =
            M > -INFINITY &&
            !__any_sync(kFull, lane < 8 && (!(s_sec[lane & 7] < cut) || (lane != mw && !(wt < cut))));
        if (unique && !A.surf_out) {
            // Every other value is below this one: it is the strict (so the first) maximum.
            pi = s_at[mw] >> 16;
            pj = s_at[mw] & 0xFFFF;
        } else {
            // Pass 2: the values whose estimate is within the bounds of M (or was not made), exactly,
            // from the numerators in shared memory (in place of the operands).
            const double nn = static_cast<double>(nnl);
            double mean = out.mean, sq = out.sq;
            if (pow2) tc2_chip_stats(nnl, cs, c2, &mean, &sq);
            const double cnorm = __dsqrt_rn(sq);
#pragma unroll
            for (int v = 0; v < 16; ++v) {
                const int i = ib0 + 8 * (v >> 2) + (v & 1), j = jb0 + ((v & 2) ? 8 : 0);
                if (i < nr && j < nc) s_num[j * A.NRS + i] = dv[v];
            }
            bar_main();
            unsigned long long best = 0ull;
            for (int e = tid; e < nr * nc; e += kTcThreads) {
                const int j = e / nr, i = e - j * nr;
                const int o = j * A.NRS + ring(i);
                const uint32_t D = s_num[j * A.NRS + i], s2 = s_S2[o];
                const float s1 = s_S1[o];
                if (__fmaf_rn(nnf, __uint2float_rn(D), -__fmul_rn(csf, s1)) * s_R[o] < cut && !A.surf_out) continue;
                const float x = tc2_exact(D, s1, s2, mean, nn, cnorm, A.measure);
                const unsigned long long key = argmax_key(x, static_cast<unsigned>(i * nc + j));
                best = key > best ? key : best;
                if (A.surf_out) A.surf_out[k * static_cast<int64_t>(A.NRM) * A.NCM + e] = x;
            }
            best = block_max_u64<true>(best, reinterpret_cast<unsigned long long*>(s_red));
            unsigned rm = 0;
            float pv = 0.0f;
            if (key_decode(best, &rm, &pv)) {
                pi = static_cast<int>(rm / nc);
                pj = static_cast<int>(rm % nc);
            }
            bar_main();  // s_num and s_red are read
        }
        TC_PHASE(7)
        if (A.flops && tid == 0)
            atomicAdd(A.flops, 2ull * static_cast<unsigned long long>(nnl) * nr * nc);
        // The peak's or the patch's numerators and sums, to the helper.
        const bool single = A.up == 1 || nr < 5 || nc < 5;
        const int pi0 = single ? pi : min(max(pi - 2, 0), max(nr - 5, 0));
        const int pj0 = single ? pj : min(max(pj - 2, 0), max(nc - 5, 0));
        const int span = single ? 1 : 5;
        if (pi0 < 32 * half + 32 && pi0 + span > 32 * half && pj0 < 16 * quarter + 16 &&
            pj0 + span > 16 * quarter) {
#pragma unroll
            for (int v = 0; v < 16; ++v) {
                const int i = ib0 + 8 * (v >> 2) + (v & 1), j = jb0 + ((v & 2) ? 8 : 0);
                const unsigned a = static_cast<unsigned>(i - pi0), c = static_cast<unsigned>(j - pj0);
                if (a < static_cast<unsigned>(span) && c < static_cast<unsigned>(span)) {  // inside the surface
                    const int o = j * A.NRS + ring(i);
                    out.D[c * 5 + a] = dv[v];
                    out.s1[c * 5 + a] = s_S1[o];
                    out.s2[c * 5 + a] = s_S2[o];
                }
            }
        }
        if (tid == 0) {
            out.kind = single ? 1 : 2;
            out.pi = pi0;
            out.pj = pj0;
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&s_outb[mb]);
        mb ^= 1;
        TC_PHASE(8)
        TC_PHASE_POINT
    }
    TC_PHASE_FLUSH
    if (failed) {
        if (tid == 0) atomicExch(A.status, 1);
        // Products may still be in flight: a bounded time before the accumulators are freed.
        tc::mbar_wait(&s_mbar, phase ^ 1u, kTcWaitPolls);
    }
    tc::tmem_wait_st();
    if (tid == 0) s_more[mb] = 0;
    bar_products();
    }
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0 && s_lost) atomicExch(A.status, 1);
    if (warp == 0) tc::tmem_dealloc(taddr, A.tmem_cols);
}

// ----------------------------------------------------------------------------------------------
// Split-BF16 tensor-core correlation for UInt16, Int16 and Float32 imagery (k_corr_bf).
//
// The numerator of the CUDA-core kernel, sum_{a,b} C'[a, b] W'[i + a, j + b], with C' the chip of
// prepare_chip! (src/correlate.jl:423-453: Float32(x - mean)) and W' the window shifted by a
// centring constant (W' = Float32(w - cshift), cshift the chip mean rounded to an integer for
// integer imagery and to Float32 otherwise; num = sum C' W' + cshift sum C'), as products on the
// tensor cores (tcgen05.mma kind::f16, BF16 operands, FP32 accumulators in Tensor Memory). Each
// operand is split into three BF16 limbs, v = v0 + v1 + v2 with v0 = bf16(v), v1 = bf16(v - v0),
// v2 = bf16(v - v0 - v1) (24 significant bits: a Float32 value exactly), and the numerator is the
// sum of the six products whose order is at least 2^-16 -- c0 w0, c0 w1, c1 w0, c1 w1, c2 w0,
// c0 w2 -- which recovers FP32 accuracy. The integer windows of UInt16 and Int16 imagery are
// exactly w0 + w1 (an integer below 2^16 in magnitude is the sum of two BF16 values), so their
// c0 w2 product is skipped.
//
// Layout (as the UInt8 kernels, with 2-byte elements and one chip column per product):
//   A[j, (q, b, r)] = W'[16 q + r, j + b]    r < 16, stored as two 8-row halves h:
//                                            s_W[limb][q][h][x] (16 bytes), row j of A 16 bytes
//                                            after row j - 1, the halves LW x 16 bytes apart;
//   B[i, (q, b, r)] = E_b[i - 16 q][r]       E_b[u][r] = C'[r - u, b], stored s_E[limb][b][h][e].
// Block q meets surface rows [16 q - ch + 1, 16 q + 15]: NB = 16 ceil((ch + 15) / 16) operand rows,
// surface row i in accumulator column i (rows trimmed to 0 <= i < nr in steps of 16).
//
// Per point: the chip's statistics; the window's box sums (integral_both!, boxsum,
// src/integral.jl:141-170, 244-247) in FP64 from the image values, a stripe of window columns
// at a time in shared memory -- column sums of ch rows, then a running sum along each surface
// row whose differences cw columns apart are the box sums -- and from them each surface value's
// FP64 denominator (src/correlate.jl:575-630); then the window's limbs for as many chip columns
// as shared memory holds (all of them up to 64-px chips), and the products chunk by chunk of BC
// chip columns. Four threads issue a chunk's products, each into an accumulator of its own (one
// thread issues an MMA about every 120 cycles, so the small M = 64 products need several issuers
// to keep the tensor core busy). Two sets of four accumulators take alternate chunks: while the
// tensor core runs chunk c, the threads build chunk c + 1's chip operand and add chunk c - 1's
// accumulators into FP64 sums they keep in registers (the tensor core's FP32 accumulation does
// not round to nearest, so a long chain of products into one accumulator drifts: ~1e-4 of the
// numerator over the ~1,000 products per accumulator of a 192-px chip; a chunk's chain is kept
// near kBfChain). Surfaces up to 64 x 64.

constexpr int kBfThreads = 256;
constexpr int kBfLimbs = 3;        // BF16 limbs per operand
constexpr int kBfPadL = 16;        // zero elements before each staged chip column
constexpr int kBfChain = 24;       // accumulating products per accumulator element per chunk
constexpr int kBfIssuers = 4;      // issuing threads (and accumulators) per set
constexpr int kBfPre = 4;          // staged chip elements per thread and chunk
constexpr int kBfBatch = 8;        // global loads a thread issues before using them

struct BfArgs {
    const void* ref;
    const void* sec;
    const uint8_t* valid;
    int64_t nrows, ncols;
    DevPoints pts;
    int64_t padx, pady;
    int up, measure;
    int CHM, CWM, NRM, NCM;
    int NB;                          // chip operand rows per column (multiple of 16)
    int BC;                          // chip columns per chunk
    int OB;                          // chip columns per window staging (multiple of BC)
    int LW;                          // window columns staged (OB + 63)
    int PC;                          // staged chip column length (elements, even)
    int NRS;                         // surface, box-sum and denominator row stride
    int AC;                          // columns per accumulator (multiple of 16)
    int RS;                          // row stride of a box-sum stripe's window columns (odd)
    int VS;                          // row stride of a stripe's column sums (nr + 1)
    int XS;                          // window columns per box-sum stripe
    unsigned off_S2, off_raw, off_V; // box-sum phase (S1 at 0)
    unsigned off_den, off_E, off_P, off_red;
    unsigned Eb, Pb;                 // bytes per chip-operand / staged-chip buffer
    uint32_t tmem_cols;
    DevOutputs out;
    int* sub_count;
    int64_t* sub_point;
    int32_t* sub_origin;
    float* sub_patch;
    float* surf_out;
    unsigned long long* flops;
    int* status;
};

// The three BF16 limbs of v, as raw 16-bit patterns: l[0] = bf16(v), l[1] = bf16(v - l[0]),
// l[2] = bf16(v - l[0] - l[1]). Each difference is exact in FP32 (its operands are within a
// factor of two of each other), and the last remainder has at most 8 significant bits, so
// v = l[0] + l[1] + l[2] for every normal v.
__device__ __forceinline__ void bf16_split3(float v, uint32_t (&l)[kBfLimbs]) {
    float r = v;
#pragma unroll
    for (int t = 0; t < kBfLimbs; ++t) {
        const __nv_bfloat16 h = __float2bfloat16_rn(r);
        l[t] = static_cast<uint32_t>(__bfloat16_as_ushort(h));
        r = __fsub_rn(r, __bfloat162float(h));
    }
}

template <typename T>
__global__ void __launch_bounds__(kBfThreads, 1) k_corr_bf(const BfArgs A) {
    typedef Traits<T> Tr;
    extern __shared__ __align__(1024) unsigned char smem_bf[];
    __shared__ uint64_t s_mbar[2];
    __shared__ uint32_t s_taddr;
    const int tid = threadIdx.x, bd = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5;
    const T* ref = static_cast<const T*>(A.ref);
    const T* sec = static_cast<const T*>(A.sec);
    // Window limbs [limb][q][h][x] (16 bytes each) from offset 0, where the box-sum phase keeps
    // S1 and S2 [j][NRS] (FP64) and the epilogue the surface; the stripe buffers of the box sums
    // reach into the region of the denominators [j][NRS] (FP64), the two chip-operand buffers
    // [limb][b][h][e] and the two staged-chip buffers [limb][b][PC] (raw BF16 bits).
    unsigned char* s_W = smem_bf;
    double* s_S1 = reinterpret_cast<double*>(smem_bf);
    double* s_S2 = reinterpret_cast<double*>(smem_bf + A.off_S2);
    float* s_raw = reinterpret_cast<float*>(smem_bf + A.off_raw);
    double* s_V = reinterpret_cast<double*>(smem_bf + A.off_V);
    double* s_den = reinterpret_cast<double*>(smem_bf + A.off_den);
    unsigned char* s_E = smem_bf + A.off_E;
    unsigned char* s_Pb = smem_bf + A.off_P;
    double* s_red = reinterpret_cast<double*>(smem_bf + A.off_red);
    float* s_surf = reinterpret_cast<float*>(smem_bf);
    const size_t wlimb = static_cast<size_t>((A.CHM + A.NRM - 1 + 15) / 16) * 2 * A.LW * 16;
    const size_t elimb = static_cast<size_t>(A.BC) * 2 * A.NB * 16;
    const int plimb = A.BC * A.PC;
    const int64_t NR = A.nrows + 2 * A.pady, NC = A.ncols + 2 * A.padx;
    const double shx = static_cast<double>(A.padx) + 0.5;
    const double shy = static_cast<double>(A.pady) + 0.5;

    if (warp == 0) {
        tc::tmem_alloc(&s_taddr, A.tmem_cols);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        tc::mbar_init(&s_mbar[0], kBfIssuers);  // one commit per issuer and chunk
        tc::mbar_init(&s_mbar[1], kBfIssuers);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t taddr = s_taddr;
    uint32_t ph[2] = {0u, 0u};
    bool pend[2] = {false, false};
    bool failed = false;
    TC_PHASE_INIT

    // Accumulator values of a thread after a chunk: value v is surface row
    // i = 32 half + 8 (v / 4) + 2 (lane % 4) + v % 2, column j = 16 quarter + lane / 4 (+ 8 when
    // v % 4 >= 2) -- the 16x256b read pattern of its lane quarter's half.
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t qbase = taddr + (static_cast<uint32_t>(32 * quarter) << 16) +
                           static_cast<uint32_t>(32 * half);
    // Zeros into this warp's lane quarter and half of the columns of set s's accumulators
    // (columns [32 half, 32 half + 32) of each, as far as the accumulator reaches): the warps
    // of the two halves together clear the set, each after reading its own values.
    auto clear_half = [&](int s) {
        uint32_t z[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) z[t] = 0u;
        const int c1 = min(32 * (half + 1), A.AC);
        for (int t = 0; t < kBfIssuers; ++t) {
            const uint32_t a0 = qbase - static_cast<uint32_t>(32 * half) +
                                static_cast<uint32_t>((kBfIssuers * s + t) * A.AC);
            for (int c = 32 * half; c < c1; c += 16) tc::tmem_st16(a0 + static_cast<uint32_t>(c), z);
        }
        tc::tmem_wait_st();
    };
    // Bounded wait for set s's products; on success the set is no longer pending.
    auto wait_set = [&](int s) -> bool {
        const bool ok = tc::mbar_wait(&s_mbar[s], ph[s], kTcWaitPolls);
        if (ok) {
            ph[s] ^= 1u;
            pend[s] = false;
        }
        return ok;
    };

    for (int64_t k = blockIdx.x; k < A.pts.n && !failed; k += gridDim.x) {
        tc::fence_before_sync();
        __syncthreads();  // the previous point's buffers and accumulators are no longer read
        tc::fence_after_sync();
        TC_PHASE(0)
        const int64_t prx = A.pts.rx[k], pry = A.pts.ry[k];
        if (!(prx > 0 && pry > 0)) continue;
        const double xs = A.pts.x[k] + shx, ys = A.pts.y[k] + shy;
        const int64_t hx = A.pts.csx[k] / 2, hy = A.pts.csy[k] / 2;
        const int64_t ccx = static_cast<int64_t>(floor(__dsub_rn(xs, A.pts.dx0[k])));
        const int64_t ccy = static_cast<int64_t>(floor(__dsub_rn(ys, A.pts.dy0[k])));
        const int64_t wcx = static_cast<int64_t>(floor(xs)), wcy = static_cast<int64_t>(floor(ys));
        const int64_t cr0 = ccy - hy, cr1 = ccy + hy - 1, cc0 = ccx - hx, cc1 = ccx + hx - 1;
        const int64_t wr0 = wcy - hy - pry, wr1 = wcy + hy + pry - 2;
        const int64_t wc0 = wcx - hx - prx, wc1 = wcx + hx + prx - 2;
        const bool chip_in = (cr1 < cr0 || cc1 < cc0) ||
                             (cr0 >= 1 && cr1 <= NR && cc0 >= 1 && cc1 <= NC);
        const bool win_in = (wr1 < wr0 || wc1 < wc0) ||
                            (wr0 >= 1 && wr1 <= NR && wc0 >= 1 && wc1 <= NC);
        if (!chip_in || !win_in) continue;
        const int ch = static_cast<int>(2 * hy), cw = static_cast<int>(2 * hx);
        const int nr = static_cast<int>(2 * pry), nc = static_cast<int>(2 * prx);
        if (ch <= 0 || cw <= 0) continue;
        if (ch > A.CHM || cw > A.CWM || nr > A.NRM || nc > A.NCM || nr > 64 || nc > 64) continue;
        const int64_t chip_r = cr0 - 1 - A.pady, chip_c = cc0 - 1 - A.padx;
        const int64_t win_r = wr0 - 1 - A.pady, win_c = wc0 - 1 - A.padx;
        const int nn_i = ch * cw;

        // _any_valid over the chip (src/track.jl:416-421).
        int any = 0;
        for (int e0 = tid; e0 < nn_i && !any; e0 += kBfBatch * bd) {
            uint8_t v[kBfBatch];
#pragma unroll
            for (int u = 0; u < kBfBatch; ++u) {
                const int e = e0 + u * bd;
                const int64_t r = chip_r + e % ch, c = chip_c + e / ch;
                v[u] = (e < nn_i && r >= 0 && r < A.nrows && c >= 0 && c < A.ncols)
                           ? A.valid[r + c * A.nrows] : static_cast<uint8_t>(0);
            }
#pragma unroll
            for (int u = 0; u < kBfBatch; ++u) any |= v[u] ? 1 : 0;
        }
        if (!__syncthreads_or(any)) continue;
        if (tid == 0) A.out.searched[k] = 1;
        TC_PHASE(1)

        // prepare_chip! as the CUDA-core kernel (the same per-thread order): FP64 mean, FP64 sum
        // of squares of the deviations, FP64 sum of the Float32-rounded deviations.
        double st[1] = {0.0};
        for (int e0 = tid; e0 < nn_i; e0 += kBfBatch * bd) {
            double v[kBfBatch];
#pragma unroll
            for (int u = 0; u < kBfBatch; ++u) {
                const int e = e0 + u * bd;
                v[u] = e < nn_i ? pixel(sec, A.nrows, A.ncols, chip_r + e % ch, chip_c + e / ch) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kBfBatch; ++u)
                if (e0 + u * bd < nn_i) st[0] = __dadd_rn(st[0], v[u]);
        }
        block_sum_f64<1>(st, s_red);
        const double nn = static_cast<double>(nn_i);
        const double mean = __ddiv_rn(st[0], nn);
        const int chp = (ch + kUA - 1) & ~(kUA - 1);
        double acc2[2] = {0.0, 0.0};
        for (int e0 = tid; e0 < chp * cw; e0 += kBfBatch * bd) {
            double v[kBfBatch];
#pragma unroll
            for (int u = 0; u < kBfBatch; ++u) {
                const int e = e0 + u * bd, a = e % chp, b = e / chp;
                v[u] = (e < chp * cw && a < ch) ? pixel(sec, A.nrows, A.ncols, chip_r + a, chip_c + b) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kBfBatch; ++u) {
                const int e = e0 + u * bd;
                if (e < chp * cw && e % chp < ch) {
                    const double d = __dsub_rn(v[u], mean);
                    acc2[0] = __dadd_rn(acc2[0], __dmul_rn(d, d));
                    acc2[1] = __dadd_rn(acc2[1], static_cast<double>(__double2float_rn(d)));
                }
            }
        }
        block_sum_f64<2>(acc2, s_red);
        const double sq = acc2[0], sumd = acc2[1];
        if (!(sq > __dmul_rn(__dmul_rn(DBL_EPSILON, static_cast<double>(ch)), static_cast<double>(cw))))
            continue;  // degenerate chip: searched, no measurement (src/track.jl:286)
        const double cnorm = __dsqrt_rn(sq);
        const double cshift = Tr::integer ? rint(mean) : static_cast<double>(__double2float_rn(mean));
        const float csf = static_cast<float>(cshift);
        TC_PHASE(2)

        // Box sums in FP64, a stripe of window columns at a time: the stripe's image values
        // (exact in FP32 for every element type), its column sums V(i, x) of ch rows, then the
        // running sum Q along each surface row i (a thread per row and sum): the box sum at column
        // j is Q after window column j + cw - 1 less Q before column j.
        const int RW = ch + nr - 1, XW = cw + nc - 1;
        double qrun = 0.0;
        for (int x0 = 0; x0 < XW; x0 += A.XS) {
            const int xn = min(A.XS, XW - x0);
            for (int e0 = tid; e0 < xn * RW; e0 += kBfBatch * bd) {
                double v[kBfBatch];
#pragma unroll
                for (int u = 0; u < kBfBatch; ++u) {
                    const int e = e0 + u * bd;
                    v[u] = e < xn * RW ? pixel(ref, A.nrows, A.ncols, win_r + e % RW, win_c + x0 + e / RW) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < kBfBatch; ++u) {
                    const int e = e0 + u * bd;
                    if (e < xn * RW) s_raw[(e / RW) * A.RS + e % RW] = static_cast<float>(v[u]);
                }
            }
            __syncthreads();
            TC_PHASE(3)
            {
                const int segs = max(1, min(nr, bd / xn));
                const int len = (nr + segs - 1) / segs;
                for (int t = tid; t < xn * segs; t += bd) {
                    const int x = t % xn, i0 = (t / xn) * len, i1 = min(nr, i0 + len);
                    if (i0 >= i1) continue;
                    const float* col = s_raw + x * A.RS;
                    double h1 = 0.0, h2 = 0.0;
                    int nz = 0;  // Float32: values other than zero
                    for (int a = i0; a < i0 + ch; ++a) {
                        const double w = static_cast<double>(col[a]);
                        h1 = __dadd_rn(h1, w);
                        h2 = __dadd_rn(h2, __dmul_rn(w, w));
                        if (!Tr::integer) nz += w != 0.0;
                    }
                    for (int i = i0; i < i1; ++i) {
                        // A column of zeros sums to zero, which sliding sums of Float32 values may miss
                        // by a rounding; the running sum along the row then stays as it is.
                        if (!Tr::integer && nz == 0 && h2 == h2) h1 = h2 = 0.0;
                        s_V[2 * (x * A.VS + i)] = h1;
                        s_V[2 * (x * A.VS + i) + 1] = h2;
                        if (i + 1 < i1) {
                            const double wo = static_cast<double>(col[i]);
                            const double wn = static_cast<double>(col[i + ch]);
                            h1 = __dadd_rn(__dsub_rn(h1, wo), wn);
                            h2 = __dadd_rn(__dsub_rn(h2, __dmul_rn(wo, wo)), __dmul_rn(wn, wn));
                            if (!Tr::integer) nz += (wn != 0.0) - (wo != 0.0);
                        }
                    }
                }
            }
            __syncthreads();
            TC_PHASE(4)
            if (tid < 2 * nr) {
                const int i = tid >> 1, comp = tid & 1;
                double* S = comp ? s_S2 : s_S1;
                for (int x = 0; x < xn; ++x) {
                    const int xg = x0 + x;
                    if (xg < nc) S[xg * A.NRS + i] = qrun;
                    qrun = __dadd_rn(qrun, s_V[2 * (x * A.VS + i) + comp]);
                    const int j = xg - cw + 1;
                    if (j >= 0 && j < nc) S[j * A.NRS + i] = __dsub_rn(qrun, S[j * A.NRS + i]);
                }
            }
            __syncthreads();
            TC_PHASE(5)
        }
        TC_PHASE(5)
        // FP64 denominators (src/correlate.jl:591-600, 624-628).
        for (int e = tid; e < nr * nc; e += bd) {
            const int i = e % nr, j = e / nr;
            const double s1 = s_S1[j * A.NRS + i], s2 = s_S2[j * A.NRS + i];
            double den;
            if (A.measure == AR_NCC) {
                den = __dmul_rn(cnorm, __dsqrt_rn(s2 > 0.0 ? s2 : 0.0));
            } else {
                double wvar = __dsub_rn(s2, __ddiv_rn(__dmul_rn(s1, s1), nn));
                if (!(wvar > 0.0)) wvar = 0.0;
                den = __dmul_rn(cnorm, __dsqrt_rn(wvar));
            }
            s_den[j * A.NRS + i] = den;
        }
        clear_half(0);
        clear_half(1);
        __syncthreads();  // S1 and S2 read before the window limbs replace them
        TC_PHASE(6)

        double accd[16];
#pragma unroll
        for (int v = 0; v < 16; ++v) accd[v] = 0.0;
        auto flush_set = [&](int s) {
            if (32 * half < nr) {
                uint32_t r[kBfIssuers][16];
#pragma unroll
                for (int t = 0; t < kBfIssuers; ++t)
                    tc::tmem_ld16dp(qbase + static_cast<uint32_t>((kBfIssuers * s + t) * A.AC), r[t]);
                tc::tmem_wait_ld();
#pragma unroll
                for (int v = 0; v < 16; ++v)
#pragma unroll
                    for (int t = 0; t < kBfIssuers; ++t)
                        accd[v] = __dadd_rn(accd[v], static_cast<double>(__uint_as_float(r[t][v])));
            }
        };
        // A chunk's chip columns C'[a, b0 + bl] as BF16 limbs, zero-padded: the loads first
        // (into registers), the conversion after other work.
        auto p_load = [&](int b0, int bcn, double (&pr)[kBfPre], int t0, int nt) {
#pragma unroll
            for (int u = 0; u < kBfPre; ++u) {
                const int e = (tid - t0) + u * nt;
                const int bl = e / A.PC, a = e - bl * A.PC - kBfPadL;
                pr[u] = (e < plimb && bl < bcn && a >= 0 && a < ch)
                            ? pixel(sec, A.nrows, A.ncols, chip_r + a, chip_c + b0 + bl) : 0.0;
            }
        };
        auto p_store = [&](int buf, int bcn, const double (&pr)[kBfPre], int t0, int nt) {
            uint16_t* P = reinterpret_cast<uint16_t*>(s_Pb + buf * A.Pb);
#pragma unroll
            for (int u = 0; u < kBfPre; ++u) {
                const int e = (tid - t0) + u * nt;
                if (e < plimb) {
                    const int bl = e / A.PC, a = e - bl * A.PC - kBfPadL;
                    uint32_t l[kBfLimbs] = {0u, 0u, 0u};
                    if (bl < bcn && a >= 0 && a < ch) bf16_split3(__double2float_rn(__dsub_rn(pr[u], mean)), l);
#pragma unroll
                    for (int limb = 0; limb < kBfLimbs; ++limb) P[limb * plimb + e] = static_cast<uint16_t>(l[limb]);
                }
            }
        };

        const int QBp = (ch + nr - 1 + 15) / 16;
        const int gp = 2 * QBp;  // 8-row groups per window column
        bool ok = true;
        for (int ob0 = 0; ob0 < cw && ok; ob0 += A.OB) {
            const int obn = min(A.OB, cw - ob0);
            const int xneed = obn + nc - 1;
            // Window limbs of columns ob0 .. ob0 + LW - 1 (zero past the columns and rows the
            // valid surface values read): item (x, q, h) = 8 consecutive rows of column x,
            // consecutive threads on consecutive row groups of one column; two items' loads at once.
            const int items = A.LW * gp;
            for (int it0 = tid; it0 < items; it0 += 2 * bd) {
                float wv[2][8];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int it = it0 + u * bd;
                    const int x = it / gp, g = it - x * gp;
                    const int r0 = 8 * g;  // 16 q + 8 h
#pragma unroll
                    for (int t = 0; t < 8; ++t)
                        wv[u][t] = (it < items && x < xneed && r0 + t < RW)
                                       ? static_cast<float>(pixel(ref, A.nrows, A.ncols, win_r + r0 + t, win_c + ob0 + x))
                                       : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int it = it0 + u * bd;
                    if (it < items) {
                        const int x = it / gp, g = it - x * gp;
                        const int r0 = 8 * g;
                        uint32_t lw[kBfLimbs][4] = {};
#pragma unroll
                        for (int t = 0; t < 8; ++t) {
                            uint32_t l[kBfLimbs] = {0u, 0u, 0u};
                            if (x < xneed && r0 + t < RW) bf16_split3(__fsub_rn(wv[u][t], csf), l);
#pragma unroll
                            for (int limb = 0; limb < kBfLimbs; ++limb) lw[limb][t >> 1] |= l[limb] << (16 * (t & 1));
                        }
                        const size_t o = (static_cast<size_t>(g) * A.LW + x) * 16;
#pragma unroll
                        for (int limb = 0; limb < kBfLimbs; ++limb)
                            *reinterpret_cast<uint4*>(s_W + limb * wlimb + o) =
                                make_uint4(lw[limb][0], lw[limb][1], lw[limb][2], lw[limb][3]);
                    }
                }
            }
            // Chip operand rows for the chunk in buffer `buf` (threads [t0, t0 + nt)):
            // E_b[h][e] = 8 elements of the staged column from element kBfPadL + 8 h - e + NB - 16
            // (C'[r - u, b] with u = e - NB + 16, r = 8 h + t).
            auto build_E = [&](int buf, int t0, int nt) {
                const uint16_t* P = reinterpret_cast<const uint16_t*>(s_Pb + buf * A.Pb);
                unsigned char* E = s_E + buf * A.Eb;
                for (int it = tid - t0; it < A.BC * 2 * A.NB; it += nt) {
                    const int bl = it / (2 * A.NB), rem = it - bl * 2 * A.NB;
                    const int h = rem / A.NB, e = rem - h * A.NB;
                    const int src = kBfPadL + 8 * h - e + A.NB - 16;  // element index, >= 1
                    const size_t o = (static_cast<size_t>(bl * 2 + h) * A.NB + e) * 16;
#pragma unroll
                    for (int limb = 0; limb < kBfLimbs; ++limb) {
                        const uint16_t* col = P + limb * plimb + bl * A.PC;
                        const uint32_t* w = reinterpret_cast<const uint32_t*>(col + (src & ~1));
                        const uint32_t sh = (src & 1) ? 16u : 0u;
                        uint4 v;
                        v.x = __funnelshift_r(w[0], w[1], sh);
                        v.y = __funnelshift_r(w[1], w[2], sh);
                        v.z = __funnelshift_r(w[2], w[3], sh);
                        v.w = __funnelshift_r(w[3], w[4], sh);
                        *reinterpret_cast<uint4*>(E + limb * elimb + o) = v;
                    }
                }
            };
            const int nch = (obn + A.BC - 1) / A.BC;
            auto chunk_b0 = [&](int c) { return ob0 + c * A.BC; };
            auto chunk_n = [&](int c) { return min(A.BC, ob0 + obn - chunk_b0(c)); };
            // Chunk 0's chip columns and operand, chunk 1's chip columns, by every thread.
            {
                double pr[kBfPre];
                p_load(chunk_b0(0), chunk_n(0), pr, 0, bd);
                p_store(0, chunk_n(0), pr, 0, bd);
                __syncthreads();
                build_E(0, 0, bd);
                if (nch > 1) {
                    p_load(chunk_b0(1), chunk_n(1), pr, 0, bd);
                    p_store(1, chunk_n(1), pr, 0, bd);
                }
            }
            tc::fence_proxy_async_smem();
            tc::fence_before_sync();
            __syncthreads();  // limbs, chunk 0's operand and chunk 1's chip columns complete
            TC_PHASE(7)

            // Chunk c: lane 0 of warps 0-3 issue its products into set c & 1 while warps 4-7 take
            // chunk c - 1's values out of set c & 1 ^ 1 (their half of the columns), build chunk
            // c + 1's operand into the buffer chunk c - 1 used and stage chunk c + 2's chip
            // columns; warps 0-3 then take their half of chunk c - 1's values. One barrier per
            // chunk: set c & 1 ^ 1 is clear and chunk c + 1's operand complete after it.
            for (int c = 0; c < nch && ok; ++c) {
                const int s = c & 1;
                const int b0 = chunk_b0(c), bcn = chunk_n(c);
                bool okc = true;
                if (warp < kBfIssuers) {
                    // Lane 0 of warps 0-3 issue the chunk's products, each into an accumulator of
                    // its own (one thread issues a product about every 120 cycles; four keep the
                    // tensor core busy): issuer t takes the window blocks q of parity t & 1 and
                    // the limb pairs (chip, window) (0,0), (1,1), (2,0) when t < 2, else (0,1),
                    // (1,0), (0,2) (integer windows have no third limb).
                    if (lane == 0) {
                        tc::fence_after_sync();
                        const uint32_t wb = tc::smem_u32(s_W);
                        const uint32_t eb = tc::smem_u32(s_E) + static_cast<uint32_t>(s * A.Eb);
                        const int par = warp & 1;
                        const uint32_t dacc = taddr + static_cast<uint32_t>((kBfIssuers * s + warp) * A.AC);
#pragma unroll 1
                        for (int pp = 0; pp < 3; ++pp) {
                            const int cl = warp < 2 ? pp : (pp == 1 ? 1 : 0);
                            const int wl = warp < 2 ? (pp == 1 ? 1 : 0) : (pp == 0 ? 1 : pp == 2 ? 2 : 0);
                            if (Tr::integer && wl == 2) continue;
                            const uint64_t da0 = tc::smem_desc(wb + static_cast<uint32_t>(wl * wlimb),
                                                               static_cast<uint32_t>(A.LW * 16), 128);
                            const uint64_t db0 = tc::smem_desc(eb + static_cast<uint32_t>(cl * elimb),
                                                               static_cast<uint32_t>(A.NB * 16), 128);
                            const uint32_t a_hi = static_cast<uint32_t>(da0 >> 32);
                            const uint32_t b_hi = static_cast<uint32_t>(db0 >> 32);
                            for (int q = par; q < QBp; q += 2) {
                                int elo, n;
                                if (!block_rows(q, A.NB, nr, &elo, &n)) continue;
                                const uint32_t idesc = tc::idesc_bf16_f32(64, n);
                                const uint32_t dcol = static_cast<uint32_t>(16 * q + elo - (A.NB - 16));
                                for (int bl = 0; bl < bcn; ++bl) {
                                    // A: block q, first half, window column x = b0 - ob0 + bl.
                                    const uint32_t a_lo = static_cast<uint32_t>(da0) +
                                                          static_cast<uint32_t>((q * 2) * A.LW + (b0 - ob0) + bl);
                                    const uint32_t b_lo = static_cast<uint32_t>(db0) +
                                                          static_cast<uint32_t>((bl * 2) * A.NB + elo);
                                    tc::mma_bf16_halves(dacc + dcol, a_lo, a_hi, b_lo, b_hi, idesc, 1u);
                                }
                            }
                        }
                        tc::mma_commit(&s_mbar[s]);
                    }
                    __syncwarp();
                    TC_PHASE(9)
                    if (c >= 1) {
                        okc = tc::mbar_wait(&s_mbar[s ^ 1], ph[s ^ 1], kTcWaitPolls);
                        if (okc) {
                            tc::fence_after_sync();
                            flush_set(s ^ 1);
                            clear_half(s ^ 1);
                        }
                    }
                } else {
                    // Chunk c + 2's chip columns are loaded first and converted last, so the
                    // loads are in flight through the wait, the flush and the operand build.
                    const bool stage = c + 2 < nch;
                    double pr[kBfPre];
                    if (stage) p_load(chunk_b0(c + 2), chunk_n(c + 2), pr, 32 * kBfIssuers, bd - 32 * kBfIssuers);
                    if (c >= 1) {
                        okc = tc::mbar_wait(&s_mbar[s ^ 1], ph[s ^ 1], kTcWaitPolls);
                        if (okc) {
                            tc::fence_after_sync();
                            flush_set(s ^ 1);
                            clear_half(s ^ 1);
                        }
                    }
                    if (okc && c + 1 < nch) build_E(s ^ 1, 32 * kBfIssuers, bd - 32 * kBfIssuers);
                    if (okc && stage) p_store(s, chunk_n(c + 2), pr, 32 * kBfIssuers, bd - 32 * kBfIssuers);
                }
                pend[s] = true;
                tc::fence_proxy_async_smem();
                tc::fence_before_sync();
                if (__syncthreads_or(!okc)) {
                    ok = false;
                    break;
                }
                if (c >= 1) {
                    ph[s ^ 1] ^= 1u;
                    pend[s ^ 1] = false;
                }
                TC_PHASE(8)
            }
            if (ok) {
                // The last chunk's values; each warp clears its half of the set.
                const int sl = (nch - 1) & 1;
                ok = wait_set(sl);
                if (__syncthreads_or(!ok)) {
                    ok = false;
                } else {
                    tc::fence_after_sync();
                    flush_set(sl);
                    clear_half(sl);
                    tc::fence_before_sync();
                    __syncthreads();  // the window limbs are replaced next
                }
            }
            TC_PHASE(8)
        }
        if (!ok) {
            if (tid == 0) atomicExch(A.status, 1);
            failed = true;
            break;
        }

        // Epilogue: every value normalised in FP64 into the surface in shared memory.
        {
            const int ib0 = 32 * half + 2 * (lane & 3);
            const int jb0 = 16 * quarter + (lane >> 2);
            if (32 * half < nr) {
#pragma unroll
                for (int v = 0; v < 16; ++v) {
                    const int i = ib0 + 8 * (v >> 2) + (v & 1), j = jb0 + ((v & 2) ? 8 : 0);
                    if (i < nr && j < nc) {
                        const double num = __dadd_rn(accd[v], __dmul_rn(cshift, sumd));
                        const double den = s_den[j * A.NRS + i];
                        s_surf[j * A.NRS + i] = den > 0.0 ? __double2float_rn(__ddiv_rn(num, den)) : 0.0f;
                    }
                }
            }
        }
        __syncthreads();
        TC_PHASE(10)
        if (A.flops && tid == 0)
            atomicAdd(A.flops, 2ull * static_cast<unsigned long long>(ch) * cw * nr * nc);
        // Integer peak (src/peak.jl:32-61).
        unsigned long long key = 0ull;
        for (int e = tid; e < nr * nc; e += bd) {
            const int i = e % nr, j = e / nr;
            const unsigned long long kk = argmax_key(s_surf[j * A.NRS + i], static_cast<unsigned>(i * nc + j));
            key = kk > key ? kk : key;
        }
        key = block_max_u64(key, reinterpret_cast<unsigned long long*>(s_red));
        if (A.surf_out) {
            float* so = A.surf_out + k * static_cast<int64_t>(A.NRM) * A.NCM;
            for (int e = tid; e < nr * nc; e += bd) so[e] = s_surf[(e / nr) * A.NRS + (e % nr)];
        }
        unsigned rm = 0;
        float pv = 0.0f;
        int pi = 0, pj = 0;
        if (key_decode(key, &rm, &pv)) {
            pi = static_cast<int>(rm / nc);
            pj = static_cast<int>(rm % nc);
        }
        if (A.up == 1 || nr < 5 || nc < 5) {
            if (tid == 0) {
                A.out.dx[k] = __double2float_rn(
                    __dadd_rn(static_cast<double>(pj - static_cast<int>(prx)), A.pts.dx0[k]));
                A.out.dy[k] = __double2float_rn(
                    __dadd_rn(static_cast<double>(pi - static_cast<int>(pry)), A.pts.dy0[k]));
                A.out.corr[k] = s_surf[pj * A.NRS + pi];
            }
        } else {
            const int pi0 = min(max(pi - 2, 0), max(nr - 5, 0));
            const int pj0 = min(max(pj - 2, 0), max(nc - 5, 0));
            // The products were here and nothing gave up: the slot of the refinement queue that is taken now
            // is written (k_refine trusts the count).
            if (warp == 0) {
                int slot = 0;
                if (lane == 0) slot = atomicAdd(A.sub_count, 1);
                slot = __shfl_sync(kFull, slot, 0);
                if (lane < 25) {
                    const int a = lane % 5, b = lane / 5;
                    A.sub_patch[static_cast<int64_t>(slot) * 25 + lane] = s_surf[(pj0 + b) * A.NRS + (pi0 + a)];
                }
                if (lane == 0) {
                    A.sub_point[slot] = k;
                    A.sub_origin[2 * slot] = pi0;
                    A.sub_origin[2 * slot + 1] = pj0;
                }
            }
        }
        TC_PHASE(11)
        TC_PHASE_POINT
    }
    TC_PHASE_FLUSH
    // Products still in flight after a failed wait finish before their columns are freed.
    for (int s = 0; s < 2; ++s)
        if (pend[s]) tc::mbar_wait(&s_mbar[s], ph[s], kTcWaitPolls);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(taddr, A.tmem_cols);
}

// ----------------------------------------------------------------------------------------------
// Sub-pixel cascade kernel (src/peak.jl:456-522 from the patch onward), one warp per patch.
//
// The cascade is a subdivision scheme (each pyrUp step is one step of the cubic B-spline's, with
// an even reflection before the first sample and a constant extension after the last), so the
// kernel zooms in on the maximum instead of computing the (5 2^L)^2 samples of the final level.
// Second differences shrink by at least 4 a level, and a step moves a sample by at most an
// eighth of its second difference along each axis, so the final samples of a level's cell (the
// square between four neighbouring nodes) differ from the bilinear interpolant of its nodes by at
// most e = (Dr + Dc) / 6, with Dr and Dc the largest second differences around it: they are below
// the largest corner plus e, and the final sample at a node is at least the node less e. At each
// level the warp keeps the cells that touch a node whose value plus e reaches the best lower bound
// seen, computes the next level over the box of those cells only (for a single peak 3 to 4 cells a
// side, so about 12 x 12 samples a level), and takes the maximum over the last box. Boxes wider
// than kZT cells are cut into tiles that are visited depth first, each skipped when its bound is
// below the best value by then; patches with infinities or magnitudes beyond 1e30 are
// searched whole, tile by tile. A final sample that is not NaN comes from nodes that are not, so NaN
// nodes are left out like small ones; only a node whose neighbours are all numbers has a
// final sample to bound from below. A patch of zeros is its own answer (searched, one of them took 1.3 ms
// at 64x and 5 ms at 128x: nothing is ever below its bound). Rounding: every step is within 2^-20 max|patch| of the exact step
// on the same samples, and e carries that for all levels. Every computed sample is the same
// function of the same inputs as in the full cascade and every sample left out is strictly below
// another one, so the value and its row-major-first position are exactly the full cascade's.
//
// Bound: dependent shared-memory loads and arithmetic of one warp (no HBM traffic to speak of).
// Tiles are as wide as the 16 rows a half warp takes; the next patch is fetched while the current
// one is searched. Measured at 64x: 251 001 patches 3.69 -> 1.11 ms, 1.8 M patches of a
// 10980 x 10980 scene 27.7 ms before (all three levels materialised, then a block search).

constexpr int kRefineWarps = 8;
constexpr int kRefineSplit = 4;      // warps to a patch in passes of few patches
constexpr int kZT = 6;               // level cells per tile side
constexpr int kZR = 2 * (kZT + 2);   // side of a stored region (rows, and its leading dimension)
constexpr int kZC = kZT + 4;         // source columns of a tile's vertical pass
constexpr int kZStack = 16;          // ints of tile state per level

struct RefineArgs {
    const int* count;       // device count of queued items (or null: use n_items)
    int64_t n_items;
    const int64_t* point;   // point index per item (null for bare patches)
    const int32_t* origin;  // patch origin per item (null for bare patches)
    const float* patch;     // 25 floats per item
    DevPoints pts;
    DevOutputs out;
    int32_t* orow;          // bare-patch outputs (when point is null)
    int32_t* ocol;
    float* oval;
    int levels;             // log2(upsampling) >= 1
    int warp_floats;        // shared floats per warp
};

// (value, row-major index) pairs: larger value wins, equal values go to the smaller index;
// NaN never wins.
__device__ __forceinline__ void best_update(float v, int idx, float& bv, int& bi) {
    if (v > bv || (v == bv && idx < bi)) {
        bv = v;
        bi = idx;
    }
}

__device__ __forceinline__ void warp_best(float& bv, int& bi) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float v2 = __shfl_xor_sync(kFull, bv, o);
        const int i2 = __shfl_xor_sync(kFull, bi, o);
        best_update(v2, i2, bv, bi);
    }
}

// A region of a level: rows r0 .. and columns c0 .. stored column-major with leading dimension
// kZR from `p`.
struct Region {
    float* p;
    int r0, c0;
};

// A window of nodes [a, b] x [c, d] of a level.
struct Window {
    int a, b, c, d;
};

// One pyrUp step of nodes [lo_r, hi_r] x [lo_c, hi_c] of a level with n samples a side: nodes 2k
// and 2k + 1 of an axis come from samples k - 1 (1 at k = 0), k and k + 1 (k at the last), which
// is the closed form of src/peak.jl:312-324, in the reference's operation order, vertical pass
// first (src/peak.jl:261-292). `emit(row, column, value)` receives output (row, column) relative
// to (2 lo_r, 2 lo_c). The even outputs of the first node read sample lo - 1, which a region that
// does not start there does not hold: they are computed from sample lo instead and never used.
template <typename Emit>
__device__ __forceinline__ void zoom_step(const Region& S, int n, int lo_r, int hi_r, int lo_c,
                                          int hi_c, float* tmp, Emit emit) {
    const int lane = threadIdx.x & 31;
    const int cs = max(lo_c - 1, S.c0), ce = min(hi_c + 1, n - 1);
    {
        const int r = lo_r + (lane & 7);
        if (r <= hi_r) {
            const int m = max(r == 0 ? 1 : r - 1, S.r0) - S.r0, q = min(r + 1, n - 1) - S.r0;
            const float* col = S.p + (cs + (lane >> 3) - S.c0) * kZR;
            float* t = tmp + (lane >> 3) * kZR + 2 * (lane & 7);
            for (int c = cs + (lane >> 3); c <= ce; c += 4) {
                const float a = col[m], b = col[r - S.r0], d = col[q];
                *reinterpret_cast<float2*>(t) =
                    make_float2(pyr_sample(3, a, b, d), pyr_sample(2, b, b, d));
                col += 4 * kZR;
                t += 4 * kZR;
            }
        }
    }
    __syncwarp();
    {
        const int row = lane & 15;
        if (row <= 2 * (hi_r - lo_r) + 1) {
            for (int c = lo_c + (lane >> 4); c <= hi_c; c += 2) {
                const int m = max(c == 0 ? 1 : c - 1, cs) - cs, q = min(c + 1, n - 1) - cs;
                const float a = tmp[m * kZR + row], b = tmp[(c - cs) * kZR + row];
                const float d = tmp[q * kZR + row];
                emit(row, 2 * (c - lo_c), pyr_sample(3, a, b, d));
                emit(row, 2 * (c - lo_c) + 1, pyr_sample(2, b, b, d));
            }
        }
    }
    __syncwarp();
}

// SPLIT: the warps of a block (kRefineSplit) search one patch. They do the same until a level's box has
// more than one tile, which they then deal out, and the block takes the best of what they found.
template <bool SPLIT>
__global__ void __launch_bounds__(kRefineWarps * 32, 4) k_refine(const RefineArgs A) {
    extern __shared__ __align__(16) float rsm[];
    __shared__ float s_best[kRefineSplit], s_v0[kRefineSplit];
    __shared__ int s_at[kRefineSplit];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int L = A.levels;
    // Per warp: the patch (5 columns), the vertical pass of a tile, a region for each level
    // 1 .. L - 1, the tiles still to visit of each level.
    float* P0 = rsm + warp * A.warp_floats;
    float* tmp = P0 + 5 * kZR;
    float* reg = tmp + kZC * kZR;
    int* stk = reinterpret_cast<int*>(reg + (L - 1) * kZR * kZR);
    const int nfinal = 5 << L;
    const int64_t count = A.count ? static_cast<int64_t>(*A.count) : A.n_items;
    const int64_t step = SPLIT ? gridDim.x : static_cast<int64_t>(gridDim.x) * warps;
    int64_t item = SPLIT ? blockIdx.x : static_cast<int64_t>(blockIdx.x) * warps + warp;
    float next = item < count && lane < 25 ? A.patch[item * 25 + lane] : 0.0f;
    for (; item < count; item += step) {
        const float pv = next;
        if (item + step < count && lane < 25) next = A.patch[(item + step) * 25 + lane];
        const float amax = warp_max(isnan(pv) ? 0.0f : fabsf(pv) <= 1e30f ? fabsf(pv) : INFINITY);
        const bool prune = amax <= 1e30f;  // no infinity, and far from overflow
        const bool gaps = __any_sync(kFull, isnan(pv));
        // A patch of zeros (a window without variance) stays zeros: its first sample is the answer.
        const bool zeros = amax == 0.0f && !__any_sync(kFull, __float_as_uint(pv) != 0u);
        const float slack = static_cast<float>(L + 2) * fmaf(amax, 9.5367431640625e-07f, 2.3509887e-38f);
        if (lane < 25) P0[(lane / 5) * kZR + lane % 5] = pv;
        __syncwarp();
        float esum = 0.0f;   // (Dr + Dc) / 6 at level 1
        float lb = -INFINITY;
        float bv = -INFINITY;
        int bi = INT_MAX;
        float v0 = NAN;
        int pending = 0;     // levels with tiles left
        int l = 0;           // the level whose tiles are being visited
        Region S{P0, 0, 0};
        Window box{0, 4, 0, 4};
        int tile = 0, ntr = 1, ntc = 1;
        int dealt = -1;      // SPLIT: the level whose tiles are dealt out
        if (zeros) bv = v0 = 0.0f, bi = 0;
        while (!zeros) {
            const int n = 5 << l;
            // The next tile: kZT cells a side.
            Window t = box;
            if (ntr * ntc > 1) {
                t.a = box.a + (tile % ntr) * kZT;
                t.b = min(t.a + kZT, box.b);
                t.c = box.c + (tile / ntr) * kZT;
                t.d = min(t.c + kZT, box.d);
            }
            tile += SPLIT && l == dealt ? kRefineSplit : 1;
            const float e_l = ldexpf(esum, 2 - 2 * l) + slack;
            bool skip = false;
            if (ntr * ntc > 1) {
                const int row = t.a + (lane & 7);
                float mx = -INFINITY;
                if (row <= t.b)
                    for (int c = t.c + (lane >> 3); c <= t.d; c += 4)
                        mx = fmaxf(mx, S.p[(c - S.c0) * kZR + row - S.r0]);
                skip = warp_max(mx) + e_l < lb;
            }
            if (tile < ntr * ntc) {
                if (lane == 0) {
                    int* s = stk + l * kZStack;
                    s[0] = box.a; s[1] = box.b; s[2] = box.c; s[3] = box.d;
                    s[4] = S.r0; s[5] = S.c0; s[6] = tile; s[7] = ntr; s[8] = ntc;
                }
                pending |= 1 << l;
            } else {
                pending &= ~(1 << l);
            }
            bool descend = !skip;
            if (descend) {
                const int lo_r = max(t.a - 1, 0), lo_c = max(t.c - 1, 0);
                const Window w{2 * t.a, t.b == n - 1 ? 2 * n - 1 : 2 * t.b, 2 * t.c,
                               t.d == n - 1 ? 2 * n - 1 : 2 * t.d};
                if (l + 1 == L) {
                    zoom_step(S, n, lo_r, t.b, lo_c, t.d, tmp, [&](int r, int c, float v) {
                        const int i = 2 * lo_r + r, j = 2 * lo_c + c;
                        if (i >= w.a && i <= w.b && j >= w.c && j <= w.d) {
                            best_update(v, i * nfinal + j, bv, bi);
                            if (i == 0 && j == 0) v0 = v;
                        }
                    });
                    if (pending && prune) lb = fmaxf(lb, warp_max(bv));
                    descend = false;
                } else {
                    Region D{reg + l * kZR * kZR, 2 * lo_r, 2 * lo_c};
                    zoom_step(S, n, lo_r, t.b, lo_c, t.d, tmp,
                              [&](int r, int c, float v) { D.p[c * kZR + r] = v; });
                    // The nodes of the window that can hold the maximum, as a box.
                    const int row = D.r0 + (lane & 15);
                    const float* col = D.p + (lane & 15) - D.c0 * kZR;
                    const bool mine = row >= w.a && row <= w.b;
                    auto keep_box = [&](float e) {
                        const float cut = lb - e;
                        unsigned cm = 0u;
                        if (mine)
                            for (int c = w.c + (lane >> 4); c <= w.d; c += 2)
                                if (col[c * kZR] >= cut) cm |= 1u << (c - w.c);
                        const unsigned rows = __ballot_sync(kFull, cm != 0u);
                        const unsigned rm = (rows | (rows >> 16)) & 0xffffu;
                        cm = __reduce_or_sync(kFull, cm);
                        Window k{0, -1, 0, -1};
                        if (cm) {
                            k.a = max(D.r0 + __ffs(rm) - 2, w.a);
                            k.b = min(D.r0 + 32 - __clz(rm), w.b);
                            k.c = max(w.c + __ffs(cm) - 2, w.c);
                            k.d = min(w.c + 32 - __clz(cm), w.d);
                        }
                        return k;
                    };
                    Window k = w;
                    if (prune) {
                        float mx = -INFINITY;
                        if (mine && !gaps) {
#pragma unroll 4
                            for (int c = w.c + (lane >> 4); c <= w.d; c += 2) mx = fmaxf(mx, col[c * kZR]);
                        } else if (mine) {
                            // Of the nodes whose final samples are no NaN (they come from the node and
                            // its neighbours).
                            for (int c = w.c + (lane >> 4); c <= w.d; c += 2) {
                                const float* p = col + c * kZR;
                                const int up = row == 0 ? 1 : -1, dn = row == 2 * n - 1 ? 0 : 1;
                                const float* q = p + (c == 0 ? kZR : -kZR);
                                const float* r = p + (c == 2 * n - 1 ? 0 : kZR);
                                const float near = p[up] + p[dn] + q[0] + q[up] + q[dn] + r[0] + r[up] + r[dn];
                                if (!isnan(near)) mx = fmaxf(mx, p[0]);
                            }
                        }
                        const float top = warp_max(mx);
                        if (l == 0) {
                            // Second differences of the patch bound level 1's loosely; then
                            // level 1's own over the box they leave.
                            float dd = 0.0f, dc = 0.0f;
                            if (lane < 25) {
                                const int r = lane % 5, c = lane / 5;
                                const float* p = P0 + c * kZR + r;
                                const float v2 = 2.0f * p[0];
                                dd = fmaxf(0.0f, fabsf(p[r == 0 ? 1 : -1] + p[r == 4 ? 0 : 1] - v2));
                                dc = fmaxf(0.0f, fabsf(p[c == 0 ? kZR : -kZR] + p[c == 4 ? 0 : kZR] - v2));
                            }
                            esum = (warp_max(dd) + warp_max(dc)) * (1.001f / 24.0f);
                            lb = top - (esum + slack);
                            k = keep_box(esum + slack);
                            float d1 = 0.0f, d2 = 0.0f;
                            if (row >= k.a - 1 && row <= k.b + 1 && row < 10) {
                                for (int c = max(k.c - 1, 0) + (lane >> 4); c <= min(k.d + 1, 9); c += 2) {
                                    const float* p = col + c * kZR;
                                    const float v2 = 2.0f * p[0];
                                    if (row >= k.a && row <= k.b)
                                        d1 = fmaxf(d1, fabsf(p[row == 0 ? 1 : -1] + p[row == 9 ? 0 : 1] - v2));
                                    if (c >= k.c && c <= k.d)
                                        d2 = fmaxf(d2, fabsf(p[c == 0 ? kZR : -kZR] + p[c == 9 ? 0 : kZR] - v2));
                                }
                            }
                            esum = fminf(esum, (warp_max(d1) + warp_max(d2)) * (1.001f / 6.0f));
                        }
                        const float e = ldexpf(esum, -2 * l) + slack;
                        lb = fmaxf(lb, top - e);
                        k = keep_box(e);
                    }
                    if (k.b >= k.a) {
                        S = D;
                        box = k;
                        ++l;
                        tile = 0;
                        ntr = max(1, (k.b - k.a + kZT - 1) / kZT);
                        ntc = max(1, (k.d - k.c + kZT - 1) / kZT);
                        if (SPLIT && dealt < 0 && ntr * ntc > 1) {
                            dealt = l;
                            tile = warp;
                            if (tile >= ntr * ntc) break;  // none for this warp (and no other level pending)
                        }
                    } else {
                        descend = false;
                    }
                }
            }
            if (descend) continue;
            if (!pending) break;
            // Back to the deepest level with tiles left.
            l = 31 - __clz(pending);
            __syncwarp();
            const int* s = stk + l * kZStack;
            box = Window{s[0], s[1], s[2], s[3]};
            S = Region{l == 0 ? P0 : reg + (l - 1) * kZR * kZR, s[4], s[5]};
            tile = s[6];
            ntr = s[7];
            ntc = s[8];
            __syncwarp();
        }
        warp_best(bv, bi);
        if (L > 3) {
            v0 = NAN;
        } else {
            v0 = __shfl_sync(kFull, v0, 0);  // lane 0 computes sample (0, 0)
        }
        if constexpr (SPLIT) {
            if (lane == 0) {
                s_best[warp] = bv;
                s_at[warp] = bi;
                s_v0[warp] = v0;
            }
            __syncthreads();
            for (int w = 0; w < kRefineSplit; ++w) {
                best_update(s_best[w], s_at[w], bv, bi);
                v0 = isnan(v0) ? s_v0[w] : v0;
            }
            __syncthreads();  // read before the next patch's
        }
        if (lane == 0 && (!SPLIT || warp == 0)) {
            int si = 0, sj = 0;
            float v = bv;
            if (bi != INT_MAX && bv != -INFINITY) {
                si = bi / nfinal;
                sj = bi - si * nfinal;
            } else {
                v = v0;  // nothing above -Inf: the reference reports (1,1)
            }
            if (A.point) {
                const int64_t k = A.point[item];
                const int i0 = A.origin[2 * item], j0 = A.origin[2 * item + 1];
                const double factor = static_cast<double>(1 << L);
                const double row = __dadd_rn(__ddiv_rn(static_cast<double>(si), factor), static_cast<double>(i0));
                const double col = __dadd_rn(__ddiv_rn(static_cast<double>(sj), factor), static_cast<double>(j0));
                const double dx = __dsub_rn(col, static_cast<double>(A.pts.rx[k]));
                const double dy = __dsub_rn(row, static_cast<double>(A.pts.ry[k]));
                A.out.dx[k] = __double2float_rn(__dadd_rn(dx, A.pts.dx0[k]));
                A.out.dy[k] = __double2float_rn(__dadd_rn(dy, A.pts.dy0[k]));
                A.out.corr[k] = v;
            } else {
                A.orow[item] = si;
                A.ocol[item] = sj;
                A.oval[item] = v;
            }
        }
        __syncwarp();
    }
}

// ----------------------------------------------------------------------------------------------
// Small helpers

__global__ void k_init_outputs(DevOutputs out, int64_t n, int* sub_count) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i == 0 && sub_count) *sub_count = 0;
    if (i < n) {
        out.dx[i] = __int_as_float(0x7fc00000);
        out.dy[i] = __int_as_float(0x7fc00000);
        out.corr[i] = __int_as_float(0x7fc00000);
        out.searched[i] = 0;
    }
}

// geom: [0] max ch, [1] max cw, [2] max nr, [3] max nc, [4] max px term, [5] max py term,
// [6] 1 while every window fits, [7] searchable count. Warp reductions, one atomic per warp.
__global__ void k_pass_geometry(DevPoints p, int64_t nrows, int64_t ncols, long long* geom) {
    const int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    long long v[6] = {0, 0, 0, 0, 0, 0};
    int fits = 1, cnt = 0;
    if (k < p.n) {
        const int64_t rx = p.rx[k], ry = p.ry[k];
        if (rx > 0 && ry > 0) {
            const int64_t hx = p.csx[k] / 2, hy = p.csy[k] / 2;
            v[0] = 2 * hy;
            v[1] = 2 * hx;
            v[2] = 2 * ry;
            v[3] = 2 * rx;
            v[4] = hx + rx + static_cast<int64_t>(ceil(fabs(p.dx0[k])));
            v[5] = hy + ry + static_cast<int64_t>(ceil(fabs(p.dy0[k])));
            const int64_t wcx = static_cast<int64_t>(floor(p.x[k]));
            const int64_t wcy = static_cast<int64_t>(floor(p.y[k]));
            fits = (wcy - hy - ry) >= 1 && (wcy + hy + ry - 2) <= nrows &&
                   (wcx - hx - rx) >= 1 && (wcx + hx + rx - 2) <= ncols;
            cnt = 1;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] = max(v[q], __shfl_xor_sync(kFull, v[q], o));
        fits &= __shfl_xor_sync(kFull, fits, o);
        cnt += __shfl_xor_sync(kFull, cnt, o);
    }
    if ((threadIdx.x & 31) == 0 && cnt > 0) {
#pragma unroll
        for (int q = 0; q < 6; ++q) atomicMax(&geom[q], v[q]);
        if (!fits) atomicMin(&geom[6], 0ll);
        atomicAdd(reinterpret_cast<unsigned long long*>(&geom[7]), static_cast<unsigned long long>(cnt));
    }
}

inline int round_up(int v, int m) { return (v + m - 1) / m * m; }

// Window stride: even with an odd half, so that 16 lanes reading float2 at consecutive
// columns hit 16 distinct 8-byte bank pairs.
inline int window_stride(int rows) {
    int s = round_up(rows, 2);
    if ((s / 2) % 2 == 0) s += 2;
    return s;
}

struct CorrPlan {
    int TI, TJ, CHP, CWM, WS, PHS, NRS, NCM, BC;
    unsigned off_win, off_ph1, off_ph2, off_surf, off_red, off_surf2;
    size_t smem;
};

// `rot`: the rotation search, which stages the whole chip (it is resampled once per angle) and
// holds a second surface, the best one so far.
bool plan_corr(const PassGeometry& g, size_t ph_bytes, size_t smem_cap, CorrPlan* P,
               bool rot = false) {
    const int ch = static_cast<int>(g.max_ch), cw = static_cast<int>(g.max_cw);
    const int nr = static_cast<int>(g.max_nr), nc = static_cast<int>(g.max_nc);
    P->CHP = round_up(std::max(ch, 1), kUA);
    P->CWM = std::max(cw, 1);
    P->NRS = std::max(nr, 1);
    P->NCM = std::max(nc, 1);
    // The whole chip staged once per point if it fits, otherwise chunks of BC chip columns
    // (even, so FP32 partial flushes fall where they would unchunked). Within that, columns
    // per tile: as many as fit one thread each with at least one row group, rows to fill the
    // block; shrink until the shared-memory budget is met.
    const int bcs[] = {P->CWM, 64, 32, 16, 8, 4, 2};
    for (int bc : bcs) {
        if (bc > P->CWM || (bc < P->CWM && (bc & 1)) || (rot && bc < P->CWM)) continue;
        for (int TJ = std::min(nc, kCorrThreads); TJ >= 1; TJ = (TJ > 8 ? TJ - 8 : TJ - 1)) {
            const int groups = std::max(1, kCorrThreads / TJ);
            for (int TI = std::min(round_up(nr, kMI), groups * kMI); TI >= kMI; TI -= kMI) {
                const int WS = window_stride(TI + P->CHP);
                const int PHS = TI + ch + 1;
                size_t off = static_cast<size_t>(P->CHP) * bc * 4;
                off = (off + 15) & ~size_t(15);
                const unsigned off_win = static_cast<unsigned>(off);
                off += static_cast<size_t>(WS) * (TJ + bc - 1) * 4;
                off = (off + 15) & ~size_t(15);
                const unsigned off_ph1 = static_cast<unsigned>(off);
                off += static_cast<size_t>(PHS) * TJ * ph_bytes;
                off = (off + 15) & ~size_t(15);
                const unsigned off_ph2 = static_cast<unsigned>(off);
                off += static_cast<size_t>(PHS) * TJ * ph_bytes;
                off = (off + 15) & ~size_t(15);
                const unsigned off_surf = static_cast<unsigned>(off);
                off += static_cast<size_t>(P->NRS) * P->NCM * 4;
                off = (off + 15) & ~size_t(15);
                const unsigned off_red = static_cast<unsigned>(off);
                off += 3 * 32 * 8;
                off = (off + 15) & ~size_t(15);
                unsigned off_surf2 = off_surf;
                if (rot) {
                    off_surf2 = static_cast<unsigned>(off);
                    off += static_cast<size_t>(P->NRS) * P->NCM * 4;
                }
                if (off <= smem_cap) {
                    P->TI = TI;
                    P->TJ = TJ;
                    P->WS = WS;
                    P->PHS = PHS;
                    P->BC = bc;
                    P->off_win = off_win;
                    P->off_ph1 = off_ph1;
                    P->off_ph2 = off_ph2;
                    P->off_surf = off_surf;
                    P->off_red = off_red;
                    P->off_surf2 = off_surf2;
                    P->smem = off;
                    return true;
                }
            }
            if (TJ == 1) break;
        }
    }
    return false;
}

// Plan of k_corr_fp; false when the surface exceeds one tile (a row group of a column pair per
// thread), the window one column per thread, or shared memory.
bool plan_corr_fp(const PassGeometry& g, size_t smem_cap, bool rot, bool integer, CorrPlan* P) {
    if (g.max_ch > 1024 || g.max_cw > 1024 || g.max_nr > 512 || g.max_nc > 512) return false;
    const int ch = static_cast<int>(g.max_ch), cw = static_cast<int>(g.max_cw);
    const int nr = static_cast<int>(g.max_nr), nc = static_cast<int>(g.max_nc);
    if (ch < 2 || cw < 2 || nr < 2 || nc < 2) return false;
    if (ch * cw > 66000) return false;  // UInt8 sums of squares stay below 2^32
    const int ngrp = (nr + kMI - 1) / kMI;
    if (ngrp * (nc / 2) > kCorrThreads || cw + nc - 1 > kCorrThreads) return false;
    P->CHP = round_up(ch, kUA);
    P->CWM = cw;
    P->NRS = nr | 1;
    P->NCM = nc;
    P->BC = cw;
    P->TJ = P->PHS = 0;
    P->WS = (ngrp * kMI + P->CHP) | 1;  // pairs; odd
    auto a16 = [](size_t v) { return (v + 15) & ~size_t(15); };
    size_t off = a16(static_cast<size_t>(cw) * P->CHP * 4);
    P->off_win = static_cast<unsigned>(off);
    // Every column's run of rows is read to its end by the products' loads.
    const size_t win = static_cast<size_t>(2 * ((cw + nc) / 2)) * P->WS * 8 + 128;
    // The partial sums of split products (20 FP64 values of half of the threads) take the window's
    // place; with the rotation search of an integer image, whose window stays, the column sums',
    // which are done by then.
    const size_t ex = static_cast<size_t>(2 * kMI) * (kCorrThreads / 2) * 8;
    const bool keep = rot && integer;
    P->off_surf2 = static_cast<unsigned>(off);
    off += a16(keep ? win : std::max(win, ex));
    P->off_ph1 = static_cast<unsigned>(off);
    if (keep) P->off_surf2 = static_cast<unsigned>(off);
    // Rows of each segment's column sums: eight where two CTAs per SM (112 KB each) still fit, else
    // four.
    const size_t raw = rot ? a16(static_cast<size_t>(cw) * P->CHP * 4) : 0;
    const size_t rest = raw + a16(static_cast<size_t>(nc) * P->NRS * 8) + 3 * 32 * 8;
    const size_t row = 2 * static_cast<size_t>(kCorrThreads) * 8;
    P->TI = off + std::max(8 * row, keep ? ex : 0) + rest <= 111 * 1024 ? 8 : 4;
    off += std::max(P->TI * row, keep ? ex : 0);
    P->off_ph2 = static_cast<unsigned>(off);
    off += a16(static_cast<size_t>(nc) * P->NRS * 8);
    P->off_surf = static_cast<unsigned>(off);
    off += raw;
    P->off_red = static_cast<unsigned>(off);
    off += 3 * 32 * 8;
    P->smem = off;
    return off <= smem_cap;
}

// Whether k_corr_fp is the faster kernel of a one-tile surface. What it saves grows with the chip
// and the surface, while its barriers and half-filled steps around the products do not shrink with them.
// k_corr's time over k_corr_fp's on some 4000 points, without refinement: Float32 and UInt16 chip 4 radius 6
// 0.88, chip 8 radius 12 0.95 and 16 1.15, chip 12 radius 10 0.97 and 16 1.09, chip 16 radius 4 0.93, 8 1.00
// and 10 1.12, chip 24 from 1.13 up; three turned Float32 chips (sums afresh for every angle) chip 8 radius 12
// 0.94 and 16 1.15, chip 16 radius 8 0.95 and 10 1.12, chip 24 from 1.08 up; turned integer chips (sums once)
// chip 4 radius 4 0.96 and 5 1.02, chip 12 radius 4 0.97 and 5 1.05, chip 16 from 1.07 up.
bool corr_fp_pays(const PassGeometry& g, bool rot, bool integer) {
    const int64_t chip = g.max_ch * g.max_cw, surface = g.max_nr * g.max_nc;
    if (rot && integer) return surface >= 100 || chip >= 256;
    return 3 * chip + surface >= (rot ? 1100 : 960);
}

int ilog2_exact(int up) {
    int L = 0;
    while ((1 << L) < up) ++L;
    return (1 << L) == up ? L : -1;
}

struct RefinePlan {
    int levels, warp_floats;
    int warps;    // warps per CTA
    int per_sm;   // CTAs per SM
    size_t smem;
};

// Shared floats per warp of k_refine: the patch, a tile's vertical pass, the regions of levels
// 1 .. L - 1 and the tile state.
RefinePlan plan_refine(int up) {
    RefinePlan R{};
    R.levels = ilog2_exact(up);
    R.warp_floats = (5 + kZC) * kZR + (R.levels - 1) * kZR * kZR + R.levels * kZStack;
    // Warps per CTA for the most resident warps per SM (228 KB of shared memory, 1 KB charged
    // per CTA): the kernel is issue-bound on dependent shared-memory arithmetic, so resident
    // warps, not CTA size, hide its latencies.
    const size_t per_warp = static_cast<size_t>(R.warp_floats) * sizeof(float);
    int best_w = 1, best_sm = 0;
    for (int w = 1; w <= kRefineWarps; ++w) {
        const size_t cta = w * per_warp + 1024;
        if (w * per_warp > static_cast<size_t>(kDynSmemCap)) break;
        const int ctas = static_cast<int>(std::min<size_t>(32, (228 * 1024) / cta));
        if (ctas * w >= best_w * best_sm) {
            best_w = w;
            best_sm = ctas;
        }
    }
    R.warps = best_w;
    R.per_sm = std::max(1, best_sm);
    R.smem = static_cast<size_t>(R.warps) * per_warp;
    return R;
}

// Refinement of at most n patches. Up to four patches an SM a block of kRefineSplit warps takes each: the
// call then waits for its slowest patch, and one whose box does not shrink (noise, ties) visits many tiles.
// Noise, us a call of bare patches with a warp each and split: 50 at 16x 77 and 66, at 64x 92 and 78, 592 at
// 16x 83 and 68; smooth peaks 592 at 16x 59 and 61, 1184 65 and 75.
cudaError_t launch_refine(const RefinePlan& R, const RefineArgs& B, int64_t n, int num_sms, cudaStream_t stream) {
    const bool split = n <= 4 * static_cast<int64_t>(num_sms);
    const int warps = split ? kRefineSplit : R.warps;
    const size_t smem = static_cast<size_t>(warps) * R.warp_floats * sizeof(float);
    if (smem > static_cast<size_t>(kDynSmemCap)) return cudaErrorInvalidValue;
    auto kern = split ? k_refine<true> : k_refine<false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kDynSmemCap);
    if (e != cudaSuccess) return e;
    const int64_t blocks = split ? n : std::min<int64_t>((n + R.warps - 1) / R.warps,
                                                         static_cast<int64_t>(num_sms) * R.per_sm);
    kern<<<static_cast<unsigned>(std::max<int64_t>(1, blocks)), warps * 32, smem, stream>>>(B);
    return cudaGetLastError();
}

// Dynamic shared memory a CTA holding `cols` Tensor Memory columns reserves, for a kernel with
// `static_smem` bytes of static shared memory (see the launch below): with the 1 KB the SM
// charges each CTA, its footprint is at least cols/512 of the SM's 228 KB.
size_t tmem_smem_floor(uint32_t cols, size_t static_smem) {
    const size_t share = static_cast<size_t>(cols) * (228 * 1024) / 512;
    return share > 1024 + static_smem ? share - 1024 - static_smem : 0;
}

struct TcPlan {
    int NB, QM, QS, PS, PC, XS, NRS, NRM, NCM, CHM, CWM, BC, big, MT;
    unsigned off_E, off_W, off_P, off_V, off_S1, off_S2, off_R = 0, off_num, off_est, off_red;
    unsigned off_L = 0, off_rawW = 0, off_rawC = 0;
    int XV = 0, VR = 0, roots = 0, acc1_col = 0, issuers = 2;
    uint32_t tmem_cols;
    size_t smem;
};

// Shared-memory and Tensor Memory plan of k_corr_tc2 for a pass's largest geometry; false when
// the pass does not fit it (surfaces beyond 64 x 64, chip operand larger than shared memory,
// accumulator beyond 512 columns).
// Dynamic shared memory that leaves room for two CTAs (228 KB per SM, less 1 KB and the static
// shared memory of each).
constexpr size_t kTc2TwoCtas = 110 * 1024;
bool plan_corr_tc2(const PassGeometry& g, size_t smem_cap, TcPlan* P) {
    const int ch = static_cast<int>(g.max_ch), cw = static_cast<int>(g.max_cw);
    const int nr = static_cast<int>(g.max_nr), nc = static_cast<int>(g.max_nc);
    if (nc > 64 || nr > 64 || nr < 1 || nc < 1 || cw < 2 || ch < 2 || (cw & 1)) return false;
    P->CHM = ch;
    P->CWM = cw;
    P->NRM = nr;
    P->NCM = nc;
    P->MT = 64;
    P->NB = round_up(ch + 15, 16);
    if (P->NB > 256) return false;
    P->QM = (ch + nr - 1 + 15) / 16;
    P->PS = P->NB * 16;
    P->XS = 64 + cw;
    P->QS = P->XS * 16;
    P->PC = round_up(kPadL + P->NB + 20, 16);
    P->NRS = nr | 1;
    P->XV = round_up(cw + nc - 1, 32) + 4;
    // Four accumulators of 64 or 32 columns, each with an issuing thread (column i is surface row
    // i: the products write columns below round16(nr), the epilogue reads 32 columns per half of
    // the surface rows).
    P->acc1_col = nr > 32 ? 64 : 32;
    P->issuers = 4;
    P->tmem_cols = static_cast<uint32_t>(4 * P->acc1_col);
    auto a16 = [](size_t v) { return (v + 15) & ~size_t(15); };
    const size_t Eb = static_cast<size_t>(cw) * P->PS;
    const size_t Wb = static_cast<size_t>(P->QM) * P->QS;
    const size_t Pb = a16(static_cast<size_t>(cw) * P->PC);
    const size_t nbytes = a16(static_cast<size_t>(nc) * P->NRS * 4);
    const size_t rawW = static_cast<size_t>(cw + nc - 1) * (P->QM + 1) * 16;
    const size_t rawC = 2 * static_cast<size_t>(cw) * ((ch + 15) / 16 + 1) * 16;
    // [E][W][V1, V2 | raw window, raw chip and mask][P][S1][S2][R][L1, L2][red]; every value's numerator
    // takes E and W's place once the products are done. V holds the column sums of `vr` surface
    // rows.
    auto layout = [&](int vr) {
        P->VR = vr;
        size_t off = 0;
        P->off_E = P->off_num = 0;
        off += Eb;
        P->off_W = static_cast<unsigned>(off);
        off = std::max(off + Wb, nbytes);
        P->off_V = P->off_rawW = static_cast<unsigned>(off);
        P->off_rawC = static_cast<unsigned>(off + rawW);
        off += std::max(a16(2 * (static_cast<size_t>(vr) * P->XV + 16) * 4), rawW + rawC);
        P->off_P = static_cast<unsigned>(off);
        off += Pb;
        P->off_S1 = static_cast<unsigned>(off);
        off += nbytes;
        P->off_S2 = static_cast<unsigned>(off);
        off += nbytes;
        P->off_est = static_cast<unsigned>(off);
        off += nbytes;
        P->off_L = static_cast<unsigned>(off);
        off += a16(2 * static_cast<size_t>(P->XV) * 4);
        P->off_red = static_cast<unsigned>(off);
        return off + 3 * 32 * 8;
    };
    // As many rows of V as leave room for two CTAs per SM (every one of them, else multiples of
    // 16); where not even 16 do, as many as fit one.
    size_t off = 0;
    for (size_t cap : {kTc2TwoCtas, smem_cap}) {
        cap = std::min(cap, smem_cap);
        int vr = nr;
        off = layout(vr);
        while (off > cap && vr > 16) off = layout(vr = std::max(16, (vr - 1) & ~15));
        if (off <= cap) break;
    }
    P->BC = cw;
    P->big = 0;
    P->smem = off;
    return off <= smem_cap;
}

// Plan of k_corr_bf: the chunk of chip columns whose products keep each accumulator element's
// chain near kBfChain, the widest window staging that fits `smem_cap` beside the chip operand
// buffers and the denominators, and the box-sum stripes in the space of both; false when the
// pass's surfaces exceed 64 x 64 or its chips 240 px.
struct BfPlan {
    int NB, QB, BC, OB, LW, PC, NRS, AC, RS, VS, XS;
    unsigned off_S2, off_raw, off_V, off_den, off_E, off_P, off_red, Eb, Pb;
    uint32_t tmem_cols;
    size_t smem;
};

bool plan_corr_bf(const PassGeometry& g, size_t smem_cap, BfPlan* P) {
    const int ch = static_cast<int>(g.max_ch), cw = static_cast<int>(g.max_cw);
    const int nr = static_cast<int>(g.max_nr), nc = static_cast<int>(g.max_nc);
    if (nr < 1 || nc < 1 || nr > 64 || nc > 64 || ch < 2 || cw < 2) return false;
    P->NB = round_up(ch + 15, 16);
    if (P->NB > 256) return false;
    P->QB = (ch + nr - 1 + 15) / 16;
    P->PC = round_up(kBfPadL + P->NB + 26, 8);
    P->NRS = nr | 1;
    // A block's products write accumulator columns [16 q + elo - NB + 16, + n), all below
    // round16(nr) (block_rows: elo, NB multiples of 16, the rows' end at most NB - 16 + nr - 16 q).
    P->AC = round_up(nr, 16);
    if (2 * kBfIssuers * P->AC > 512) return false;  // two sets of kBfIssuers accumulators
    P->tmem_cols = 512;
    P->RS = (ch + nr - 1) | 1;
    P->VS = nr + 1;
    // Window blocks meeting one surface row: (ch + 15) / 16 + 1, half of them (one parity) into
    // an accumulator, with three limb pairs each: 1.5 blocks accumulating steps per chip column.
    const int blocks = (ch + 15) / 16 + 1;
    int bc = std::max(1, 2 * kBfChain / (3 * blocks));
    bc = std::min(bc, cw);
    // The staged chip columns of a chunk: kBfPre elements per thread of warps 4-7.
    const int stagers = kBfThreads - 32 * kBfIssuers;
    while (bc > 1 && bc * P->PC > kBfPre * stagers) --bc;
    if (bc * P->PC > kBfPre * stagers) return false;
    P->BC = bc;
    auto a16 = [](size_t v) { return (v + 15) & ~size_t(15); };
    const size_t Sb = a16(static_cast<size_t>(nc) * P->NRS * 8);
    const size_t Eb = static_cast<size_t>(kBfLimbs) * bc * 2 * P->NB * 16;
    const size_t Pb = a16(static_cast<size_t>(kBfLimbs) * bc * P->PC * 2);
    const size_t red = 3 * 32 * 8;
    const size_t X = Sb + 2 * Eb + 2 * Pb + red;
    const size_t colb = static_cast<size_t>(kBfLimbs) * P->QB * 2 * 16;  // limb bytes per column
    const size_t minL = std::max(2 * Sb, a16(static_cast<size_t>(nc) * P->NRS * 4));
    auto Lof = [&](int ob) { return std::max(minL, static_cast<size_t>(ob + 63) * colb); };
    if (X >= smem_cap) return false;
    int OB = round_up(cw, bc);
    if (Lof(OB) + X > smem_cap) {
        const int lw = static_cast<int>((smem_cap - X) / colb);
        const int ob = (lw - 63) / bc * bc;
        if (ob < bc) return false;
        const int nout = (cw + ob - 1) / ob;
        OB = round_up((cw + nout - 1) / nout, bc);
    }
    P->OB = OB;
    P->LW = OB + 63;
    const size_t L = Lof(OB);
    if (L + X > smem_cap) return false;
    // Box-sum stripes after S1 and S2, up to the reduction scratch.
    const int XW = cw + nc - 1;
    const size_t avail = L + X - red - 2 * Sb;
    const size_t per_col = static_cast<size_t>(P->RS) * 4 + static_cast<size_t>(P->VS) * 16;
    if (avail < per_col + 16) return false;
    P->XS = static_cast<int>(std::min<size_t>(XW, (avail - 16) / per_col));
    P->off_S2 = static_cast<unsigned>(Sb);
    P->off_raw = static_cast<unsigned>(2 * Sb);
    P->off_V = static_cast<unsigned>(a16(2 * Sb + static_cast<size_t>(P->XS) * P->RS * 4));
    if (P->off_V + static_cast<size_t>(P->XS) * P->VS * 16 > L + X - red) return false;
    P->off_den = static_cast<unsigned>(L);
    P->off_E = static_cast<unsigned>(L + Sb);
    P->off_P = static_cast<unsigned>(L + Sb + 2 * Eb);
    P->off_red = static_cast<unsigned>(L + Sb + 2 * Eb + 2 * Pb);
    P->Eb = static_cast<unsigned>(Eb);
    P->Pb = static_cast<unsigned>(Pb);
    P->smem = L + X;
    return true;
}

// A k_corr_tc plan whose shared memory leaves room for one CTA per SM anyway has the SM's 512
// Tensor Memory columns to itself: with M = 64 products (surfaces up to 64 x 64: the chip-128
// levels), which one thread issues only about every 120 cycles, it issues them from four threads
// into four accumulators. M = 128 products are bound by the tensor pipe and keep two.
void four_issuers(TcPlan* P) {
    const bool one_per_sm = 2 * (P->smem + 2048) > 228 * 1024;
    if (one_per_sm && P->MT == 64 && P->NRM <= 64 && 4 * P->acc1_col <= 512) {
        P->issuers = 4;
        P->tmem_cols = static_cast<uint32_t>(4 * P->acc1_col);
    }
}

// Shared-memory plan of k_corr_tc for a pass's largest geometry; false when the pass does not
// fit the kernel (surface wider than 128 columns, more than 256 rows, chips taller than 226).
// [box sums of W and W^2][reciprocal roots][red][P][W][V of a stripe of surface rows][E]: with the
// whole chip operand E beside the stripe the box sums run beside the products. Otherwise the box sums
// come first and the chip operand in chunks of BC columns in the stripe's place, without the
// roots (they would cost a chip-64, radius-48 pass a chunk more). Either in half of an SM's
// shared memory comes before either in all of it: 1.24 ms with two CTAs and chunks against 1.55
// with one and the whole operand (14 400 points, chip 32, radius 44). Not so for passes without a
// point for each SM and one more (`many`), which wait for one point's latency (56 points at chip 16,
// radius 40: 77 us a call with two, 75 with one), nor in chunks for surfaces up to 64 x 64, whose products
// four threads issue where the SM is theirs alone (13 689 points at chip 128, radius 25: 3.93 ms
// with two, 3.83 with one). The list of candidates of
// surfaces up to 64 x 64 takes the place of W, V and E once the products are done (P keeps its
// zero padding between points).
bool plan_corr_tc(const PassGeometry& g, size_t smem_cap, bool many, TcPlan* P) {
    const int ch = static_cast<int>(g.max_ch), cw = static_cast<int>(g.max_cw);
    const int nr = static_cast<int>(g.max_nr), nc = static_cast<int>(g.max_nc);
    if (nc > 128 || nr > 256 || nr < 1 || nc < 1 || cw < 2 || ch < 2 || (cw & 1)) return false;
    P->CHM = ch;
    P->CWM = cw;
    P->NRM = nr;
    P->NCM = nc;
    P->MT = nc <= 64 ? 64 : 128;
    P->NB = round_up(ch + 30, 16);
    if (P->NB > 256) return false;
    P->QM = (15 + ch + nr - 1 + 15) / 16;
    P->PS = P->NB * 16;
    P->XS = P->MT + cw;
    P->QS = P->XS * 16;
    P->XV = round_up(cw + nc - 1, 4);
    P->PC = round_up(kPadL + P->NB + 20, 16);
    P->NRS = nr | 1;
    // Two accumulators, each holding the columns of surface rows 0 .. nr + 15 (the products'
    // rows are trimmed to the surface rows) and whatever the epilogue's reads reach.
    const int used = (nr + 16 + 15) & ~15;
    const int reads = P->MT == 64 ? 32 * ((nr + 31) / 32) : 16 * ((nr + 15) / 16);
    uint32_t cols = 32;
    while (static_cast<int>(cols) < std::max(used, reads)) cols <<= 1;
    if (2 * cols > 512) return false;
    P->acc1_col = static_cast<int>(cols);
    P->tmem_cols = 2 * cols;
    auto a16 = [](size_t v) { return (v + 15) & ~size_t(15); };
    const size_t Eb = static_cast<size_t>(cw) * P->PS;
    const size_t Wb = static_cast<size_t>(P->QM) * P->QS;
    const size_t Pb = a16(static_cast<size_t>(cw) * P->PC);
    const size_t nbytes = a16(static_cast<size_t>(nc) * P->NRS * 4);
    const size_t red = 3 * 32 * 8;
    const size_t row = 2 * static_cast<size_t>(P->XV) * 4;
    const bool listed = P->MT == 64 && nr <= 64;
    auto front = [&](int roots) {
        P->roots = roots;
        size_t off = 0;
        P->off_S1 = 0;
        off += nbytes;
        P->off_S2 = static_cast<unsigned>(off);
        off += nbytes;
        P->off_R = static_cast<unsigned>(off);
        off += roots ? nbytes : 0;
        P->off_red = static_cast<unsigned>(off);
        off = a16(off + red);
        P->off_P = static_cast<unsigned>(off);
        off += Pb;
        P->off_W = P->off_num = static_cast<unsigned>(off);
        P->off_est = static_cast<unsigned>(off + nbytes);
        off += Wb;
        P->off_V = static_cast<unsigned>(off);
        return off;
    };
    auto stripe = [&](size_t avail) {
        return std::min(round_up(nr, 4), static_cast<int>(avail / row) & ~3);
    };
    for (size_t cap : {kTc2TwoCtas, smem_cap}) {
        if (cap < smem_cap && !many) continue;
        const int least = cap < smem_cap ? 8 : 16;  // rows of a stripe (and columns of a chunk)
        size_t off = front(listed ? 0 : 1);
        size_t num_end = listed ? P->off_est + nbytes : 0;
        if (std::max(num_end, off + least * row + Eb) <= cap) {
            P->VR = stripe(cap - off - Eb);
            P->off_E = static_cast<unsigned>(off + P->VR * row);
            P->BC = cw;
            P->big = 0;
            P->smem = std::max(num_end, off + P->VR * row + Eb);
            four_issuers(P);
            return true;
        }
        if (cap < smem_cap && listed) continue;
        off = front(0);
        num_end = listed ? P->off_est + nbytes : 0;
        const size_t columns = std::min(cw, cap < smem_cap ? least : 2);
        if (std::max(num_end, off + std::max(least * row, columns * P->PS)) <= cap) {
            const int most = static_cast<int>(std::min<size_t>(cw, (cap - off) / P->PS)) & ~1;
            const int n = (cw + most - 1) / most;
            P->BC = std::min(most, round_up((cw + n - 1) / n, 2));
            P->big = 1;
            P->VR = stripe(cap - off);
            P->off_E = P->off_V;
            P->smem = std::max(num_end, off + std::max(P->VR * row, static_cast<size_t>(P->BC) * P->PS));
            four_issuers(P);
            return true;
        }
    }
    return false;
}

template <typename T>
cudaError_t launch_corr_t(const CorrArgs& A, const CorrPlan& P, int grid, cudaStream_t stream, bool fp) {
    if (P.smem > static_cast<size_t>(kDynSmemCap)) return cudaErrorInvalidValue;
    auto kern = A.rot.count > 0 ? k_corr<T, true> : k_corr<T, false>;
    if (fp) {
        if constexpr (Traits<T>::raw) {
            kern = k_corr_fp<T, true>;  // the integer numerator stays with k_corr
        } else {
            kern = A.rot.count > 0 ? k_corr_fp<T, true> : k_corr_fp<T, false>;
        }
    }
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kDynSmemCap);
    if (e != cudaSuccess) return e;
    kern<<<grid, kCorrThreads, P.smem, stream>>>(A);
    return cudaGetLastError();
}


std::atomic<long long> g_scratch_allocs{0};

cudaError_t ensure_scratch(TrackScratch& s, int64_t n, cudaStream_t stream) {
    if (s.fixed) {
        // Caller-provided buffers: never allocate; a pass beyond them is an error.
        if (!s.geom || !s.sub_count || !s.status || !s.sub_point || !s.sub_origin || !s.sub_patch)
            return cudaErrorInvalidValue;
        return s.capacity >= n ? cudaSuccess : cudaErrorMemoryAllocation;
    }
    if (!s.geom) {
        cudaError_t e = cudaMalloc(&s.geom, 8 * sizeof(int64_t));
        if (e != cudaSuccess) return e;
        ++g_scratch_allocs;
    }
    if (!s.sub_count) {
        cudaError_t e = cudaMalloc(&s.sub_count, sizeof(int));
        if (e != cudaSuccess) return e;
        ++g_scratch_allocs;
    }
    if (!s.status) {
        cudaError_t e = cudaMalloc(&s.status, sizeof(int));
        if (e == cudaSuccess) e = cudaMemset(s.status, 0, sizeof(int));
        if (e != cudaSuccess) return e;
        ++g_scratch_allocs;
    }
    if (s.capacity >= n) return cudaSuccess;
    const int64_t cap = std::max<int64_t>(n, 1024);
    cudaError_t e = cudaSuccess;
    g_scratch_allocs += 3;
    if (s.pool) {
        // Stream-ordered: the old queue is released after the work already on `stream`.
        if (s.sub_point) cudaFreeAsync(s.sub_point, stream);
        if (s.sub_origin) cudaFreeAsync(s.sub_origin, stream);
        if (s.sub_patch) cudaFreeAsync(s.sub_patch, stream);
        s.sub_point = nullptr;
        s.sub_origin = nullptr;
        s.sub_patch = nullptr;
        s.capacity = 0;
        void* a = nullptr;
        void* b = nullptr;
        void* c = nullptr;
        e = cudaMallocFromPoolAsync(&a, cap * sizeof(int64_t), s.pool, stream);
        if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&b, cap * 2 * sizeof(int32_t), s.pool, stream);
        if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&c, cap * 25 * sizeof(float), s.pool, stream);
        s.sub_point = static_cast<int64_t*>(a);
        s.sub_origin = static_cast<int32_t*>(b);
        s.sub_patch = static_cast<float*>(c);
    } else {
        cudaFree(s.sub_point);
        cudaFree(s.sub_origin);
        cudaFree(s.sub_patch);
        s.sub_point = nullptr;
        s.sub_origin = nullptr;
        s.sub_patch = nullptr;
        s.capacity = 0;
        e = cudaMalloc(&s.sub_point, cap * sizeof(int64_t));
        if (e == cudaSuccess) e = cudaMalloc(&s.sub_origin, cap * 2 * sizeof(int32_t));
        if (e == cudaSuccess) e = cudaMalloc(&s.sub_patch, cap * 25 * sizeof(float));
    }
    if (e != cudaSuccess) return e;
    s.capacity = cap;
    return cudaSuccess;
}

}  // namespace

bool make_rotation(const double* deg, int count, Rotation* out, std::string* err) {
    if (count < 1 || count > kMaxAngles) {
        if (err) *err = "the rotation search needs 1 to " + std::to_string(kMaxAngles) + " angles";
        return false;
    }
    if (!deg) {
        if (err) *err = "null rotation angles";
        return false;
    }
    for (int i = 0; i < count; ++i) {
        if (!std::isfinite(deg[i])) {
            if (err) *err = "rotation angles must be finite";
            return false;
        }
        for (int j = 0; j < i; ++j)
            if (deg[j] == deg[i]) {
                if (err) *err = "rotation angles must be distinct";
                return false;
            }
    }
    out->count = count;
    for (int i = 0; i < count; ++i) {
        // deg2rad (deg * (pi / 180)), then the C library's sin and cos.
        const double r = deg[i] * (M_PI / 180.0);
        out->sn[i] = std::sin(r);
        out->cs[i] = std::cos(r);
        out->turn[i] = deg[i] != 0.0 ? 1 : 0;
    }
    for (int i = count; i < kMaxAngles; ++i) {
        out->sn[i] = 0.0;
        out->cs[i] = 1.0;
        out->turn[i] = 0;
    }
    return true;
}

cudaEvent_t KernelTimer::get() {
    if (!pool.empty()) {
        cudaEvent_t e = pool.back();
        pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}

PassGeometry pass_geometry_host(const ar_points& p, int64_t nrows, int64_t ncols) {
    PassGeometry g;
    bool fits = true;
    int64_t px = 0, py = 0;
    for (int64_t k = 0; k < p.n; ++k) {
        const int64_t rx = p.radius_x[k], ry = p.radius_y[k];
        if (!(rx > 0 && ry > 0)) continue;
        const int64_t hx = p.chip_size_x[k] / 2, hy = p.chip_size_y[k] / 2;
        g.max_ch = std::max(g.max_ch, 2 * hy);
        g.max_cw = std::max(g.max_cw, 2 * hx);
        g.max_nr = std::max(g.max_nr, 2 * ry);
        g.max_nc = std::max(g.max_nc, 2 * rx);
        px = std::max(px, hx + rx + static_cast<int64_t>(std::ceil(std::fabs(p.dx_prior[k]))));
        py = std::max(py, hy + ry + static_cast<int64_t>(std::ceil(std::fabs(p.dy_prior[k]))));
        const int64_t wcx = static_cast<int64_t>(std::floor(p.x[k]));
        const int64_t wcy = static_cast<int64_t>(std::floor(p.y[k]));
        fits = fits && (wcy - hy - ry) >= 1 && (wcy + hy + ry - 2) <= nrows &&
               (wcx - hx - rx) >= 1 && (wcx + hx + rx - 2) <= ncols;
        ++g.searchable;
    }
    g.padx = fits ? 0 : px + 2;
    g.pady = fits ? 0 : py + 2;
    return g;
}

cudaError_t scratch_acquire(TrackScratch& s, cudaStream_t stream);

cudaError_t read_status(TrackScratch& scratch, cudaStream_t stream, int* status) {
    *status = 0;
    if (!scratch.status) return cudaSuccess;
    cudaError_t e = cudaMemcpyAsync(status, scratch.status, sizeof(int), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e == cudaSuccess && *status) e = cudaMemsetAsync(scratch.status, 0, sizeof(int), stream);
    return e;
}

cudaError_t pass_geometry_device(const DevPoints& pts, int64_t nrows, int64_t ncols,
                                 TrackScratch& scratch, cudaStream_t stream, PassGeometry* out) {
    cudaError_t e = scratch_acquire(scratch, stream);
    if (e != cudaSuccess) return e;
    e = ensure_scratch(scratch, 0, stream);
    if (e != cudaSuccess) return e;
    long long init[8] = {0, 0, 0, 0, 0, 0, 1, 0};
    e = cudaMemcpyAsync(scratch.geom, init, sizeof(init), cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return e;
    if (pts.n > 0) {
        const int threads = 256;
        const int64_t blocks = (pts.n + threads - 1) / threads;
        k_pass_geometry<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(
            pts, nrows, ncols, reinterpret_cast<long long*>(scratch.geom));
        scratch.timer.launches += 1;
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    long long g[8];
    e = cudaMemcpyAsync(g, scratch.geom, sizeof(g), cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess) return e;
    e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return e;
    out->max_ch = g[0];
    out->max_cw = g[1];
    out->max_nr = g[2];
    out->max_nc = g[3];
    const bool fits = g[6] != 0;
    out->padx = fits ? 0 : g[4] + 2;
    out->pady = fits ? 0 : g[5] + 2;
    out->searchable = g[7];
    return cudaSuccess;
}

// The scratch buffers are shared by the passes of a context; a pass on one stream waits for
// the last pass that used them, whichever stream that ran on.
cudaError_t scratch_acquire(TrackScratch& s, cudaStream_t stream) {
    if (!s.done) {
        if (s.fixed) return cudaSuccess;  // no event is created for a caller-provided view
        ++g_scratch_allocs;
        return cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming);
    }
    return cudaStreamWaitEvent(stream, s.done, 0);
}

long long scratch_allocations() { return g_scratch_allocs.load(); }

// Passes of at least this many points enter the context's table of geometries and kernels.
constexpr int64_t kTuneMinPoints = 8192;

cudaError_t launch_track_impl(int dtype, const void* ref, const void* sec, const uint8_t* valid,
                              int64_t nrows, int64_t ncols, const DevPoints& pts,
                              const PassGeometry& geom, int up, int measure,
                              const DevOutputs& out, TrackScratch& scratch, int num_sms,
                              cudaStream_t stream, std::string* err, float* surf_out,
                              const Rotation* rot) {
    cudaError_t e = ensure_scratch(scratch, pts.n, stream);
    if (e != cudaSuccess) return e;
    if (pts.n > 0) {
        const int threads = 256;
        k_init_outputs<<<static_cast<unsigned>((pts.n + threads - 1) / threads), threads, 0, stream>>>(
            out, pts.n, scratch.sub_count);
        scratch.timer.launches += 1;
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (geom.searchable == 0 || geom.max_cw == 0 || geom.max_ch == 0) return cudaSuccess;

    const bool rotating = rot && rot->count > 0;
    const size_t ph_bytes = dtype == AR_U8 && !rotating ? 4 : 8;
    CorrPlan P{};
    // One-tile surfaces with an FP32 numerator take k_corr_fp: turned chips (but not with a
    // diagnostic surface, which k_corr keeps across angles) and the types other than UInt8 (surfaces of
    // more than one point, at max_nr rows each, are k_corr's: k_corr_fp's have a row more).
    const bool fp = (rotating ? !surf_out : dtype != AR_U8 && (!surf_out || pts.n == 1)) && corr_fp_pays(geom, rotating, dtype != AR_F32) &&
                    plan_corr_fp(geom, 220 * 1024, rotating, dtype != AR_F32, &P);
    if (!fp && !plan_corr(geom, ph_bytes, 220 * 1024, &P, rotating)) {
        if (err) *err = rotating ? "chip and search geometry too large for shared memory with "
                                   "the rotation search"
                                 : "chip and search geometry too large for shared memory";
        return cudaErrorInvalidValue;
    }
    CorrArgs A{};
    if (rotating) A.rot = *rot;
    A.off_surf2 = P.off_surf2;
    A.ref = ref;
    A.sec = sec;
    A.valid = valid;
    A.nrows = nrows;
    A.ncols = ncols;
    A.pts = pts;
    A.padx = geom.padx;
    A.pady = geom.pady;
    A.up = up;
    A.measure = measure;
    A.TI = P.TI;
    A.TJ = P.TJ;
    if (fp && dtype == AR_F32) {
        CorrPlan G{};
        const bool fits = plan_corr(geom, ph_bytes, 220 * 1024, &G, rotating);
        A.GTI = fits ? G.TI : P.NRS;
        A.GTJ = fits ? G.TJ : P.NCM;
    }
    A.CHP = P.CHP;
    A.CWM = P.CWM;
    A.BC = P.BC;
    A.WS = P.WS;
    A.PHS = P.PHS;
    A.NRS = P.NRS;
    A.NCM = P.NCM;
    A.off_win = P.off_win;
    A.off_ph1 = P.off_ph1;
    A.off_ph2 = P.off_ph2;
    A.off_surf = P.off_surf;
    A.off_red = P.off_red;
    A.out = out;
    A.sub_count = scratch.sub_count;
    A.sub_point = scratch.sub_point;
    A.sub_origin = scratch.sub_origin;
    A.sub_patch = scratch.sub_patch;
    A.surf_out = surf_out;
    A.flops = scratch.timer.enabled ? scratch.timer.flops : nullptr;

    KernelTimer& T = scratch.timer;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr;
    if (T.enabled) {
        ev0 = T.get();
        ev1 = T.get();
        ev2 = T.get();
        cudaEventRecord(ev0, stream);
    }
    // The UInt8 tensor-core kernels: k_corr_tc2 (`tc2`, surfaces up to 64 x 64 with the chip
    // operand whole) or k_corr_tc (surfaces up to 128 columns), planned by `TP`.
    auto launch_tc = [&](bool tc2, const TcPlan& TP, const DevPoints& pts, int up,
                         const DevOutputs& out, unsigned long long* flops) -> cudaError_t {
        TcArgs B{};
        B.ref = static_cast<const uint8_t*>(ref);
        B.sec = static_cast<const uint8_t*>(sec);
        B.valid = valid;
        B.nrows = nrows;
        B.ncols = ncols;
        B.pts = pts;
        B.padx = geom.padx;
        B.pady = geom.pady;
        B.up = up;
        B.measure = measure;
        B.NB = TP.NB;
        B.QM = TP.QM;
        B.QS = TP.QS;
        B.PS = TP.PS;
        B.PC = TP.PC;
        B.XS = TP.XS;
        B.NRS = TP.NRS;
        B.NRM = TP.NRM;
        B.NCM = TP.NCM;
        B.CHM = TP.CHM;
        B.CWM = TP.CWM;
        B.BC = TP.BC;
        B.big = TP.big;
        B.VR = TP.VR;
        B.MT = TP.MT;
        B.off_E = TP.off_E;
        B.off_W = TP.off_W;
        B.off_R = TP.off_R;
        B.roots = TP.roots;
        B.off_P = TP.off_P;
        B.off_V = TP.off_V;
        B.off_S1 = TP.off_S1;
        B.off_S2 = TP.off_S2;
        B.off_num = TP.off_num;
        B.off_est = TP.off_est;
        B.off_red = TP.off_red;
        B.off_L = TP.off_L;
        B.off_rawW = TP.off_rawW;
        B.off_rawC = TP.off_rawC;
        B.XV = TP.XV;
        B.acc1_col = TP.acc1_col;
        B.issuers = TP.issuers;
        B.tmem_cols = TP.tmem_cols;
        B.out = out;
        B.sub_count = scratch.sub_count;
        B.sub_point = scratch.sub_point;
        B.sub_origin = scratch.sub_origin;
        B.sub_patch = scratch.sub_patch;
        B.surf_out = surf_out;
        B.flops = flops;
        B.status = scratch.status;
        // Each CTA holds its Tensor Memory columns for its lifetime, so the CTAs one SM holds
        // must fit its 512 columns together -- including CTAs of other launches running
        // concurrently (other streams, the request loop's slots), or an allocation would wait
        // for a whole persistent launch to end. A CTA of T columns therefore reserves at least
        // T/512 of the SM's 228 KB of shared memory (less the 1 KB each CTA is charged): any set
        // of CTAs that fits an SM's shared memory fits its Tensor Memory.
        const bool reg = TP.MT == 64 && TP.NRM <= 64;
        auto kern = tc2 ? k_corr_tc2 : reg ? k_corr_tc<true> : k_corr_tc<false>;
        cudaFuncAttributes fa{};
        e = cudaFuncGetAttributes(&fa, kern);
        if (e != cudaSuccess) return e;
        // The per-block limit (227 KB, static included) is this kernel's fixed attribute value.
        const size_t dyn_max = 232448 - fa.sharedSizeBytes;
        const size_t tc_smem = std::max<size_t>(TP.smem, tmem_smem_floor(TP.tmem_cols, fa.sharedSizeBytes));
        const int per_sm_tc = static_cast<int>(std::max<size_t>(
            1, std::min<size_t>(2, (228 * 1024) / (tc_smem + fa.sharedSizeBytes + 1024))));
        if (tc_smem > dyn_max) return cudaErrorInvalidValue;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(dyn_max));
        if (e != cudaSuccess) return e;
        const int grid = static_cast<int>(
            std::max<int64_t>(1, std::min<int64_t>(pts.n, static_cast<int64_t>(num_sms) * per_sm_tc)));
        kern<<<grid, tc2 ? kTc2Threads : kTcThreads, tc_smem, stream>>>(B);
        e = cudaGetLastError();
            return e;
    };
    // The CUDA-core kernel (the plain method) for any element type.
    auto launch_direct = [&](const DevPoints& pts_, int up_, const DevOutputs& out_,
                             unsigned long long* flops_) -> cudaError_t {
        CorrArgs A2 = A;
        A2.pts = pts_;
        A2.up = up_;
        A2.out = out_;
        A2.flops = flops_;
        const int per_sm = P.smem <= 100 * 1024 ? 2 : 1;
        const int64_t want = static_cast<int64_t>(num_sms) * per_sm * 8;
        const int grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(pts_.n, want)));
        switch (dtype) {
            case AR_U8: return launch_corr_t<uint8_t>(A2, P, grid, stream, fp);
            case AR_U16: return launch_corr_t<uint16_t>(A2, P, grid, stream, fp);
            case AR_I16: return launch_corr_t<int16_t>(A2, P, grid, stream, fp);
            case AR_F32: return launch_corr_t<float>(A2, P, grid, stream, fp);
            default: return cudaErrorInvalidValue;
        }
    };
    if (dtype != AR_U8 && dtype != AR_U16 && dtype != AR_I16 && dtype != AR_F32) {
        if (err) *err = "unsupported element type";
        return cudaErrorInvalidValue;
    }
    // The rotation search correlates Float32 (resampled) chips: CUDA cores for every type.
    const bool tc_ok = dtype == AR_U8 && scratch.tensor_cores && !rotating;
    // Split-BF16 tensor-core products for the other element types (by default for chips of
    // 64 px and up, where the products are a dense contraction worth the limb splitting).
    bool bf_done = false;
    const bool bf_ok = (dtype == AR_U16 || dtype == AR_I16 || dtype == AR_F32) &&
                       scratch.tensor_cores && !rotating && scratch.split_bf16 != 0 &&
                       (scratch.split_bf16 == 2 || (geom.max_ch >= 64 && geom.max_cw >= 64));
    if (bf_ok) {
        auto kern = dtype == AR_U16 ? k_corr_bf<uint16_t> : dtype == AR_I16 ? k_corr_bf<int16_t>
                                                                             : k_corr_bf<float>;
        cudaFuncAttributes fa{};
        e = cudaFuncGetAttributes(&fa, kern);
        if (e != cudaSuccess) return e;
        const size_t dyn_max = 232448 - fa.sharedSizeBytes;
        BfPlan BPl{};
        if (plan_corr_bf(geom, dyn_max, &BPl)) {
            BfArgs B{};
            B.ref = ref;
            B.sec = sec;
            B.valid = valid;
            B.nrows = nrows;
            B.ncols = ncols;
            B.pts = pts;
            B.padx = geom.padx;
            B.pady = geom.pady;
            B.up = up;
            B.measure = measure;
            B.CHM = static_cast<int>(geom.max_ch);
            B.CWM = static_cast<int>(geom.max_cw);
            B.NRM = static_cast<int>(geom.max_nr);
            B.NCM = static_cast<int>(geom.max_nc);
            B.NB = BPl.NB;
            B.BC = BPl.BC;
            B.OB = BPl.OB;
            B.LW = BPl.LW;
            B.PC = BPl.PC;
            B.NRS = BPl.NRS;
            B.AC = BPl.AC;
            B.RS = BPl.RS;
            B.VS = BPl.VS;
            B.XS = BPl.XS;
            B.off_S2 = BPl.off_S2;
            B.off_raw = BPl.off_raw;
            B.off_V = BPl.off_V;
            B.off_den = BPl.off_den;
            B.off_E = BPl.off_E;
            B.off_P = BPl.off_P;
            B.off_red = BPl.off_red;
            B.Eb = BPl.Eb;
            B.Pb = BPl.Pb;
            B.tmem_cols = BPl.tmem_cols;
            B.out = out;
            B.sub_count = scratch.sub_count;
            B.sub_point = scratch.sub_point;
            B.sub_origin = scratch.sub_origin;
            B.sub_patch = scratch.sub_patch;
            B.surf_out = surf_out;
            B.flops = A.flops;
            B.status = scratch.status;
            // 512 Tensor Memory columns: one CTA per SM, which its shared memory reserves too
            // (no CTA of another launch can wait on this one's columns).
            const size_t bf_smem = std::max<size_t>(BPl.smem, tmem_smem_floor(BPl.tmem_cols, fa.sharedSizeBytes));
            if (bf_smem > dyn_max) return cudaErrorInvalidValue;
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(dyn_max));
            if (e != cudaSuccess) return e;
            const int bgrid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(pts.n, num_sms)));
            kern<<<bgrid, kBfThreads, bf_smem, stream>>>(B);
            e = cudaGetLastError();
            bf_done = true;
        }
    }
    if (!bf_done) {
        // UInt8: the three kernels are exact and give identical results; the tensor-core kernel
        // whose plan fits runs, k_corr_tc2 before k_corr_tc. Over chips of 4 to 80 px, radii of 2
        // to 32 and consecutive or scattered points, k_corr_tc2 took 0.37 to 0.85 of k_corr_tc's
        // time and at most 0.90 of k_corr's (chip 4, radius 2); where only k_corr_tc fits
        // (chips of 96 and 128 px, surfaces beyond 64 x 64) it took 0.40 of k_corr's at most. On a
        // pass of radii 4 to 32 the two tie (73 523 points at chip 16: 3.9 ms).
        TcPlan TP2{}, TP1{};
        const bool fit2 = tc_ok && plan_corr_tc2(geom, 220 * 1024, &TP2);
        const bool fit1 = tc_ok && plan_corr_tc(geom, 220 * 1024, pts.n > num_sms, &TP1);
        int kind = fit2 ? 2 : fit1 ? 1 : 0;
        const int force = scratch.uint8_kernel;
        if (force == 0 || (force == 1 && fit1) || (force == 2 && fit2)) kind = force;
        if (force < 0 && (fit2 || fit1) && scratch.autotune && !scratch.fixed &&
            pts.n >= kTuneMinPoints) {
            const uint64_t key = (static_cast<uint64_t>(geom.max_ch) << 48) |
                                 (static_cast<uint64_t>(geom.max_cw) << 32) |
                                 (static_cast<uint64_t>(geom.max_nr) << 16) |
                                 static_cast<uint64_t>(geom.max_nc);
            scratch.tuned[key] = kind;
        }
        if (kind == 2) {
            e = launch_tc(true, TP2, pts, up, out, A.flops);
        } else if (kind == 1) {
            e = launch_tc(false, TP1, pts, up, out, A.flops);
        } else {
            e = launch_direct(pts, up, out, A.flops);
        }
    }
    if (e != cudaSuccess) return e;
    T.launches += 1;
    if (T.enabled) cudaEventRecord(ev1, stream);
    if (up == 1) {
        if (T.enabled) {
            cudaEventRecord(ev2, stream);
            T.recs.push_back({ev0, ev1, ev2});
        }
        return cudaSuccess;
    }

    const RefinePlan R = plan_refine(up);
    RefineArgs B{};
    B.count = scratch.sub_count;
    B.n_items = 0;
    B.point = scratch.sub_point;
    B.origin = scratch.sub_origin;
    B.patch = scratch.sub_patch;
    B.pts = pts;
    B.out = out;
    B.levels = R.levels;
    B.warp_floats = R.warp_floats;
    e = launch_refine(R, B, pts.n, num_sms, stream);
    if (e != cudaSuccess) return e;
    T.launches += 1;
    if (T.enabled) {
        cudaEventRecord(ev2, stream);
        T.recs.push_back({ev0, ev1, ev2});
    }
    return e;
}

cudaError_t launch_track(int dtype, const void* ref, const void* sec, const uint8_t* valid,
                         int64_t nrows, int64_t ncols, const DevPoints& pts,
                         const PassGeometry& geom, int up, int measure, const DevOutputs& out,
                         TrackScratch& scratch, int num_sms, cudaStream_t stream,
                         std::string* err, float* surf_out, const Rotation* rot) {
    cudaError_t e = scratch_acquire(scratch, stream);
    if (e != cudaSuccess) return e;
    e = launch_track_impl(dtype, ref, sec, valid, nrows, ncols, pts, geom, up, measure, out,
                          scratch, num_sms, stream, err, surf_out, rot);
    const cudaError_t r = scratch.done ? cudaEventRecord(scratch.done, stream) : cudaSuccess;
    return e != cudaSuccess ? e : r;
}

cudaError_t launch_refine_patches(const float* patches, int64_t count, int up, int32_t* row,
                                  int32_t* col, float* value, int num_sms, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    const RefinePlan R = plan_refine(up);
    RefineArgs B{};
    B.count = nullptr;
    B.n_items = count;
    B.point = nullptr;
    B.origin = nullptr;
    B.patch = patches;
    B.orow = row;
    B.ocol = col;
    B.oval = value;
    B.levels = R.levels;
    B.warp_floats = R.warp_floats;
    return launch_refine(R, B, count, num_sms, stream);
}

}  // namespace ar

// ---------------------------------------------------------------------------------------------
// Allocation-free track entry point.
//
// Some callers cannot allocate device memory at the time they correlate: a host that owns the
// whole device pool and hands out only the buffers it planned (an embedded or real-time
// service with a fixed memory budget), code running under another framework's allocator, or
// a caller that must not trigger cudaMalloc's implicit device synchronisation in the middle
// of a pipeline. For them the track pass can run with its scratch -- the refinement queue and
// the pass-geometry words -- in a fixed array in this file instead of context-owned buffers.
//
// The array is sized for kStaticMaxPoints points per call (about 3.8 MB, held by every GPU
// that loads the library until the process exits). Calls share it and it keeps the last
// call's contents; the queue counter and the geometry words are reset by every call before
// use, and so is the status word a bounded tensor-core wait sets when it runs out. Two calls
// that overlap on the GPU (different streams, or different host threads) race on it and must
// not be issued.

namespace ar {
namespace {

constexpr int64_t kStaticMaxPoints = 32768;
constexpr size_t kStaticGeomOff = 0;                                   // 8 x int64
constexpr size_t kStaticCountOff = 64;                                 // int
constexpr size_t kStaticStatusOff = 128;                               // int
constexpr size_t kStaticPointOff = 256;                                // int64 per point
constexpr size_t kStaticOriginOff = kStaticPointOff + 8 * kStaticMaxPoints;   // 2 x int32
constexpr size_t kStaticPatchOff = kStaticOriginOff + 8 * kStaticMaxPoints;   // 25 x float
constexpr size_t kStaticBytes = kStaticPatchOff + 100 * kStaticMaxPoints;

static __device__ __align__(256) unsigned char g_static_scratch[kStaticBytes];

constexpr int kStaticMaxDevices = 64;
std::mutex g_static_mu;
unsigned char* g_static_addr[kStaticMaxDevices] = {};

// The device address of g_static_scratch on the current device, looked up once per device.
cudaError_t static_scratch(unsigned char** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kStaticMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess) return e;
        g_static_addr[dev] = static_cast<unsigned char*>(p);
    }
    *out = g_static_addr[dev];
    return cudaSuccess;
}

void static_message(char* buf, size_t size, const char* msg) {
    if (!buf || size == 0) return;
    size_t n = 0;
    while (msg[n] && n + 1 < size) {
        buf[n] = msg[n];
        ++n;
    }
    buf[n] = '\0';
}

}  // namespace
}  // namespace ar

extern "C" int ar_track_device_static(const void* ref, const void* sec, const uint8_t* valid,
                                      int64_t nrows, int64_t ncols, int dtype,
                                      const ar_points* pts, int upsampling, int measure,
                                      float* dx, float* dy, float* correlation,
                                      uint8_t* searched, void* stream, char* err,
                                      size_t err_size) {
    using namespace ar;
    if (!ref || !sec || !valid || !pts || nrows <= 0 || ncols <= 0) {
        static_message(err, err_size, "null or empty input");
        return AR_ERR_ARG;
    }
    if (pts->n < 0 || pts->n > kStaticMaxPoints) {
        static_message(err, err_size,
                       "point count outside [0, 32768], the capacity of the static scratch; "
                       "split the point set or use ar_track_device");
        return AR_ERR_SIZE;
    }
    if (pts->n > 0 && (!dx || !dy || !correlation || !searched || !pts->x || !pts->y ||
                       !pts->radius_x || !pts->radius_y || !pts->dx_prior || !pts->dy_prior ||
                       !pts->chip_size_x || !pts->chip_size_y)) {
        static_message(err, err_size, "null point-set field or output");
        return AR_ERR_ARG;
    }
    if (upsampling < 1 || upsampling > 128 || (upsampling & (upsampling - 1))) {
        static_message(err, err_size, "`upsampling` must be 1 or a power of 2 up to 128");
        return AR_ERR_ARG;
    }
    if (measure != AR_ZNCC && measure != AR_NCC) {
        static_message(err, err_size, "unknown measure");
        return AR_ERR_ARG;
    }
    if (dtype != AR_U8 && dtype != AR_U16 && dtype != AR_I16 && dtype != AR_F32) {
        static_message(err, err_size, "unsupported element type");
        return AR_ERR_UNSUPPORTED;
    }
    if (pts->n == 0) return AR_OK;
    unsigned char* base = nullptr;
    cudaError_t e = static_scratch(&base);
    if (e != cudaSuccess) {
        static_message(err, err_size, cudaGetErrorString(e));
        return AR_ERR_CUDA;
    }
    // A view of the static array in the scratch layout the track launch expects. Its capacity
    // covers the call, so the launch allocates nothing; timing stays off (no events).
    TrackScratch view;
    view.geom = reinterpret_cast<int64_t*>(base + kStaticGeomOff);
    view.sub_count = reinterpret_cast<int*>(base + kStaticCountOff);
    view.sub_point = reinterpret_cast<int64_t*>(base + kStaticPointOff);
    view.sub_origin = reinterpret_cast<int32_t*>(base + kStaticOriginOff);
    view.sub_patch = reinterpret_cast<float*>(base + kStaticPatchOff);
    view.status = reinterpret_cast<int*>(base + kStaticStatusOff);
    view.capacity = kStaticMaxPoints;
    view.fixed = true;  // the launch helpers then neither allocate nor create events
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    e = cudaMemsetAsync(view.status, 0, sizeof(int), s);
    if (e != cudaSuccess) {
        static_message(err, err_size, cudaGetErrorString(e));
        return AR_ERR_CUDA;
    }
    DevPoints dp{pts->x, pts->y, pts->radius_x, pts->radius_y, pts->dx_prior, pts->dy_prior,
                 pts->chip_size_x, pts->chip_size_y, pts->n};
    PassGeometry geom;
    e = pass_geometry_device(dp, nrows, ncols, view, s, &geom);
    int num_sms = 148;
    int dev = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    std::string msg;
    DevOutputs out{dx, dy, correlation, searched};
    if (e == cudaSuccess)
        e = launch_track(dtype, ref, sec, valid, nrows, ncols, dp, geom, upsampling, measure, out,
                         view, num_sms, s, &msg);
    if (e != cudaSuccess) {
        static_message(err, err_size, msg.empty() ? cudaGetErrorString(e) : msg.c_str());
        return msg.empty() ? AR_ERR_CUDA : AR_ERR_UNSUPPORTED;
    }
    // Wait for the pass and read its status word: a bounded tensor-core wait that ran out
    // leaves the outputs incomplete, which the caller must learn of.
    int status = 0;
    e = cudaMemcpyAsync(&status, view.status, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        static_message(err, err_size, cudaGetErrorString(e));
        return AR_ERR_CUDA;
    }
    if (status) {
        static_message(err, err_size, "a device wait ran out; results incomplete");
        return AR_ERR_TIMEOUT;
    }
    return AR_OK;
}

extern "C" int ar_scratch_allocations(int64_t* count) {
    if (!count) return AR_ERR_ARG;
    *count = ar::scratch_allocations();
    return AR_OK;
}

#ifdef AR_TC_PHASES
// Profiling builds only: the phase counters of k_corr_tc (16 entries), then cleared.
extern "C" int ar_tc_phase_read(unsigned long long* out) {
    cudaDeviceSynchronize();
    if (cudaMemcpyFromSymbol(out, ar::g_tc_phase, 16 * sizeof(unsigned long long)) != cudaSuccess)
        return 1;
    const unsigned long long z[16] = {};
    return cudaMemcpyToSymbol(ar::g_tc_phase, z, sizeof(z)) == cudaSuccess ? 0 : 1;
}
#endif
