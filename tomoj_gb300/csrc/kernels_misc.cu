// Supporting kernels: per-tilt alignment resample, WBP row filter (batched FFT),
// deterministic residual reductions, TV denoise stencils, FISTA momentum, fills
// and the long-object normalisation.  The library is compiled with -fmad=false,
// so every a*b+c here rounds twice like the Java reference unless fmaf is used.
#include <cmath>

#include "device_util.cuh"
#include "tomo_internal.h"

namespace tomo {
namespace {

// AffineAlignment.applyTransformOnImage (TomoJ_Base/.../align/AffineAlignment.java:136-259):
// inverse-map every output pixel through Tinv around (w/2, h/2), Java (int) truncation,
// bilinear in double with the floor pixel on the last row/column, optional
// (x - mean) / stdDev, and the TiltSeries fill policy outside the image.

// One pixel in the reference's double expressions (pix before normalisation; false: outside).
__device__ __noinline__ bool align_pixel_exact(const float* __restrict__ un, const double* __restrict__ T, int i, int j,
                                               int w, int h, float* pix) {
    // T: {i00, i10, i01, i11, i02, i12}
    const double cx = w / 2.0, cy = h / 2.0;
    const double px = (double)i - cx, jc = (double)j - cy;
    const double xx = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(T[0], px), __dmul_rn(T[2], jc)), T[4]), cx);
    const double yy = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(T[1], px), __dmul_rn(T[3], jc)), T[5]), cy);
    const int ix0 = __double2int_rz(xx), iy0 = __double2int_rz(yy);
    const double dx0 = __dsub_rn(xx, (double)ix0), dy0 = __dsub_rn(yy, (double)iy0);
    if (ix0 < 0 || ix0 >= w || iy0 < 0 || iy0 >= h) return false;
    if (ix0 == w - 1 || iy0 == h - 1) {
        *pix = un[ix0 + (size_t)iy0 * w];
        return true;
    }
    const double fac4 = __dmul_rn(dx0, dy0);
    const size_t pos = ix0 + (size_t)iy0 * w;
    const double v1 = un[pos], v3 = un[pos + w], v2 = un[pos + 1], v4 = un[pos + 1 + w];
    const double w1 = __dadd_rn(__dsub_rn(__dsub_rn(1.0, dx0), dy0), fac4);
    const double acc = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(v1, w1), __dmul_rn(v2, __dsub_rn(dx0, fac4))),
                                           __dmul_rn(v3, __dsub_rn(dy0, fac4))),
                                 __dmul_rn(v4, fac4));
    *pix = __double2float_rn(acc);
    return true;
}

// Pairs of floats (hi + lo, about 48 bits): a + t (b - a) for float or pair a, b and pair t.
struct FPair {
    float hi, lo;
};
__device__ __forceinline__ FPair pair_sum(float a, float b) {
    const float s = a + b, u = s - a;
    return FPair{s, (a - (s - u)) + (b - u)};
}
__device__ __forceinline__ FPair pair_lerp(FPair a, FPair b, FPair t) {
    FPair d = pair_sum(b.hi, -a.hi);
    d.lo += b.lo - a.lo;
    const float p = t.hi * d.hi;
    const float e = fmaf(t.hi, d.hi, -p) + (t.hi * d.lo + t.lo * d.hi);
    FPair r = pair_sum(a.hi, p);
    r.lo += a.lo + e;
    return r;
}

// One pixel from 64-bit fixed-point coordinates (known to 2^-47 pixel: steps of 2^-64, so that
// thousands of columns and rows add nothing; the double expressions round to 2^-40 at x = 4096) and
// bilinear weights and sums in pairs of floats (a few parts in 2^46 of the largest neighbour),
// rounded once at the end.  F: whole parts in units of 2^-48, then the rest in units of 2^-64.
// 0: outside, 1: *pix set, 2: not decided here (a coordinate within 2^-20 of a whole
// pixel, where truncation is the reference's double rounding's, or neighbours that are not
// finite, or so large or small that a pair would lose bits).
__device__ __forceinline__ int align_pixel_fixed(const float* __restrict__ un, const long long* __restrict__ F, int md,
                                                 int i, int j, int w, int h, float* pix) {
    // (rests below 2^16, columns + rows at most 2^16: the sum fits 32 bits)
    auto rest = [&](int k) { return ((unsigned)F[6 + k] * i + (unsigned)F[8 + k] * j + (unsigned)F[10 + k]) >> 16; };
    const long long X = F[0] * i + F[2] * j + F[4] + rest(0), Y = F[1] * i + F[3] * j + F[5] + rest(1);
    constexpr long long kOne = 1LL << 48, kNear = 1LL << 28;
    const long long nx = md & 4 ? 0 : kNear, ny = md & 8 ? 0 : kNear;
    if (((X + nx) & (kOne - 1)) < 2 * nx || ((Y + ny) & (kOne - 1)) < 2 * ny) return 2;
    // truncation toward zero: a coordinate in (-1, 0) takes pixel 0 with a negative fraction
    const int ix = X >= 0 ? (int)(X >> 48) : -(int)(-X >> 48), iy = Y >= 0 ? (int)(Y >> 48) : -(int)(-Y >> 48);
    if (ix < 0 || ix >= w || iy < 0 || iy >= h) return 0;
    const size_t pos = ix + (size_t)iy * w;
    const float v1 = un[pos];
    if (ix == w - 1 || iy == h - 1) {
        *pix = v1;
        return 1;
    }
    const float v2 = un[pos + 1], v3 = un[pos + w], v4 = un[pos + 1 + w];
    const float mag = fabsf(v1) + fabsf(v2) + fabsf(v3) + fabsf(v4);
    if (!(mag < 1e38f) || (mag > 0.0f && mag < 1e-30f)) return 2;
    auto frac = [](long long f) {  // |f| < 2^48: both parts are exact
        return FPair{(float)(int)(f >> 24) * (1.0f / 16777216.0f),
                     (float)(unsigned)(f & 0xFFFFFF) * (1.0f / 16777216.0f / 16777216.0f)};
    };
    const FPair dx = frac(X - ((long long)ix << 48)), dy = frac(Y - ((long long)iy << 48));
    const FPair top = pair_lerp(FPair{v1, 0.0f}, FPair{v2, 0.0f}, dx);
    const FPair bot = pair_lerp(FPair{v3, 0.0f}, FPair{v4, 0.0f}, dx);
    const FPair r = pair_lerp(top, bot, dy);
    *pix = r.hi + r.lo;
    return 1;
}

// mode per image: 0 double expressions, 1 identity, 2 fixed-point coordinates (fix: {x, y per
// column, x, y per row, x, y at pixel (0, 0)} in two parts, see align_pixel_fixed) with + 4 and + 8 where x and y are
// exact in both forms (whole or dyadic shifts).  flags: bit 0 a NaN was written, bit 1 an
// infinity, bit 2 set where a pixel took the fill.  This part's FP64 rate is 1/64 of FP32: 61 images of 512 x 256 took 628
// us in doubles and take 69 us in fixed point and float pairs, with the scan for
// non-finite pixels (9 us) in the same pass (66 us without the steps' second parts).
constexpr int kAlignPix = 4;  // pixels per thread

__global__ void __launch_bounds__(256) align_kernel(const float* __restrict__ raw, float* __restrict__ out,
                                                    const double* __restrict__ tinv, const long long* __restrict__ fix,
                                                    const double* __restrict__ stats, int w, int h, int normalize,
                                                    int fill, const unsigned char* __restrict__ mode, int* flags) {
    const int t = blockIdx.y;
    const size_t npix = (size_t)w * h;
    const float* un = raw + t * npix;
    float* dst = out + t * npix;
    const int md = mode[t];
    const double mean = stats ? stats[2 * t] : 0.0;
    const double sd = stats ? stats[2 * t + 1] : 1.0;
    const float outside = fill == 1 ? (normalize ? 0.0f : __double2float_rn(mean))
                          : fill == 2 ? __int_as_float(0x7fc00000) : 0.0f;
    int f = 0;
#pragma unroll
    for (int q = 0; q < kAlignPix; q++) {
        const size_t e = ((size_t)blockIdx.x * kAlignPix + q) * 256 + threadIdx.x;
        if (e >= npix) break;
        float pix;
        bool in = true;
        if (md == 1) {
            pix = un[e];
        } else {
            const int j = e >> 32 ? (int)(e / w) : (int)((unsigned)e / (unsigned)w), i = (int)(e - (size_t)j * w);
            int st = 2;
            if (md & 2) st = align_pixel_fixed(un, fix + 12 * t, md, i, j, w, h, &pix);
            if (st == 2) in = align_pixel_exact(un, tinv + 6 * t, i, j, w, h, &pix);
            else in = st == 1;
        }
        if (!in) {
            pix = outside;
            f |= 4;
        } else if (normalize) {
            pix = __double2float_rn(__ddiv_rn(__dsub_rn((double)pix, mean), sd));
        }
        dst[e] = pix;
        if (isnan(pix)) f |= 1;
        else if (isinf(pix)) f |= 2;
    }
    f = __reduce_or_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0 && f) atomicOr(flags, f);
}

// --- WBP row filter --------------------------------------------------------------
// FFTWeighting.weighting (FFTWeighting.java:87-112) multiplies the 2-D spectrum by
// a mask that, for a zero tilt-axis angle, depends on the column frequency only;
// the 2-D filter is then exactly a filter of every row.  Two real rows are packed
// into one complex sequence (the mask is real and even, so the packed halves
// stay separate), transformed, multiplied by the mask, transformed back and scaled.
//
// Any width: the filter is a circular convolution of length w with the real kernel
// h = IDFT_w(mask).  A row is laid out twice ([row, row], the periodic extension) in a
// zero-padded sequence of M >= 2w - 1 points; the linear convolution with h (spectrum H,
// M points) equals the circular one on outputs [w, 2w).
//
// One CTA per pair of rows; in-place passes of radix 8 (the first of 2, 4 or 8) over one
// padded buffer in shared memory: decimation in frequency down to groups of 8 points,
// which are transformed, multiplied by the spectrum (stored in the order the passes leave
// it, fft_slot_frequency; twiddles in the order of use, fft_pass_twiddles) and transformed back in registers, then decimation in time back
// up.  The first pass reads the image and the last one writes it, so M = 2048 crosses
// shared memory 6 times each way and nothing is reordered; radix-2 stages with
// bit-reversed copies crossed it 24 times.  Bound by shared memory and FP32 issue, about
// evenly.  73 images of 750 x 333 (M = 2048): 881 -> 184 us; 61 of 512 x 256 (M = 512):
// 121 -> 23 us (284 and 29 us with the twiddles gathered from one table by stride).
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 caddf(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csubf(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a * (-i) (forward) or a * i (inverse)
template <bool INV>
__device__ __forceinline__ float2 quarter(float2 a) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// R-point transform in registers, outputs in natural order.
template <int R, bool INV>
__device__ __forceinline__ void fft_points(float2* v) {
    if constexpr (R == 2) {
        const float2 d = csubf(v[0], v[1]);
        v[0] = caddf(v[0], v[1]);
        v[1] = d;
    } else if constexpr (R == 4) {
        const float2 a = caddf(v[0], v[2]), b = csubf(v[0], v[2]);
        const float2 c = caddf(v[1], v[3]), d = quarter<INV>(csubf(v[1], v[3]));
        v[0] = caddf(a, c);
        v[1] = caddf(b, d);
        v[2] = csubf(a, c);
        v[3] = csubf(b, d);
    } else if constexpr (R == 8) {
        float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        fft_points<4, INV>(e);
        fft_points<4, INV>(o);
        const float r = 0.70710678118654752f;
        const float2 q1 = quarter<INV>(o[1]), q3 = quarter<INV>(o[3]);
        o[1] = make_float2(r * (o[1].x + q1.x), r * (o[1].y + q1.y));
        o[2] = quarter<INV>(o[2]);
        o[3] = make_float2(r * (q3.x - o[3].x), r * (q3.y - o[3].y));
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = caddf(e[k], o[k]);
            v[k + 4] = csubf(e[k], o[k]);
        }
    }
}

// Shared-memory place of point i: one spare place per 8 points keeps the accesses of a pass
// with stride 1, 8 or >= 64 on different banks.
__device__ __forceinline__ int fft_pad(int i) { return i + (i >> 3); }

// One pass over groups of 2^logL points (sub-transforms of R points, stride 2^logL / R) of
// an M-point sequence: load(i) and store(i, v) read and write point i.  Forward: transform,
// then twiddles; inverse: twiddles, then transform.
template <int R, bool INV, class Load, class Store>
__device__ __forceinline__ void fft_pass(const float2* __restrict__ tw, int logM, int logL, Load load, Store store) {
    constexpr int kLogR = R == 8 ? 3 : R == 4 ? 2 : R == 2 ? 1 : 0;
    const int logS = logL - kLogR, cnt = 1 << (logM - kLogR);
    for (int b = threadIdx.x; b < cnt; b += blockDim.x) {
        const int k = b & ((1 << logS) - 1), i0 = ((b >> logS) << logL) + k;
        float2 v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = load(i0 + (m << logS));
        if (!INV) fft_points<R, INV>(v);
#pragma unroll
        for (int m = 1; m < R; m++) {
            float2 t = tw[(1 << logM) - (1 << logL) + ((m - 1) << logS) + k];
            if (INV) t.y = -t.y;
            v[m] = cmulf(v[m], t);
        }
        if (INV) fft_points<R, INV>(v);
#pragma unroll
        for (int m = 0; m < R; m++) store(i0 + (m << logS), v[m]);
    }
}

// The groups of R contiguous points in between: transform, spectrum, inverse transform.
template <int R, class Load, class Store, class Spec>
__device__ __forceinline__ void fft_middle(int logM, Load load, Store store, Spec spec) {
    constexpr int kLogR = R == 8 ? 3 : R == 4 ? 2 : R == 2 ? 1 : 0;
    for (int b = threadIdx.x; b < 1 << (logM - kLogR); b += blockDim.x) {
        float2 v[R];
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = load(b * R + m);
        fft_points<R, false>(v);
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = spec(b * R + m, v[m]);
        fft_points<R, true>(v);
#pragma unroll
        for (int m = 0; m < R; m++) store(b * R + m, v[m]);
    }
}

// in(i): point i of the packed rows; out(i, v): point i of the filtered sequence times M.
template <class In, class Out, class Spec>
__device__ __forceinline__ void fft_filter(float2* s, const float2* __restrict__ tw, int logM, In in, Out out, Spec spec) {
    auto ld = [s](int i) { return s[fft_pad(i)]; };
    auto st = [s](int i, float2 v) { s[fft_pad(i)] = v; };
    if (logM <= 3) {  // one group
        if (logM == 3) fft_middle<8>(logM, in, out, spec);
        else if (logM == 2) fft_middle<4>(logM, in, out, spec);
        else if (logM == 1) fft_middle<2>(logM, in, out, spec);
        else fft_middle<1>(logM, in, out, spec);
        return;
    }
    const int first = logM % 3;
    if (first == 1) fft_pass<2, false>(tw, logM, logM, in, st);
    else if (first == 2) fft_pass<4, false>(tw, logM, logM, in, st);
    else fft_pass<8, false>(tw, logM, logM, in, st);
    const int top = logM - (first ? first : 3);
    for (int l = top; l > 3; l -= 3) {
        __syncthreads();
        fft_pass<8, false>(tw, logM, l, ld, st);
    }
    __syncthreads();
    fft_middle<8>(logM, ld, st, spec);
    for (int l = 6; l <= top; l += 3) {
        __syncthreads();
        fft_pass<8, true>(tw, logM, l, ld, st);
    }
    __syncthreads();
    if (first == 1) fft_pass<2, true>(tw, logM, logM, ld, out);
    else if (first == 2) fft_pass<4, true>(tw, logM, logM, ld, out);
    else fft_pass<8, true>(tw, logM, logM, ld, out);
}

// bad (optional): per-image flag of a non-finite pixel.  The reference's 2-D transform
// spreads one NaN or Inf over the whole image; a row filter alone would keep it in
// its row, so rows of a flagged image are written as NaN.
__device__ __forceinline__ bool image_bad(const int* bad, int row, int rows_per_img) {
    return bad != nullptr && bad[row / rows_per_img] != 0;
}

// Row of the source of filtered row r: img itself, or the row of image pick[r / rows_per_img] of src.
__device__ __forceinline__ const float* source_row(const float* img, const float* src, const int* pick, int r, int w,
                                                   int rows_per_img) {
    if (!src) return img + (size_t)r * w;
    const int t = r / rows_per_img;
    return src + ((size_t)pick[t] * rows_per_img + (r - t * rows_per_img)) * w;
}

__global__ void __launch_bounds__(512) row_filter_kernel(float* img, const float* src, const int* pick,
                                                         const float* __restrict__ mask, const float2* __restrict__ tw,
                                                         int rows, int n, int logn, const int* __restrict__ bad,
                                                         int rows_per_img) {
    extern __shared__ float2 sbuf[];
    const int r0 = 2 * blockIdx.x, r1 = r0 + 1;
    float* row0 = img + (size_t)r0 * n;
    float* row1 = (r1 < rows) ? img + (size_t)r1 * n : nullptr;
    const float* in0 = source_row(img, src, pick, r0, n, rows_per_img);
    const float* in1 = row1 ? source_row(img, src, pick, r1, n, rows_per_img) : nullptr;
    const float inv = 1.0f / (float)n;
    const bool bad0 = image_bad(bad, r0, rows_per_img), bad1 = row1 && image_bad(bad, r1, rows_per_img);
    fft_filter(
        sbuf, tw, logn, [=](int i) { return make_float2(in0[i], in1 ? in1[i] : 0.0f); },
        [=](int i, float2 v) {
            row0[i] = bad0 ? __int_as_float(0x7fc00000) : v.x * inv;
            if (row1) row1[i] = bad1 ? __int_as_float(0x7fc00000) : v.y * inv;
        },
        [=](int i, float2 v) { return make_float2(v.x * mask[i], v.y * mask[i]); });
}

__global__ void __launch_bounds__(512) row_filter_conv_kernel(float* img, const float* src, const int* pick,
                                                              const float2* __restrict__ H,
                                                              const float2* __restrict__ tw, int rows, int w, int M,
                                                              int logM, const int* __restrict__ bad, int rows_per_img) {
    extern __shared__ float2 sbuf[];
    const int r0 = 2 * blockIdx.x, r1 = r0 + 1;
    float* row0 = img + (size_t)r0 * w;
    float* row1 = (r1 < rows) ? img + (size_t)r1 * w : nullptr;
    const float* in0 = source_row(img, src, pick, r0, w, rows_per_img);
    const float* in1 = row1 ? source_row(img, src, pick, r1, w, rows_per_img) : nullptr;
    const float inv = 1.0f / (float)M;
    const bool bad0 = image_bad(bad, r0, rows_per_img), bad1 = row1 && image_bad(bad, r1, rows_per_img);
    fft_filter(
        sbuf, tw, logM,
        [=](int i) {
            if (i >= 2 * w) return make_float2(0.0f, 0.0f);
            const int m = i < w ? i : i - w;
            return make_float2(in0[m], in1 ? in1[m] : 0.0f);
        },
        [=](int i, float2 v) {
            const int k = i - w;
            if (k < 0 || k >= w) return;
            row0[k] = bad0 ? __int_as_float(0x7fc00000) : v.x * inv;
            if (row1) row1[k] = bad1 ? __int_as_float(0x7fc00000) : v.y * inv;
        },
        [=](int i, float2 v) { return cmulf(v, H[i]); });
}

// --- 2-D weighting (tilt axis not vertical) ----------------------------------------
// FFTWeighting.weighting (FFTWeighting.java:87-112) with a mask that depends on both
// frequencies: forward DFT of every row, transpose, per column (now a row) forward
// DFT, multiply by the mask, inverse DFT, transpose back, inverse DFT of every row,
// real part scaled by 1/(w h).  Each transform runs in shared memory: radix-2 when
// the length is a power of two, otherwise Bluestein's chirp-z algorithm on a radix-2
// grid of M >= 2n - 1 points:
//   X[k] = c[k] * sum_j (x[j] c[j]) conj(c[k - j]),  c[j] = exp(-i pi j^2 / n),
// the convolution done by an M-point FFT with the precomputed spectrum of the
// wrapped conj(c).  Inverse transforms are conj(DFT(conj(x))).
__device__ __forceinline__ unsigned bitrev(unsigned v, int bits) { return __brev(v) >> (32 - bits); }

__device__ void fft_stages(float2* s, const float2* __restrict__ tw, int n, int logn, bool inverse) {
    for (int len = 2, stage = 0; len <= n; len <<= 1, stage++) {
        const int half = len >> 1;
        const int tstride = n / len;
        __syncthreads();
        for (int b = threadIdx.x; b < n / 2; b += blockDim.x) {
            const int grp = b / half, k = b % half;
            const int ia = grp * len + k, ib = ia + half;
            float2 wv = tw[k * tstride];
            if (inverse) wv.y = -wv.y;
            const float2 xb = s[ib], xa = s[ia];
            const float2 t = make_float2(xb.x * wv.x - xb.y * wv.y, xb.x * wv.y + xb.y * wv.x);
            s[ib] = make_float2(xa.x - t.x, xa.y - t.y);
            s[ia] = make_float2(xa.x + t.x, xa.y + t.y);
        }
    }
    __syncthreads();
}

// Forward DFT (conjugated on input and output when conj_io: the inverse) of x[0, n)
// in shared memory, in place; a and b are M-point work buffers.
__device__ void dft_row(float2* x, float2* a, float2* b, const DftRowPlan& P, bool conj_io) {
    const int n = P.n, M = P.M, logM = P.logM;
    const float cs = conj_io ? -1.0f : 1.0f;
    if (M == n) {
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            const float2 v = x[k];
            a[bitrev(k, logM)] = make_float2(v.x, cs * v.y);
        }
        fft_stages(a, P.tw, M, logM, false);
        for (int k = threadIdx.x; k < n; k += blockDim.x) x[k] = make_float2(a[k].x, cs * a[k].y);
        __syncthreads();
        return;
    }
    for (int k = threadIdx.x; k < M; k += blockDim.x) {
        float2 v = make_float2(0.0f, 0.0f);
        if (k < n) v = cmulf(make_float2(x[k].x, cs * x[k].y), P.chirp[k]);
        a[bitrev(k, logM)] = v;
    }
    fft_stages(a, P.tw, M, logM, false);
    for (int k = threadIdx.x; k < M; k += blockDim.x) b[bitrev(k, logM)] = cmulf(a[k], P.bspec[k]);
    fft_stages(b, P.tw, M, logM, true);
    const float inv = 1.0f / (float)M;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const float2 v = cmulf(b[k], P.chirp[k]);
        x[k] = make_float2(v.x * inv, cs * v.y * inv);
    }
    __syncthreads();
}

// MODE 0: real rows -> spectra; 1: spectra x mask row (row index mod mask_rows),
// inverse; 2: spectra -> real rows (real part x scale).  One row per CTA.
template <int MODE>
__global__ void dft2_rows_kernel(const float* __restrict__ rin, float2* cio, float* rout, const float* __restrict__ mask,
                                 DftRowPlan P, int mask_rows, float scale) {
    extern __shared__ float2 sbuf[];
    float2* x = sbuf;
    float2* a = sbuf + P.n;
    float2* b = a + P.M;
    const size_t r = blockIdx.x;
    const int n = P.n;
    for (int k = threadIdx.x; k < n; k += blockDim.x)
        x[k] = MODE == 0 ? make_float2(rin[r * n + k], 0.0f) : cio[r * n + k];
    __syncthreads();
    dft_row(x, a, b, P, MODE == 2);
    if (MODE == 1) {
        const float* m = mask + (size_t)(r % (size_t)mask_rows) * n;
        for (int k = threadIdx.x; k < n; k += blockDim.x) x[k] = make_float2(x[k].x * m[k], x[k].y * m[k]);
        __syncthreads();
        dft_row(x, a, b, P, true);
    }
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        if (MODE == 2)
            rout[r * n + k] = x[k].x * scale;
        else
            cio[r * n + k] = x[k];
    }
}

// [T][R][C] -> [T][C][R], 32 x 32 tiles.
__global__ void transpose_c_kernel(const float2* __restrict__ in, float2* __restrict__ out, int R, int Cc) {
    __shared__ float2 tile[32][33];
    const size_t base = (size_t)blockIdx.z * R * Cc;
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
        const int r = r0 + dy, c = c0 + threadIdx.x;
        if (r < R && c < Cc) tile[dy][threadIdx.x] = in[base + (size_t)r * Cc + c];
    }
    __syncthreads();
    for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
        const int c = c0 + dy, r = r0 + threadIdx.x;
        if (r < R && c < Cc) out[base + (size_t)c * R + r] = tile[threadIdx.x][dy];
    }
}

// bad[t] = 1 when image t holds a NaN or an Inf.
__global__ void image_nonfinite_kernel(const float* __restrict__ imgs, size_t npix, int* bad) {
    const float* im = imgs + (size_t)blockIdx.y * npix;
    int f = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < npix; i += (size_t)gridDim.x * blockDim.x)
        f |= !isfinite(im[i]);
    f = __reduce_or_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0 && f) atomicOr(bad + blockIdx.y, 1);
}

// Sum over rows of the per-row residuals, one thread per tilt, fixed order.
// Sum of one projection's per-row residual sums by one warp: lane l adds rows
// l, l + 32, ... in order, then a fixed butterfly combines the lanes (deterministic).
__device__ __forceinline__ double warp_row_sum(const double* __restrict__ rows, int h) {
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    for (int j = lane; j < h; j += 32) s += rows[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

constexpr int kErrWarps = 4;  // projections per 128-thread block

__global__ void reduce_err_kernel(const double* __restrict__ errpart, double* __restrict__ err, int T, int h) {
    const int t = blockIdx.x * kErrWarps + (threadIdx.x >> 5);
    if (t >= T) return;
    const double s = warp_row_sum(errpart + (size_t)t * h, h);
    if ((threadIdx.x & 31) == 0) err[t] = s;
}

__global__ void reduce_err_batch_kernel(const ErrReduce* __restrict__ jobs) {
    const ErrReduce j = jobs[blockIdx.y];
    const int t = blockIdx.x * kErrWarps + (threadIdx.x >> 5);
    if (t >= j.T) return;
    const double s = warp_row_sum(j.errpart + (size_t)t * j.h, j.h);
    if ((threadIdx.x & 31) == 0) j.err[t] = s;
}

// TotalVariationDenoising_3D (Filters/.../TotalVariationDenoising_3D.java:84-202): inner
// steps of updateP (:115-156) then updateU (:158-202), fused.  The step k -> k + 1 needs
// u_k = f - theta * div p_k only where updateP reads it (the voxel and its +x, +y, +z
// neighbours), so one kernel rebuilds u_k plane by plane in shared memory from p_k and f
// and writes p_{k+1}; u itself is never stored between steps.  p is double-buffered
// (a CTA reads p_k of its -x / -y / -z neighbours while others write p_{k+1}).  Every
// value is computed with updateU's and updateP's float expressions in their order, so
// the result is the unfused sequence's bit for bit.

// u = f - theta * div p at flat index o = (z, y, x), with updateU's boundary rules.
__device__ __forceinline__ float tv_u_point(const float* f, const float* __restrict__ px, const float* __restrict__ py,
                                            const float* __restrict__ pz, size_t o, int x, int y, int z, int W, int H,
                                            int D, float theta) {
    float div;
    if (x == 0) div = px[o];
    else if (x == W - 1) div = -px[o];
    else div = px[o] - px[o - 1];
    if (y == 0) div += py[o];
    else if (y == H - 1) div += -py[o];
    else div += py[o] - py[o - W];
    if (z == 0) div += pz[o];
    else if (z == D - 1) div += -pz[o];
    else div += pz[o] - pz[o - (size_t)W * H];
    return f[o] - theta * div;
}

constexpr int kTvX = 32, kTvY = 8, kTvZ = 32;  // CTA: 32 x 8 columns, marching 32 planes
// One thread per element of the tile and its +x / +y halo (33 x 9): every u of a plane is
// one thread's, computed once.  A thread keeps its column's p_k of the current plane in
// registers (the update reads them, and pz of the plane is the next plane's -z neighbour),
// so a plane costs it f, px, py, pz and the -x / -y neighbours (L1 hits of the adjacent
// threads' loads).
constexpr int kTvFX = kTvX + 1, kTvFY = kTvY + 1, kTvThreads = kTvFX * kTvFY;

// One inner step: p_b = updateP(u_a, p_a) with u_a = updateU(f, p_a); FIRST: p_a = 0, u_a = f.
template <bool FIRST>
__global__ void __launch_bounds__(kTvThreads) tv_step_kernel(const float* __restrict__ f, const float* __restrict__ pxa,
                                                           const float* __restrict__ pya, const float* __restrict__ pza,
                                                           float* __restrict__ pxb, float* __restrict__ pyb,
                                                           float* __restrict__ pzb, int W, int H, int D, float theta,
                                                           float g, float dt) {
    __shared__ float us[2][kTvFY][kTvFX];  // u of planes z and z + 1 over the tile and its halo
    const int lx = threadIdx.x % kTvFX, ly = threadIdx.x / kTvFX;
    const int x = blockIdx.x * kTvX + lx, y = blockIdx.y * kTvY + ly;
    const int z0 = blockIdx.z * kTvZ, z1 = min(z0 + kTvZ, D);
    const size_t WH = (size_t)W * H;
    const bool in = x < W && y < H;
    const bool inner = in && lx < kTvX && ly < kTvY;  // writes p_b
    const float k = dt / theta;
    // A plane's inputs are loaded one iteration before its u is computed, so the loads
    // overlap the update of the plane before.
    struct In {
        float f, px, py, pz, pxm, pym;  // pxm / pym: the -x / -y neighbours' p (0 where unused)
    };
    auto load = [&](int z) -> In {
        In v{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (!in) return v;
        const size_t o = (size_t)z * WH + (size_t)y * W + x;
        v.f = f[o];
        if (!FIRST) {
            v.px = pxa[o];
            v.py = pya[o];
            v.pz = pza[o];
            if (x > 0 && x < W - 1) v.pxm = pxa[o - 1];
            if (y > 0 && y < H - 1) v.pym = pya[o - W];
        }
        return v;
    };
    // pz of this column at the plane before the one whose u is computed next
    float pzm = 0.0f;
    if (!FIRST && in && z0 > 0 && z0 < D - 1) pzm = pza[(size_t)(z0 - 1) * WH + (size_t)y * W + x];
    // u from loaded inputs (updateU's expressions and order, as tv_u_point)
    auto u_of = [&](const In& v, int z) -> float {
        if (!in) return 0.0f;
        if (FIRST) return v.f;
        float div;
        if (x == 0) div = v.px;
        else if (x == W - 1) div = -v.px;
        else div = v.px - v.pxm;
        if (y == 0) div += v.py;
        else if (y == H - 1) div += -v.py;
        else div += v.py - v.pym;
        if (z == 0) div += v.pz;
        else if (z == D - 1) div += -v.pz;
        else div += v.pz - pzm;
        pzm = v.pz;
        return v.f - theta * div;
    };
    In c = load(z0);                             // plane z0
    In nx = z0 + 1 < D ? load(z0 + 1) : c;      // plane z0 + 1, in flight
    us[0][ly][lx] = u_of(c, z0);
    int cur = 0;
    for (int z = z0; z < z1; z++) {
        const float cpx = c.px, cpy = c.py, cpz = c.pz;  // p_a at (x, y, z)
        if (z + 1 < D) {
            us[cur ^ 1][ly][lx] = u_of(nx, z + 1);
            c = nx;
            if (z + 2 < D && z + 1 < z1) nx = load(z + 2);
        }
        __syncthreads();
        if (inner) {
            const size_t o = (size_t)z * WH + (size_t)y * W + x;
            const float u0 = us[cur][ly][lx];
            const float duy = (y < H - 1) ? us[cur][ly + 1][lx] - u0 : 0.0f;
            const float dux = (x < W - 1) ? us[cur][ly][lx + 1] - u0 : 0.0f;
            const float duz = (z < D - 1) ? us[cur ^ 1][ly][lx] - u0 : 0.0f;
            const float s = duy * duy + dux * dux + duz * duz;
            const float dd1 = 1.0f + dt / theta / g * fabsf(__fsqrt_rn(s));
            pxb[o] = __fdiv_rn(cpx - k * dux, dd1);
            pyb[o] = __fdiv_rn(cpy - k * duy, dd1);
            pzb[o] = __fdiv_rn(cpz - k * duz, dd1);
        }
        __syncthreads();
        cur ^= 1;
    }
}

// The same step four columns per thread, for rows of a multiple of four floats: a warp takes
// 128 columns of one row (16-byte copies and stores), eight warps eight rows and a ninth warp
// the row below them, whose u the last row's update needs; the column right of the 128 is the
// last lane's.  Planes come through a ring of kTv4Stages shared-memory stages (asynchronous
// copies, two planes ahead of the update), so that what is in flight costs no registers; a
// plane's u stays in registers for the next plane's z neighbour and goes through shared
// memory for the row above.  One barrier per plane.
// Bound: HBM (f and p read, p written: 28 B per voxel).  512 x 256 x 512: 320 us per step;
// one column per thread 495 us (245 instructions per voxel, 82 % of the issue slots), four
// columns with the next plane's loads in registers 434 us; floor 277 us.
constexpr int kTv4Rows = 8, kTv4Z = 32, kTv4Threads = 32 * (kTv4Rows + 1), kTv4Stages = 3;

struct Tv4Plane {
    float4 f[kTv4Rows + 1][32], px[kTv4Rows + 1][32], pz[kTv4Rows + 1][32], py[kTv4Rows + 2][32];  // py[r + 1]: row r
    float ef[kTv4Rows + 1], epx[kTv4Rows + 1], epz[kTv4Rows + 1], epy[kTv4Rows + 2];  // the column right of the tile
    float lpx[kTv4Rows + 1];                                                          // px left of it
};
constexpr size_t kTv4Smem = kTv4Stages * sizeof(Tv4Plane) + 2 * sizeof(float4) * (kTv4Rows + 1) * 32;

__device__ __forceinline__ void tv_copy16(void* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void tv_copy4(void* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// updateU's x term of column x from p and its left neighbour's.
__device__ __forceinline__ float tv_dx(float p, float pm, int x, int W) {
    return x == 0 ? p : x == W - 1 ? -p : p - pm;
}
// u of one voxel from the x term (updateU's expressions and order).
__device__ __forceinline__ float tv_u1(float f, float dx, float py, float pym, float pz, float pzm, int y, int z, int H,
                                       int D, float theta) {
    float div = dx;
    if (y == 0) div += py;
    else if (y == H - 1) div += -py;
    else div += py - pym;
    if (z == 0) div += pz;
    else if (z == D - 1) div += -pz;
    else div += pz - pzm;
    return f - theta * div;
}

template <bool FIRST>
__global__ void __launch_bounds__(kTv4Threads, 3) tv_step4_kernel(const float* __restrict__ f, const float* __restrict__ pxa,
                                                               const float* __restrict__ pya,
                                                               const float* __restrict__ pza, float* __restrict__ pxb,
                                                               float* __restrict__ pyb, float* __restrict__ pzb, int W,
                                                               int H, int D, float theta, float g, float dt) {
    extern __shared__ __align__(16) unsigned char tvsm[];
    Tv4Plane* ring = reinterpret_cast<Tv4Plane*>(tvsm);
    float4(*us)[kTv4Rows + 1][32] = reinterpret_cast<float4(*)[kTv4Rows + 1][32]>(ring + kTv4Stages);
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    const int x = blockIdx.x * 128 + 4 * lane, y = blockIdx.y * kTv4Rows + wy;
    const int z0 = blockIdx.z * kTv4Z, z1 = min(z0 + kTv4Z, D), ze = min(z1 + 1, D);  // planes [z0, ze) are read
    const size_t WH = (size_t)W * H;
    const bool in = x < W && y < H;                        // holds u
    const bool inner = in && wy < kTv4Rows;                // writes p_b
    const bool edge = lane == 31 && x + 4 < W && y < H;    // also the column right of the tile
    // the halo warp also brings py of the row above the tile
    const bool top = !FIRST && wy == kTv4Rows && blockIdx.y > 0 && x < W;
    const float k = dt / theta, c = dt / theta / g;
    const size_t col = (size_t)y * W + x, tcol = top ? (size_t)(blockIdx.y * kTv4Rows - 1) * W + x : 0;
    auto issue = [&](int z) {
        if (z < ze) {
            Tv4Plane& P = ring[(z - z0) % kTv4Stages];
            const size_t o = (size_t)z * WH + col;
            if (in) {
                tv_copy16(&P.f[wy][lane], f + o);
                if (!FIRST) {
                    tv_copy16(&P.px[wy][lane], pxa + o);
                    tv_copy16(&P.py[wy + 1][lane], pya + o);
                    tv_copy16(&P.pz[wy][lane], pza + o);
                    if (lane == 0 && x > 0) tv_copy4(&P.lpx[wy], pxa + o - 1);
                }
            }
            if (edge) {
                tv_copy4(&P.ef[wy], f + o + 4);
                if (!FIRST) {
                    tv_copy4(&P.epx[wy], pxa + o + 4);
                    tv_copy4(&P.epy[wy + 1], pya + o + 4);
                    tv_copy4(&P.epz[wy], pza + o + 4);
                }
            }
            if (top) {
                tv_copy16(&P.py[0][lane], pya + (size_t)z * WH + tcol);
                if (lane == 31 && x + 4 < W) tv_copy4(&P.epy[0], pya + (size_t)z * WH + tcol + 4);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // p at the plane whose u was computed last (the update's p, and the next plane's -z neighbour)
    float4 px = zero4, py = zero4, pz = zero4;
    float epz = 0.0f, eu = 0.0f;
    if (!FIRST && in && z0 > 0) {
        const size_t o = (size_t)(z0 - 1) * WH + col;
        pz = *reinterpret_cast<const float4*>(pza + o);
        if (edge) epz = pza[o + 4];
    }
    auto u_of = [&](int z) -> float4 {
        const Tv4Plane& P = ring[(z - z0) % kTv4Stages];
        const float4 fv = P.f[wy][lane];
        if (FIRST) {
            if (edge) eu = P.ef[wy];
            return fv;
        }
        const float4 nx = P.px[wy][lane], ny = P.py[wy + 1][lane], nm = P.py[wy][lane], nz = P.pz[wy][lane];
        float left = __shfl_up_sync(0xffffffffu, nx.w, 1);
        if (lane == 0) left = P.lpx[wy];  // (column 0 does not use it)
        float4 u;
        u.x = tv_u1(fv.x, tv_dx(nx.x, left, x, W), ny.x, nm.x, nz.x, pz.x, y, z, H, D, theta);
        u.y = tv_u1(fv.y, tv_dx(nx.y, nx.x, x + 1, W), ny.y, nm.y, nz.y, pz.y, y, z, H, D, theta);
        u.z = tv_u1(fv.z, tv_dx(nx.z, nx.y, x + 2, W), ny.z, nm.z, nz.z, pz.z, y, z, H, D, theta);
        u.w = tv_u1(fv.w, tv_dx(nx.w, nx.z, x + 3, W), ny.w, nm.w, nz.w, pz.w, y, z, H, D, theta);
        if (edge) {
            const float ez = P.epz[wy];
            eu = tv_u1(P.ef[wy], tv_dx(P.epx[wy], nx.w, x + 4, W), P.epy[wy + 1], P.epy[wy], ez, epz, y, z, H, D, theta);
            epz = ez;
        }
        return u;
    };
    auto take_p = [&](int z) {
        if (FIRST) return;
        const Tv4Plane& P = ring[(z - z0) % kTv4Stages];
        px = P.px[wy][lane];
        py = P.py[wy + 1][lane];
        pz = P.pz[wy][lane];
    };
    issue(z0);
    issue(z0 + 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    float4 uc = u_of(z0);
    float euc = eu;
    take_p(z0);
    us[0][wy][lane] = uc;
    for (int z = z0; z < z1; z++) {
        const int b = (z - z0) & 1;
        // plane z + 2 takes the stage of plane z - 1, last read before the previous barrier
        issue(z + 2);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();  // plane z + 1 and this plane's u rows are visible
        float4 un = uc;
        float eun = euc;
        if (z + 1 < D) {
            un = u_of(z + 1);
            eun = eu;
            us[b ^ 1][wy][lane] = un;
        }
        float right = __shfl_down_sync(0xffffffffu, uc.x, 1);
        if (lane == 31) right = euc;
        if (inner) {
            const float4 ud = us[b][wy + 1][lane];
            float4 qx, qy, qz;
            auto upd = [&](float u0, float ur, float uy, float uz, float p, float q, float r, bool lastx, float& ox,
                           float& oy, float& oz) {
                const float duy = (y < H - 1) ? uy - u0 : 0.0f;
                const float dux = lastx ? 0.0f : ur - u0;
                const float duz = (z < D - 1) ? uz - u0 : 0.0f;
                const float s = duy * duy + dux * dux + duz * duz;
                const float dd1 = 1.0f + c * fabsf(__fsqrt_rn(s));
                ox = __fdiv_rn(p - k * dux, dd1);
                oy = __fdiv_rn(q - k * duy, dd1);
                oz = __fdiv_rn(r - k * duz, dd1);
            };
            upd(uc.x, uc.y, ud.x, un.x, px.x, py.x, pz.x, false, qx.x, qy.x, qz.x);
            upd(uc.y, uc.z, ud.y, un.y, px.y, py.y, pz.y, false, qx.y, qy.y, qz.y);
            upd(uc.z, uc.w, ud.z, un.z, px.z, py.z, pz.z, false, qx.z, qy.z, qz.z);
            upd(uc.w, right, ud.w, un.w, px.w, py.w, pz.w, x + 3 == W - 1, qx.w, qy.w, qz.w);
            const size_t o = (size_t)z * WH + col;
            *reinterpret_cast<float4*>(pxb + o) = qx;
            *reinterpret_cast<float4*>(pyb + o) = qy;
            *reinterpret_cast<float4*>(pzb + o) = qz;
        }
        if (z + 1 < z1) take_p(z + 1);
        uc = un;
        euc = eun;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The closing updateU, four columns per thread (rows of a multiple of four floats), marching
// along z: 20 B per voxel, bound by HBM.
constexpr int kTvFinalZ = 16;
__global__ void __launch_bounds__(256) tv_final4_kernel(float* fu, const float* __restrict__ px,
                                                        const float* __restrict__ py, const float* __restrict__ pz,
                                                        int W, int H, int D, float theta) {
    const int lane = threadIdx.x & 31;
    const int x = blockIdx.x * 128 + 4 * lane, y = blockIdx.y * 8 + (threadIdx.x >> 5);
    const int z0 = blockIdx.z * kTvFinalZ, z1 = min(z0 + kTvFinalZ, D);
    const bool in = x < W && y < H;
    const size_t WH = (size_t)W * H, col = (size_t)y * W + x;
    const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 pzm = in && z0 > 0 ? *reinterpret_cast<const float4*>(pz + (size_t)(z0 - 1) * WH + col) : zero4;
#pragma unroll 2
    for (int z = z0; z < z1; z++) {
        const size_t o = (size_t)z * WH + col;
        float4 a = zero4, b = zero4, bm = zero4, d = zero4, fv = zero4;
        float left = 0.0f;
        if (in) {
            fv = *reinterpret_cast<const float4*>(fu + o);
            a = *reinterpret_cast<const float4*>(px + o);
            b = *reinterpret_cast<const float4*>(py + o);
            d = *reinterpret_cast<const float4*>(pz + o);
            if (y > 0 && y < H - 1) bm = *reinterpret_cast<const float4*>(py + o - W);
            if (lane == 0 && x > 0) left = px[o - 1];
        }
        const float sh = __shfl_up_sync(0xffffffffu, a.w, 1);
        if (lane > 0) left = sh;
        if (in) {
            float4 u;
            u.x = tv_u1(fv.x, tv_dx(a.x, left, x, W), b.x, bm.x, d.x, pzm.x, y, z, H, D, theta);
            u.y = tv_u1(fv.y, tv_dx(a.y, a.x, x + 1, W), b.y, bm.y, d.y, pzm.y, y, z, H, D, theta);
            u.z = tv_u1(fv.z, tv_dx(a.z, a.y, x + 2, W), b.z, bm.z, d.z, pzm.z, y, z, H, D, theta);
            u.w = tv_u1(fv.w, tv_dx(a.w, a.z, x + 3, W), b.w, bm.w, d.w, pzm.w, y, z, H, D, theta);
            *reinterpret_cast<float4*>(fu + o) = u;
        }
        pzm = d;
    }
}

// The closing updateU, in place: fu holds f and receives u (each voxel reads only its own f).
__global__ void tv_final_kernel(float* fu, const float* __restrict__ px, const float* __restrict__ py,
                                const float* __restrict__ pz, int W, int H, int D, float theta) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y, z = blockIdx.z;
    if (x >= W) return;
    const size_t o = ((size_t)z * H + y) * W + x;
    fu[o] = tv_u_point(fu, px, py, pz, o, x, y, z, W, H, D, theta);
}

__global__ void fill_kernel(float* p, size_t n, float v) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        p[i] = v;
}

// FistaProjector3D.endOfIteration (FistaProjector3D.java:43-59) with addToPixel's NaN skip.
__global__ void fista_kernel(float* rec, const float* __restrict__ prev, size_t n, double factor) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double val = __dmul_rn(factor, (double)(rec[i] - prev[i]));
        if (!isnan(val)) rec[i] = rec[i] + __double2float_rn(val);
    }
}

// BayesianVoxelProjector3D.startOfIteration -> convolve(rec, kernel, distanceVolume, -lambda)
// (TomoJ_AdvancedReconstruction/.../projectors/BayesianVoxelProjector3D.java:131-134, 168-194):
// the 27-point stencil [1,-2,1]^3 over TomoReconstruction2.getCubicNeightborhoodWithClamp
// (TomoReconstruction2.java:317-339), whose out-of-volume neighbours read 0 through getPixel;
// float products (exact: the weights are powers of two) summed in double in the reference's
// neighbour order (x offset outermost, z innermost), times factor, rounded to float.
__global__ void bayes_conv_kernel(const float* __restrict__ rec, float* __restrict__ dist, int W, int H, int D,
                                  double factor) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y, z = blockIdx.z;
    if (x >= W) return;
    const float k1[3] = {1.0f, -2.0f, 1.0f};
    double total = 0.0;
#pragma unroll
    for (int i = -1; i <= 1; i++)
#pragma unroll
        for (int j = -1; j <= 1; j++)
#pragma unroll
            for (int k = -1; k <= 1; k++) {
                const int xx = x + i, yy = y + j, zz = z + k;
                float v = 0.0f;
                if (xx >= 0 && xx < W && yy >= 0 && yy < H && zz >= 0 && zz < D)
                    v = rec[((size_t)zz * H + yy) * W + xx];
                total = __dadd_rn(total, (double)__fmul_rn(v, k1[i + 1] * k1[j + 1] * k1[k + 1]));
            }
    dist[((size_t)z * H + y) * W + x] = __double2float_rn(__dmul_rn(total, factor));
}

// BayesianVoxelProjector3D.endOfIteration (:119-129): distance *= alpha (float pixel times
// double, rounded to float), volume += distance (float), then positivity (max with 0).
__global__ void bayes_apply_kernel(float* rec, float* dist, size_t n, double alpha, int positivity) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float d = __double2float_rn(__dmul_rn((double)dist[i], alpha));
        dist[i] = d;
        float v = __fadd_rn(d, rec[i]);
        if (positivity && 0.0f > v) v = 0.0f;
        rec[i] = v;
    }
}

// ---- BgARTVoxelProjector3D (TomoJ_AdvancedReconstruction/.../BgARTVoxelProjector3D.java) ----

// Order-preserving unsigned key of a float (-0.0 before 0.0), and back.
__device__ __forceinline__ unsigned float_key(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}
// Java's Arrays.sort(float[]) order: as float_key, with NaN last.
__device__ __forceinline__ unsigned java_sort_key(float f) { return isnan(f) ? 0xFFFFFFFFu : float_key(f); }

// keys[0] = min key, keys[1] = max key over the non-NaN voxels (keys preset to ~0 / 0).
__global__ void bg_minmax_kernel(const float* __restrict__ v, size_t n, unsigned* keys) {
    unsigned lo = 0xFFFFFFFFu, hi = 0u;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float f = v[i];
        if (isnan(f)) continue;
        const unsigned k = float_key(f);
        lo = min(lo, k);
        hi = max(hi, k);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(keys, lo);
        atomicMax(keys + 1, hi);
    }
}

// ImageJ StackStatistics histogram of 32-bit data: 256 bins over [min, max], bin
// (int)((v - min) * (256 / (max - min))) clamped to 255, all in bin 0 when max == min.
__global__ void bg_hist_kernel(const float* __restrict__ v, size_t n, const unsigned* keys,
                               unsigned long long* hist) {
    __shared__ unsigned h[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const double lo = key_float(keys[0]), hi = key_float(keys[1]);
    const double scale = __ddiv_rn(256.0, hi - lo);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float f = v[i];
        if (isnan(f)) continue;
        int b = 0;
        if (hi > lo) {
            b = (int)__dmul_rn((double)f - lo, scale);  // truncation toward zero, as Java's (int)
            if (b > 255) b = 255;
        }
        atomicAdd(&h[b], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
        if (h[i]) atomicAdd(hist + i, (unsigned long long)h[i]);
}

// collapseFilter thresholds (:29-83) in one thread: out = {background, th1, th2}.
__global__ void bg_finalize_kernel(const unsigned* keys, const unsigned long long* hist, double k, double bg_value,
                                   double* out) {
    const double histmin = key_float(keys[0]), histmax = key_float(keys[1]);
    const double bin = (histmax - histmin) / 256;
    double best = 0;
    int max_index = 0;
    for (int i = 0; i < 256; i++)
        if ((double)hist[i] > best) {
            best = (double)hist[i];
            max_index = i;
        }
    const double bg = isnan(bg_value) ? __dadd_rn(histmin, __dmul_rn((double)max_index, bin)) : bg_value;
    double sigma = 0;
    long long count = 0;
    for (int i = 0; i < max_index; i++) {
        const double d = __dsub_rn(__dadd_rn(histmin, __dmul_rn((double)i, bin)), bg);
        sigma = __dadd_rn(sigma, __dmul_rn(__dmul_rn(d, d), (double)hist[i]));
        count += (long long)hist[i];
    }
    sigma = __dsqrt_rn(__ddiv_rn(sigma, (double)count));
    out[0] = bg;
    out[1] = __dsub_rn(bg, __dmul_rn(k, sigma));
    out[2] = __dadd_rn(bg, __dmul_rn(k, sigma));
}

__global__ void bg_apply_kernel(float* v, size_t n, const double* out, int dark_bg) {
    const double bg = out[0], th1 = out[1], th2 = out[2];
    const float bgf = __double2float_rn(bg);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double val = v[i];
        if (dark_bg && val < th2) v[i] = bgf;
        if (!dark_bg && val > th1) v[i] = bgf;
    }
}

// medianFilter3Dcross (:117-145) from the copy `src` into `dst`: the voxel, its z
// neighbours (0 outside) and its in-plane neighbours by flat index within the slice
// (x neighbours wrap across rows; -1 / -W need an index > 0, +1 / +W one < W*H).
__global__ void median_cross_kernel(const float* __restrict__ src, float* __restrict__ dst, int W, int H, int D) {
    const long long P = (long long)W * H;
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int z = blockIdx.y;
    if (idx >= P) return;
    const float* cur = src + P * z;
    float nb[7];
    nb[0] = z > 0 ? cur[idx - P] : 0.0f;
    nb[1] = z < D - 1 ? cur[idx + P] : 0.0f;
    nb[2] = cur[idx];
    nb[3] = (idx + 1 < P) ? cur[idx + 1] : 0.0f;
    nb[4] = (idx - 1 > 0) ? cur[idx - 1] : 0.0f;
    nb[5] = (idx - W > 0) ? cur[idx - W] : 0.0f;
    nb[6] = (idx + W < P) ? cur[idx + W] : 0.0f;
    unsigned key[7];
#pragma unroll
    for (int a = 0; a < 7; a++) key[a] = java_sort_key(nb[a]);
    // rank selection: the element with 3 keys below it (ties broken by position) is the median
    float med = nb[0];
#pragma unroll
    for (int a = 0; a < 7; a++) {
        int below = 0;
#pragma unroll
        for (int b = 0; b < 7; b++) below += (key[b] < key[a]) || (key[b] == key[a] && b < a);
        if (below == 3) med = nb[a];
    }
    dst[P * z + idx] = med;
}

// Long-object compensation: every norm pixel of a projection becomes the projection's maximum.
__global__ void long_object_kernel(float* norm, int npix) {
    __shared__ float red[32];
    float* n = norm + (size_t)blockIdx.x * npix;
    float m = 0.0f;
    for (int i = threadIdx.x; i < npix; i += blockDim.x) m = fmaxf(m, n[i]);
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = (threadIdx.x < blockDim.x / 32) ? red[threadIdx.x] : 0.0f;
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) red[0] = m;
    }
    __syncthreads();
    m = red[0];
    for (int i = threadIdx.x; i < npix; i += blockDim.x) n[i] = m;
}

// VoxelProjector3D.difference (VoxelProjector3D.java:414-433) over precomputed projections
// (used when long-object compensation replaces the norms after projection).
__global__ void diff_kernel(const float* __restrict__ meas, const int* __restrict__ tilts, const float* __restrict__ th,
                            const float* __restrict__ norm, float* __restrict__ diff, double* __restrict__ errpart,
                            int w, int h, int j0, int j1, double factor) {
    __shared__ double red[32];
    const int b = blockIdx.y;
    const int j = blockIdx.x;
    double e2 = 0.0;
    if (j >= j0 && j < j1) {
        const float* e = meas + ((size_t)tilts[b] * h + j) * w;
        const size_t o = ((size_t)b * h + j) * w;
        for (int i = threadIdx.x; i < w; i += blockDim.x) {
            const float ev = e[i], tv = th[o + i];
            float d = 0.0f;
            if (!isnan(ev) && !isnan(tv)) {
                const float q = __fdiv_rn(ev - tv, norm[o + i]);
                const double v = (double)q * factor;
                d = __double2float_rn(v);
                e2 += v * v;
            }
            diff[o + i] = d;
        }
    } else {
        const size_t o = ((size_t)b * h + j) * w;
        for (int i = threadIdx.x; i < w; i += blockDim.x) diff[o + i] = 0.0f;
    }
    e2 = warp_sum(e2);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < (int)blockDim.x / 32; k++) s += red[k];
        errpart[(size_t)b * h + j] = s;
    }
}

// Copies image tilts[b] of src into slot b of dst (addProjection's fresh copy).
__global__ void gather_kernel(float* __restrict__ dst, const float* __restrict__ src, const int* __restrict__ tilts,
                              size_t npix) {
    const int b = blockIdx.y;
    const float* s = src + (size_t)tilts[b] * npix;
    float* d = dst + (size_t)b * npix;
    if ((npix & 3) == 0) {  // every image starts 16-byte aligned
        const float4* s4 = reinterpret_cast<const float4*>(s);
        float4* d4 = reinterpret_cast<float4*>(d);
        for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < npix / 4;
             i += (size_t)gridDim.x * blockDim.x)
            d4[i] = s4[i];
    } else {
        for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < npix; i += (size_t)gridDim.x * blockDim.x)
            d[i] = s[i];
    }
}

// flags[0] |= 1 if any NaN, flags[0] |= 2 if any +-Inf.
__global__ void scan_nonfinite_kernel(const float* __restrict__ p, size_t n, int* flags) {
    int f = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float v = p[i];
        if (isnan(v)) f |= 1;
        else if (isinf(v)) f |= 2;
    }
    f = __reduce_or_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0 && f) atomicOr(flags, f);
}

}  // namespace

static size_t row_filter_smem(int M) { return (size_t)(M + M / 8 + 1) * sizeof(float2); }
static int row_filter_threads(int M) { return std::min(std::max(M / 8, 32), 512); }

cudaError_t misc_init_attributes() {
    cudaError_t e = cudaFuncSetAttribute(row_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)row_filter_smem(4096));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(row_filter_conv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)row_filter_smem(kRowConvMaxM));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(tv_step4_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTv4Smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(tv_step4_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTv4Smem);
    if (e != cudaSuccess) return e;
    const int dft_smem = (kDft2MaxN + 2 * kRowConvMaxM) * (int)sizeof(float2);
    e = cudaFuncSetAttribute(dft2_rows_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, dft_smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(dft2_rows_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, dft_smem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(dft2_rows_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, dft_smem);
}

int device_sms() {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> cache[kMaxDevices];  // 0: not queried yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        cudaGetLastError();
        return 1;
    }
    int v = cache[dev].load(std::memory_order_relaxed);
    if (v > 0) return v;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) {
        cudaGetLastError();
        v = 1;
    }
    cache[dev].store(v, std::memory_order_relaxed);
    return v;
}

cudaError_t launch_gather(float* dst, const float* src, const int* tilts, int T, size_t npix, cudaStream_t s) {
    if (T <= 0) return cudaSuccess;
    dim3 grid((unsigned)std::min<size_t>((npix / 4 + 255) / 256 + 1, 64), T);
    gather_kernel<<<grid, 256, 0, s>>>(dst, src, tilts, npix);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_scan_nonfinite(const float* p, size_t n, int* flags, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, device_sms() * 8);
    scan_nonfinite_kernel<<<blocks, 256, 0, s>>>(p, n, flags);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_align(const float* raw, float* out, const double* tinv, const long long* fix, const double* stats,
                         int N, int w, int h, int normalize, int fill, const unsigned char* mode, int* flags,
                         cudaStream_t s) {
    const size_t npix = (size_t)w * h, per = 256 * kAlignPix;
    align_kernel<<<dim3((unsigned)((npix + per - 1) / per), N), 256, 0, s>>>(raw, out, tinv, fix, stats, w, h, normalize,
                                                                            fill, mode, flags);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_row_filter_tw(float* img, const float* src, const int* pick, const float* mask_row, const float2* tw, int rows, int w,
                                 const int* bad, int rows_per_img, cudaStream_t s) {
    int logn = 0;
    while ((1 << logn) < w) logn++;
    if ((1 << logn) != w) return cudaErrorInvalidValue;
    row_filter_kernel<<<(rows + 1) / 2, row_filter_threads(w), row_filter_smem(w), s>>>(img, src, pick, mask_row, tw, rows, w, logn, bad, rows_per_img);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_row_filter_conv(float* img, const float* src, const int* pick, const float2* H, const float2* tw,
                                   int rows, int w, int M, const int* bad, int rows_per_img, cudaStream_t s) {
    int logM = 0;
    while ((1 << logM) < M) logM++;
    if ((1 << logM) != M || M < 2 * w - 1 || M > kRowConvMaxM) return cudaErrorInvalidValue;
    row_filter_conv_kernel<<<(rows + 1) / 2, row_filter_threads(M), row_filter_smem(M), s>>>(img, src, pick, H, tw, rows, w, M, logM, bad, rows_per_img);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_image_nonfinite(const float* imgs, int T, size_t npix, int* bad, cudaStream_t s) {
    if (T <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(bad, 0, sizeof(int) * (size_t)T, s);
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)std::min<size_t>((npix + 255) / 256, 32), T);
    image_nonfinite_kernel<<<grid, 256, 0, s>>>(imgs, npix, bad);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_weighting_2d(float* imgs, int T, int w, int h, const float* maskT, const DftRowPlan& Pw,
                                const DftRowPlan& Ph, float2* sa, float2* sb, cudaStream_t s) {
    if (T <= 0) return cudaSuccess;
    if (Pw.n != w || Ph.n != h || w > kDft2MaxN || h > kDft2MaxN || T > 65535) return cudaErrorInvalidValue;
    const size_t smw = (size_t)(Pw.n + 2 * Pw.M) * sizeof(float2);
    const size_t smh = (size_t)(Ph.n + 2 * Ph.M) * sizeof(float2);
    const float scale = (float)(1.0 / ((double)w * (double)h));
    const dim3 tb(32, 8);
    dft2_rows_kernel<0><<<(unsigned)T * h, 256, smw, s>>>(imgs, sa, nullptr, nullptr, Pw, 1, 1.0f);
    count_launch();
    transpose_c_kernel<<<dim3((w + 31) / 32, (h + 31) / 32, T), tb, 0, s>>>(sa, sb, h, w);
    count_launch();
    dft2_rows_kernel<1><<<(unsigned)T * w, 256, smh, s>>>(nullptr, sb, nullptr, maskT, Ph, w, 1.0f);
    count_launch();
    transpose_c_kernel<<<dim3((h + 31) / 32, (w + 31) / 32, T), tb, 0, s>>>(sb, sa, w, h);
    count_launch();
    dft2_rows_kernel<2><<<(unsigned)T * h, 256, smw, s>>>(nullptr, sa, imgs, nullptr, Pw, 1, scale);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_reduce_err(const double* errpart, double* err, int T, int h, cudaStream_t s) {
    if (T <= 0) return cudaSuccess;
    reduce_err_kernel<<<(T + kErrWarps - 1) / kErrWarps, 32 * kErrWarps, 0, s>>>(errpart, err, T, h);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_reduce_err_batch(const ErrReduce* jobs, int n_jobs, int max_T, cudaStream_t s) {
    if (n_jobs <= 0) return cudaSuccess;
    reduce_err_batch_kernel<<<dim3((max_T + kErrWarps - 1) / kErrWarps, n_jobs), 32 * kErrWarps, 0, s>>>(jobs);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_tv_step(const float* f, const float* const pa[3], float* const pb[3], bool first, int W, int H,
                           int D, float theta, float g, float dt, cudaStream_t s) {
    uintptr_t ptrs = reinterpret_cast<uintptr_t>(f);
    for (int q = 0; q < 3; q++) ptrs |= reinterpret_cast<uintptr_t>(pa[q]) | reinterpret_cast<uintptr_t>(pb[q]);
    if ((W & 3) == 0 && (ptrs & 15) == 0) {
        const dim3 g4((W + 127) / 128, (H + kTv4Rows - 1) / kTv4Rows, (D + kTv4Z - 1) / kTv4Z);
        if (first)
            tv_step4_kernel<true><<<g4, kTv4Threads, kTv4Smem, s>>>(f, pa[0], pa[1], pa[2], pb[0], pb[1], pb[2], W, H, D,
                                                             theta, g, dt);
        else
            tv_step4_kernel<false><<<g4, kTv4Threads, kTv4Smem, s>>>(f, pa[0], pa[1], pa[2], pb[0], pb[1], pb[2], W, H, D,
                                                              theta, g, dt);
        count_launch();
        return cudaGetLastError();
    }
    dim3 grid((W + kTvX - 1) / kTvX, (H + kTvY - 1) / kTvY, (D + kTvZ - 1) / kTvZ);
    if (first)
        tv_step_kernel<true><<<grid, kTvThreads, 0, s>>>(f, pa[0], pa[1], pa[2], pb[0], pb[1], pb[2], W, H, D, theta,
                                                         g, dt);
    else
        tv_step_kernel<false><<<grid, kTvThreads, 0, s>>>(f, pa[0], pa[1], pa[2], pb[0], pb[1], pb[2], W, H, D, theta,
                                                          g, dt);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_tv_final(float* fu, const float* const p[3], int W, int H, int D, float theta, cudaStream_t s) {
    const uintptr_t ptrs = reinterpret_cast<uintptr_t>(fu) | reinterpret_cast<uintptr_t>(p[0]) |
                           reinterpret_cast<uintptr_t>(p[1]) | reinterpret_cast<uintptr_t>(p[2]);
    if ((W & 3) == 0 && (ptrs & 15) == 0) {
        tv_final4_kernel<<<dim3((W + 127) / 128, (H + 7) / 8, (D + kTvFinalZ - 1) / kTvFinalZ), 256, 0, s>>>(
            fu, p[0], p[1], p[2], W, H, D, theta);
        count_launch();
        return cudaGetLastError();
    }
    dim3 grid((W + 127) / 128, H, D);
    tv_final_kernel<<<grid, 128, 0, s>>>(fu, p[0], p[1], p[2], W, H, D, theta);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_fill(float* p, size_t n, float v, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, device_sms() * 16);
    fill_kernel<<<blocks, 256, 0, s>>>(p, n, v);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_fista(float* rec, const float* prev, size_t n, double factor, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, device_sms() * 16);
    fista_kernel<<<blocks, 256, 0, s>>>(rec, prev, n, factor);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_bayes_conv(const float* rec, float* dist, int W, int H, int D, double factor, cudaStream_t s) {
    dim3 grid((W + 127) / 128, H, D);
    bayes_conv_kernel<<<grid, 128, 0, s>>>(rec, dist, W, H, D, factor);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_bayes_apply(float* rec, float* dist, size_t n, double alpha, int positivity, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, device_sms() * 16);
    bayes_apply_kernel<<<blocks, 256, 0, s>>>(rec, dist, n, alpha, positivity);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_bgart_collapse(float* vol, size_t n, double k, int dark_bg, double bg_value, void* scratch,
                                  cudaStream_t s) {
    unsigned* keys = static_cast<unsigned*>(scratch);
    unsigned long long* hist = reinterpret_cast<unsigned long long*>(static_cast<char*>(scratch) + 16);
    double* out = reinterpret_cast<double*>(static_cast<char*>(scratch) + 16 + 256 * 8);
    cudaError_t e;
    if ((e = cudaMemsetAsync(keys, 0xFF, 4, s)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(keys + 1, 0, 4, s)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(hist, 0, 256 * 8, s)) != cudaSuccess) return e;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, device_sms() * 8);
    bg_minmax_kernel<<<blocks, 256, 0, s>>>(vol, n, keys);
    bg_hist_kernel<<<blocks, 256, 0, s>>>(vol, n, keys, hist);
    bg_finalize_kernel<<<1, 1, 0, s>>>(keys, hist, k, bg_value, out);
    bg_apply_kernel<<<blocks, 256, 0, s>>>(vol, n, out, dark_bg);
    count_launch(4);
    return cudaGetLastError();
}

cudaError_t launch_bgart_median(float* vol, float* tmp, int W, int H, int D, cudaStream_t s) {
    const size_t n = (size_t)W * H * D;
    cudaError_t e = cudaMemcpyAsync(tmp, vol, sizeof(float) * n, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    const long long P = (long long)W * H;
    median_cross_kernel<<<dim3((unsigned)((P + 255) / 256), D), 256, 0, s>>>(tmp, vol, W, H, D);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_long_object(float* norm, int T, int h, int w, cudaStream_t s) {
    if (T <= 0) return cudaSuccess;
    long_object_kernel<<<T, 512, 0, s>>>(norm, h * w);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_diff(const float* meas, const int* tilts, const float* th, const float* norm, float* diff,
                        double* errpart, int T, int w, int h, int j0, int j1, double factor, cudaStream_t s) {
    if (T <= 0) return cudaSuccess;
    diff_kernel<<<dim3(h, T), 256, 0, s>>>(meas, tilts, th, norm, diff, errpart, w, h, j0, j1, factor);
    count_launch();
    return cudaGetLastError();
}

}  // namespace tomo
