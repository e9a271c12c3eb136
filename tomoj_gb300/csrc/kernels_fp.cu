// Forward-projection dispatch: the row-vector form's plan, launches and closing pass
// (kernel in fpr_kernel.cuh, compiled once per chunk depth in fpr_kernel_z*.cu), and the
// one-row form's instantiation for the number of detector columns each thread owns
// (QP = ceil(w / threads); kernel in fp_kernel.cuh, one per (threads, QP) in fp_kernel_q*.cu).
#include <algorithm>
#include <cmath>
#include <vector>

#include "device_util.cuh"
#include "tomo_internal.h"

namespace tomo {

cudaError_t fpr_attr_z4();
cudaError_t fpr_attr_z6();
cudaError_t fpr_attr_z8();
cudaError_t fpr_launch_z4(const FpLaunch& a, dim3 grid, size_t smem, cudaStream_t s);
cudaError_t fpr_launch_z6(const FpLaunch& a, dim3 grid, size_t smem, cudaStream_t s);
cudaError_t fpr_launch_z8(const FpLaunch& a, dim3 grid, size_t smem, cudaStream_t s);
cudaError_t fpr_batch_z4(int eb, const FpLaunch* d, const int4* it, int n, size_t smem, cudaStream_t s);
cudaError_t fpr_batch_z6(int eb, const FpLaunch* d, const int4* it, int n, size_t smem, cudaStream_t s);
cudaError_t fpr_batch_z8(int eb, const FpLaunch* d, const int4* it, int n, size_t smem, cudaStream_t s);

cudaError_t fp_launch_t256_q1(const FpLaunch& a, cudaStream_t s);
cudaError_t fp_launch_t256_q2(const FpLaunch& a, cudaStream_t s);
cudaError_t fp_launch_t512_q2(const FpLaunch& a, cudaStream_t s);
cudaError_t fp_launch_t512_q4(const FpLaunch& a, cudaStream_t s);
cudaError_t fp_launch_t512_q8(const FpLaunch& a, cudaStream_t s);
cudaError_t fp_attr_t256_q1();
cudaError_t fp_attr_t256_q2();
cudaError_t fp_attr_t512_q2();
cudaError_t fp_attr_t512_q4();
cudaError_t fp_attr_t512_q8();
cudaError_t fp_batch_t256_q1(const FpLaunch* d, const int4* it, int n, int zc, size_t smem, int pk, cudaStream_t s);
cudaError_t fp_batch_t256_q2(const FpLaunch* d, const int4* it, int n, int zc, size_t smem, int pk, cudaStream_t s);
cudaError_t fp_batch_t512_q2(const FpLaunch* d, const int4* it, int n, int zc, size_t smem, int pk, cudaStream_t s);
cudaError_t fp_batch_t512_q4(const FpLaunch* d, const int4* it, int n, int zc, size_t smem, int pk, cudaStream_t s);
cudaError_t fp_batch_t512_q8(const FpLaunch* d, const int4* it, int n, int zc, size_t smem, int pk, cudaStream_t s);
cudaError_t fpr_persist_attr();

// Raises the dynamic shared-memory limit of every forward-projector variant once,
// outside any stream capture.
cudaError_t fp_init_attributes() {
    cudaError_t e;
    if ((e = fp_attr_t256_q1()) != cudaSuccess) return e;
    if ((e = fp_attr_t256_q2()) != cudaSuccess) return e;
    if ((e = fp_attr_t512_q2()) != cudaSuccess) return e;
    if ((e = fp_attr_t512_q4()) != cudaSuccess) return e;
    if ((e = fpr_attr_z4()) != cudaSuccess) return e;
    if ((e = fpr_attr_z6()) != cudaSuccess) return e;
    if ((e = fpr_attr_z8()) != cudaSuccess) return e;
    if ((e = fpr_persist_attr()) != cudaSuccess) return e;
    return fp_attr_t512_q8();
}

int fp_threads(int w) { return w <= 512 ? 256 : 512; }

int fp_qp(int w) {
    const int nt = fp_threads(w);
    const int qp = (w + nt - 1) / nt;
    return qp <= 1 ? 1 : qp <= 2 ? 2 : qp <= 4 ? 4 : qp <= 8 ? 8 : 0;
}

int fp_max_tilts_per_cta(int w) {
    const int qp = fp_qp(w);
    if (qp == 0) return 0;
    return kFpRays / qp > 0 ? kFpRays / qp : 1;
}

// Shared-memory bytes of a CTA for width W and planes per chunk ZC (matches fpk::layout):
// FP32 volumes stage 4-byte voxels and build 8-byte pairs, 16-bit volumes 2-byte voxels
// and 4-byte pairs.
size_t fp_smem_bytes(int ZC, int W, int qp, int rows, int vtype) {
    const bool h = vtype != kVolF32;
    size_t o = 16 + (size_t)rows * ZC * W * (h ? 2 : 4);
    o = (o + 15) & ~(size_t)15;
    o += (size_t)ZC * (W + 4) * (h ? 4 : 8);
    o = (o + 15) & ~(size_t)15;
    o += (kFpMaxThreads / 32) * sizeof(double) + (size_t)(kFpRays / qp > 0 ? kFpRays / qp : 1) * sizeof(long long);
    return o;
}

int fp_choose_zc(int W, int rows, int vtype, int nt) {
    for (int zc = 16; zc > 1; zc >>= 1)
        if (fp_smem_bytes(zc, W, 1, rows, vtype) <= fp_smem_budget(nt)) return zc;
    return 1;
}

#ifndef TOMO_FP_MAX_ZPARTS
#define TOMO_FP_MAX_ZPARTS 8
#endif

int fp_zparts(int ctas, int D, int zc, int sms, int ctas_per_sm) {
    const int slots = ctas_per_sm * sms;  // resident forward-projector CTAs
    if (ctas <= 0 || ctas >= slots) return 1;
    const int nch = (D + zc - 1) / zc;
    // A CTA's time is about (chunks + 1) chunk-times (the +1 is its set-up, first
    // bulk copy and partial-sum exchange), independent of what else runs on its SM:
    // minimise waves x (chunks per part + 1).
    int best = 1;
    long long best_cost = (long long)nch + 1;
    for (int P = 2; P <= TOMO_FP_MAX_ZPARTS && P <= nch; P++) {
        const int cpp = (nch + P - 1) / P;
        const long long waves = ((long long)ctas * P + slots - 1) / slots;
        const long long cost = waves * (cpp + 1);
        if (cost < best_cost) {
            best_cost = cost;
            best = P;
        }
    }
    return best;
}

cudaError_t launch_fp_batch(int qp, int nt, const FpLaunch* descs, const int4* items, int n_items, int zc,
                            size_t smem, int pk, cudaStream_t s) {
    if (nt == 256) {
        if (qp == 1) return fp_batch_t256_q1(descs, items, n_items, zc, smem, pk, s);
        if (qp == 2) return fp_batch_t256_q2(descs, items, n_items, zc, smem, pk, s);
    } else if (nt == 512) {
        switch (qp) {
            case 2: return fp_batch_t512_q2(descs, items, n_items, zc, smem, pk, s);
            case 4: return fp_batch_t512_q4(descs, items, n_items, zc, smem, pk, s);
            case 8: return fp_batch_t512_q8(descs, items, n_items, zc, smem, pk, s);
        }
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_fp_separable(const FpLaunch& a, cudaStream_t s) {
    if (a.T <= 0 || a.j1 <= a.j0) return cudaSuccess;
    const int nt = fp_threads(a.w), qp = fp_qp(a.w);
    if (nt == 256) return qp == 1 ? fp_launch_t256_q1(a, s) : fp_launch_t256_q2(a, s);
    switch (qp) {
        case 2: return fp_launch_t512_q2(a, s);
        case 4: return fp_launch_t512_q4(a, s);
        case 8: return fp_launch_t512_q8(a, s);
    }
    return cudaErrorInvalidValue;
}

// --- row-vector form ------------------------------------------------------------------------

namespace {

constexpr int kFinishThreads = 128;

// a * b in FP32 for a double b = hi + lo (lo below half an ulp of hi): the product rounded
// once from 48 bits (and its low part), without an FP64 operation per ray (this part's FP64
// rate is 1/64 of FP32: two conversions and a product per ray would take longer than the
// pass's memory traffic).
struct F2 {
    float hi, lo;
};
__device__ __forceinline__ F2 mul_split(float a, F2 b) {
    const float p = a * b.hi;
    const float e = fmaf(a, b.lo, fmaf(a, b.hi, -p));
    const float r = p + e;
    // an infinite or overflowing product keeps p (the correction is NaN)
    return isfinite(p) ? F2{r, e - (r - p)} : F2{p, 0.0f};
}

// Running sum with its error (two-sum): hi + lo carries about 48 bits.
__device__ __forceinline__ void add2(F2& s, float p, float pe) {
    const float t = s.hi + p, u = t - s.hi;
    s.lo += ((s.hi - (t - u)) + (p - u)) + pe;
    s.hi = t;
}

// Whether a pair of floats holds the square of a difference q * factor of magnitude m (not where m
// is NaN: an extreme factor, see fpr_split_factor).
__device__ __forceinline__ bool pair_range(float m, float q) { return m <= 1e15f && (m >= 1e-15f || q == 0.0f); }

// The differences of projection row j of batch slot b that pair_range leaves out, in double: written
// again, squares returned.  Over this thread's columns; out of line and from the projections and norms
// it has written, so that the pass itself carries nothing for them.
__device__ __noinline__ double far_row(const FpLaunch& a, int b, int tilt, int j) {
    double sum = 0.0;
    for (int i = threadIdx.x; i < a.w; i += kFinishThreads) {
        const size_t o = ((size_t)b * a.h + j) * a.w + i;
        const float e = a.meas[((size_t)tilt * a.h + j) * a.w + i], th = a.proj[o];
        if (isnan(e) || isnan(th)) continue;
        const float q = __fdiv_rn(__fsub_rn(e, th), a.norm[o]);
        if (pair_range(fabsf(mul_split(q, F2{a.factor_hi, a.factor_lo}).hi), q)) continue;
        const double x = (double)q * a.factor;
        a.diff[o] = __double2float_rn(x);
        sum += x * x;
    }
    return sum;
}

// Projection, norm, difference and residual of n <= RJ consecutive projection rows from their
// segment sums (the epilogue of fp_body with the sums read back, in segment order).  The
// squared differences are summed in FP32 pairs with error terms (those outside a pair's range
// in FP64 by far_row), a warp's sums in FP64; a row's order of adds depends on neither RJ nor UC.  Bound by its memory traffic (segment
// sums, measured row in; projection, norm and difference out) when RJ rows share a ray's
// 32-byte table entry, and by latency on grids of few rows, where UC columns of a row are
// read at once instead.  One row and one column at a time took 13 us for 7 tilts of 512 x 256
// in 5 segments, 482 us for 61 of 1024 x 1024 and 339 us for 12 series of 61 x 512 x 64;
// these forms take 12, 352 and 278 us (two rows: 394 and 299 us for the last two; with the
// differences outside the pairs' range in the same loop 377 and 283 us).
template <int RJ, int UC>
__device__ __forceinline__ void finish_rows(const FpLaunch& a, int b, int j0, int n) {
    __shared__ double red[RJ][kFinishThreads / 32];
    const int tilt = a.tilts[b];
    const F2 ninc{a.ftilt[tilt].ninc_hi, a.ftilt[tilt].ninc_lo}, fac{a.factor_hi, a.factor_lo};
    const size_t seg_stride = (size_t)a.T * a.h * a.w, row = ((size_t)b * a.h + j0) * a.w;
    const float inv_seg = 1.0f / (float)a.rv.seg;
    bool row_in[RJ];
    float vsc[RJ];
    F2 e2[RJ];
    bool any_far = false;  // a difference of this thread lies outside the pairs' range
#pragma unroll
    for (int y = 0; y < RJ; y++) {
        const int r = y >= n ? -1 : a.two_rows ? a.rowmap[j0 + y] : j0 + y - a.row_off;
        row_in[y] = r >= 0 && r < a.H;
        // reduced storage: ray sums are in units of the row's slab scale (a power of two)
        vsc[y] = (a.vscale != nullptr && row_in[y]) ? a.vscale[r] : 1.0f;
        e2[y] = F2{0.0f, 0.0f};
    }
    for (int i0 = threadIdx.x; i0 < a.w; i0 += kFinishThreads * UC) {
        float e[UC][RJ], sum[UC][RJ], nrm[UC];
        int s0[UC], s1[UC], smin = a.rv.nseg, smax = -1;
#pragma unroll
        for (int c = 0; c < UC; c++) {
            const int i = i0 + c * kFinishThreads;
            s0[c] = a.rv.nseg;
            s1[c] = -1;
            nrm[c] = 0.0f;
            if (i < a.w) {
                const FpRay& ray = a.rays[(size_t)tilt * a.w + i];
                const int zab = ray.zab, za = zab & 0xFFFF, cnt = (int)((uint32_t)zab >> 16);
                nrm[c] = ray.norm;
                if (cnt != 0) {
                    // floor(z / seg): z + 1/2 keeps the product clear of whole numbers (z < 2^16)
                    s0[c] = (int)((za + 0.5f) * inv_seg);
                    s1[c] = (int)((za + cnt - 0.5f) * inv_seg);
                }
            }
            smin = min(smin, s0[c]);
            smax = max(smax, s1[c]);
#pragma unroll
            for (int y = 0; y < RJ; y++) {
                e[c][y] = (a.meas != nullptr && y < n && i < a.w)
                              ? a.meas[((size_t)tilt * a.h + j0 + y) * a.w + i] : 0.0f;
                sum[c][y] = 0.0f;
            }
        }
        for (int s = smin; s <= smax; s += 4) {
            float v[4][UC][RJ];
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int c = 0; c < UC; c++)
#pragma unroll
                    for (int y = 0; y < RJ; y++)
                        v[q][c][y] = (s + q >= s0[c] && s + q <= s1[c] && row_in[y])
                                         ? __ldcg(a.part + (s + q) * seg_stride + row + (size_t)y * a.w + i0 + c * kFinishThreads)
                                         : 0.0f;
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int c = 0; c < UC; c++)
#pragma unroll
                    for (int y = 0; y < RJ; y++) sum[c][y] += v[q][c][y];
        }
#pragma unroll
        for (int c = 0; c < UC; c++) {
            const int i = i0 + c * kFinishThreads;
            if (i >= a.w) continue;
#pragma unroll
            for (int y = 0; y < RJ; y++) {
                if (y >= n) continue;
                const size_t o = row + (size_t)y * a.w + i;
                float th = __int_as_float(0x7fc00000), nr = 0.0f;
                if (s1[c] >= 0 && row_in[y]) {
                    th = mul_split(sum[c][y], ninc).hi * vsc[y];
                    nr = nrm[c];
                }
                a.proj[o] = th;
                a.norm[o] = nr;
                if (a.meas != nullptr) {
                    float d = 0.0f;
                    if (!isnan(e[c][y]) && !isnan(th)) {
                        const float q = __fdiv_rn(__fsub_rn(e[c][y], th), nr);
                        const F2 v = mul_split(q, fac);
                        d = v.hi;
                        const float m = fabsf(d);
                        if (pair_range(m, q)) {
                            const float p = d * d;
                            add2(e2[y], p, fmaf(d, d, -p) + 2.0f * d * v.lo);
                        } else {
                            any_far = true;
                        }
                    }
                    a.diff[o] = d;
                }
            }
        }
    }
    if (a.meas != nullptr) {
#pragma unroll
        for (int y = 0; y < RJ; y++) {
            // the lanes' sums in fixed order, without FP64
#pragma unroll
            for (int q = 16; q > 0; q >>= 1) {
                const float oh = __shfl_down_sync(0xffffffffu, e2[y].hi, q);
                const float ol = __shfl_down_sync(0xffffffffu, e2[y].lo, q);
                add2(e2[y], oh, ol);
            }
            double far = 0.0;
            if (__any_sync(0xffffffffu, any_far)) far = warp_sum(any_far && y < n ? far_row(a, b, tilt, j0 + y) : 0.0);
            if ((threadIdx.x & 31) == 0)
                red[y][threadIdx.x >> 5] = (double)e2[y].hi + (double)e2[y].lo + far;
        }
        __syncthreads();
        if (threadIdx.x < n) {
            double sum = 0.0;
            for (int k = 0; k < kFinishThreads / 32; k++) sum += red[threadIdx.x][k];
            a.errpart[(size_t)b * a.h + j0 + threadIdx.x] = sum;
        }
    }
}

template <int RJ, int UC>
__global__ void __launch_bounds__(kFinishThreads) fp_finish_kernel(const __grid_constant__ FpLaunch a) {
    const int j = a.j0 + blockIdx.x * RJ;
    finish_rows<RJ, UC>(a, blockIdx.y, j, min(RJ, a.j1 - j));
}

// Batched form: block b runs items[b] = {problem, tilt, first row, rows}.
__global__ void __launch_bounds__(kFinishThreads, 8)
    fp_finish_batch_kernel(const FpLaunch* __restrict__ descs, const int4* __restrict__ items) {
    const int4 it = items[blockIdx.x];
    finish_rows<kFinishRows, 1>(descs[it.x], it.y, it.z, it.w);
}

}  // namespace

size_t fpr_smem_bytes(const FprPlan& p) { return kFprFixedSmem + (size_t)p.zc * p.pitch * (64 + 4 * p.rawrows); }

// A grid on `sms` SMs: CTAs start in segment order, `per_seg` each.  Times are in units of a full
// segment's CTA; a segment away from the middle plane has fewer rays inside, the last one fewer
// planes.
namespace {
struct CtaGrid {
    int nseg, per_seg, sms;
    double last, lean;
    double weight(int s) const {
        const double d = nseg > 1 ? std::fabs((s + 0.5) / nseg - 0.5) * 2 : 0.0;
        return (s == nseg - 1 ? last : 1.0) * (1.0 - lean * d);
    }
    bool many() const { return (double)nseg * per_seg > 4.0 * sms; }
    // work per SM: the time of many CTAs, less half a CTA.  (The distances of weight() add up to
    // nseg / 2, less 1 / (2 nseg) for odd numbers of segments.)
    double mean() const {
        const double dist = nseg > 1 ? 0.5 * nseg - (nseg & 1 ? 0.5 / nseg : 0.0) : 0.0;
        const double first = nseg > 1 ? weight(0) : 1.0;  // the last one's, were it full
        return (nseg - lean * dist - first + weight(nseg - 1)) * per_seg / sms;
    }
    // No grid of few CTAs is faster: the mean, and the busiest SM's CTAs at the shortest times there are.
    double least() const {
        const double end = weight(nseg - 1), other = nseg > 1 ? weight(0) : end;  // end <= other <= the rest
        const int rounds = (int)(((long long)nseg * per_seg + sms - 1) / sms), ends = std::min(per_seg, rounds);
        return std::max(mean(), ends * end + (rounds - ends) * other) * (1.0 - 1e-9);
    }
    // Few CTAs, each taken by the SM that is free first.
    double simulated() const {
        std::vector<double> free_at(sms, 0.0);  // a binary heap, earliest first
        const long long n = (long long)nseg * per_seg;
        double end = 0;
        for (int s = 0; s < nseg; s++) {
            const double w = weight(s);
            for (int q = 0; q < per_seg; q++) {
                if (n <= sms) {  // an SM for every CTA
                    end = std::max(end, w);
                    break;
                }
                const double t = free_at[0] + w;
                end = std::max(end, t);
                int i = 0;
                for (int c; (c = 2 * i + 1) < sms; i = c) {
                    if (c + 1 < sms && free_at[c + 1] < free_at[c]) c++;
                    if (free_at[c] >= t) break;
                    free_at[i] = free_at[c];
                }
                free_at[i] = t;
            }
        }
        return end;
    }
};
}  // namespace

// Cuts a projection into CTAs by a cost model (cycles of one SM): a plane costs half a cycle
// per staged column (8 voxels transposed at 16 a cycle) and 18.4 cycles per ray block (256
// samples at 13.9 a cycle), with one plane's worth of bookkeeping per chunk; a CTA costs
// 12000 cycles besides (lists, first chunk, sums).  Fitted on 512 x 256 x 512: 7 tilts in 4 /
// 5 / 8 / 13 / 16 segments 202 / 177 / 200 / 191 / 206 us, 41 tilts in 3 / 6 / 13 segments
// 995 / 1022 / 1090 us; 256 x 64 x 256, 61 tilts in 4 / 7 / 8 segments 118 / 116 / 128 us;
// 1024 x 256 x 256, 61 tilts in 6 windows of 3 segments 1567 us, 5 of 3 1655 us.
// Deeper chunks leave narrower windows (the buffers hold zc * pitch columns), longer segments
// wider margins around a window (tilts fan out by max_step columns per plane).
// The first projection of a handle waits for this (a 128 x 32 x 128 update takes 98 us), so grids
// of few CTAs, whose time takes a simulation, are looked at in the order of their lower bounds and
// only while one could still be the cheapest: the choice is that of simulating all, in 1 to 25 us
// instead of 30 to 118 (256 x 64 x 256, 61 tilts).
FprPlan fpr_plan(const FprGeom& g, int T, int sms) {
    FprPlan best{};
    if (T <= 0 || g.w > 4096 || !(g.max_step <= 16.0) || !(g.max_space <= 64.0) || !(g.min_space > 0)) return best;
    const int NB = (g.w + kFprRays - 1) / kFprRays, cap = kFprSlots * 16;
    // eight projection rows touch the rows between their floors and one more
    const int rawrows = g.row_step > 0 ? (int)std::ceil(7 * g.row_step) + 2 : 8;
    if (rawrows > 16) return best;
    const int nrg = (g.rows + 14) / 8;
    struct Cut {
        FprPlan p;
        CtaGrid grid;
        double unit, rest, cost;  // cycles per unit of grid time and besides; cost or its lower bound
    };
    std::vector<Cut> cuts;
    cuts.reserve(72);
    for (int zc : {8, 6, 4}) {
        const int room = (int)((kFprSmemMax - kFprFixedSmem) / ((size_t)zc * (64 + 4 * rawrows)));
        for (int nch = 1; nch <= kFprMaxChunks; nch = nch < 8 ? nch + 1 : nch + (nch + 3) / 4) {
            const int seg = std::min(nch, (g.D + zc - 1) / zc) * zc;
            FprPlan p{};
            p.zc = zc;
            p.rawrows = rawrows;
            p.seg = seg;
            p.nseg = (g.D + seg - 1) / seg;
            double cols;
            int nbw;
            double nba;
            // pitches are multiples of 8: a staged row starts on a 16-byte boundary in 16 bits too
            if (((g.W + 11) & ~7) <= room) {
                p.nwin = 1;
                p.xw = g.W;
                p.pitch = (g.W + 11) & ~7;
                cols = g.W + 4;
                nbw = NB;
                nba = NB;
            } else {
                // margins: the tilts' fan over half a segment, a block's width, rounding
                const int half = (seg + 1) / 2 + 1;
                const int margin = 2 * (int)std::ceil(half * g.max_step + 1) + 2 * (int)std::ceil((kFprRays - 1) * g.max_space + 2) + 16;
                p.xw = (room & ~7) - margin;
                if (p.xw < 64) {
                    if (seg >= g.D || nch > 1) break;
                    continue;
                }
                p.nwin = (g.W + p.xw - 1) / p.xw;
                p.xw = (g.W + p.nwin - 1) / p.nwin;
                p.pitch = (p.xw + margin + 7) & ~7;
                cols = std::min<double>(g.W + 3, p.xw + half * g.max_step + kFprRays * g.max_space);
                nbw = std::min(NB, (int)(p.xw / (kFprRays * g.min_space)) + 2);
                nba = std::min<double>(NB, p.xw / (kFprRays * std::min(1.2 * g.min_space, g.max_space)) + 0.5);
            }
            int tg = std::max(1, std::min({kFprMaxTilts, T, cap / nbw}));
            const int ntg = (T + tg - 1) / tg;
            tg = (T + ntg - 1) / ntg;
            p.tg = tg;
            const int passes = (nbw * tg + cap - 1) / cap;
            // (whole rows of 16 blocks: every warp has as many ray blocks as the busiest)
            double per_plane = passes * 0.5 * cols + 18.4 * 16.0 * std::ceil(tg * nba / 16.0) * (1.0 + 1.0 / zc);
            per_plane = std::max(per_plane, 1200.0 / zc) + 600.0 / zc;
            const double last = (double)(g.D - (p.nseg - 1) * seg) / seg;
            const double lean = std::min(0.35, 0.2 * g.D * g.max_step / g.W);
            Cut c{p, CtaGrid{p.nseg, ntg * p.nwin * nrg, sms, last, lean}, std::min(seg, g.D) * per_plane + 12000.0,
                  (double)p.nseg * T * g.h * g.w * 8.0 / 3400.0, 0.0};
            c.cost = (c.grid.many() ? c.grid.mean() + 0.5 : c.grid.least()) * c.unit + c.rest;
            cuts.push_back(c);
            if (seg >= g.D) break;
        }
    }
    if (cuts.empty()) return best;
    // cheapest first (of equal ones the first listed): done when the cheapest cost is exact
    auto dearer = [&](int x, int y) { return cuts[x].cost != cuts[y].cost ? cuts[x].cost > cuts[y].cost : x > y; };
    std::vector<int> order(cuts.size());
    for (size_t i = 0; i < order.size(); i++) order[i] = (int)i;
    std::make_heap(order.begin(), order.end(), dearer);
    std::vector<bool> exact(cuts.size(), false);
    for (;;) {
        const int i = order.front();
        Cut& c = cuts[i];
        if (exact[i] || c.grid.many()) return c.p;
        std::pop_heap(order.begin(), order.end(), dearer);
        c.cost = c.grid.simulated() * c.unit + c.rest;
        exact[i] = true;
        std::push_heap(order.begin(), order.end(), dearer);
    }
}

int fpr_row_groups(const FpLaunch& a, int* jfirst) {
    if (a.two_rows) {
        *jfirst = a.j0;
        return (a.j1 - a.j0 + 7) / 8;
    }
    // groups end at the volume's last row, whose samples take another form
    const int lo = std::max(a.j0, a.row_off), hi = std::min(a.j1, a.row_off + a.H);
    if (hi <= lo) return 0;
    const int end = a.row_off + a.H;
    const int first = end - (end - lo + 7) / 8 * 8;
    *jfirst = first;
    return (hi - first + 7) / 8;
}

void fpr_split_factor(FpLaunch* a) {
    const double m = std::fabs(a->factor);
    const bool fits = m == 0.0 || (m >= 0x1p-60 && m <= 0x1p60);  // both parts, and products with them, normal
    a->factor_hi = fits ? (float)a->factor : NAN;
    a->factor_lo = fits ? (float)(a->factor - (double)a->factor_hi) : 0.0f;
}

cudaError_t launch_fpr(const FpLaunch& a0, cudaStream_t s) {
    FpLaunch a = a0;
    if (a.T <= 0 || a.j1 <= a.j0) return cudaSuccess;
    const int nrg = fpr_row_groups(a, &a.rv.jfirst);
    a.tilts_per_cta = a.rv.tg;
    fpr_split_factor(&a);
    a.rv.bulk = fp_use_tma(a.W, a.vtype, a.vol);
    if (nrg > 0) {
        const dim3 grid((unsigned)((a.T + a.rv.tg - 1) / a.rv.tg * a.rv.nwin), (unsigned)nrg, (unsigned)a.rv.nseg);
        const size_t sm = fpr_smem_bytes(a.rv);
        const cudaError_t e = a.rv.zc == 8   ? fpr_launch_z8(a, grid, sm, s)
                              : a.rv.zc == 6 ? fpr_launch_z6(a, grid, sm, s)
                                             : fpr_launch_z4(a, grid, sm, s);
        if (e != cudaSuccess) return e;
        count_launch();
    }
    // rows in groups where that still fills the resident blocks (16 per SM), else as many columns at
    // once as a row has per thread
    const long long rows = a.j1 - a.j0;
    if (rows * a.T >= 16LL * kFinishRows * device_sms())
        fp_finish_kernel<kFinishRows, 1><<<dim3((unsigned)((rows + kFinishRows - 1) / kFinishRows), (unsigned)a.T),
                                           kFinishThreads, 0, s>>>(a);
    else if (a.w > 2 * kFinishThreads)
        fp_finish_kernel<1, 4><<<dim3((unsigned)rows, (unsigned)a.T), kFinishThreads, 0, s>>>(a);
    else if (a.w > kFinishThreads)
        fp_finish_kernel<1, 2><<<dim3((unsigned)rows, (unsigned)a.T), kFinishThreads, 0, s>>>(a);
    else
        fp_finish_kernel<1, 1><<<dim3((unsigned)rows, (unsigned)a.T), kFinishThreads, 0, s>>>(a);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_fpr_batch(int zc, int eb, const FpLaunch* descs, const int4* items, int n, size_t smem,
                             cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    count_launch();
    return zc == 8   ? fpr_batch_z8(eb, descs, items, n, smem, s)
           : zc == 6 ? fpr_batch_z6(eb, descs, items, n, smem, s)
                     : fpr_batch_z4(eb, descs, items, n, smem, s);
}

cudaError_t launch_fp_finish_batch(const FpLaunch* descs, const int4* items, int n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    fp_finish_batch_kernel<<<n, kFinishThreads, 0, s>>>(descs, items);
    count_launch();
    return cudaGetLastError();
}

}  // namespace tomo
