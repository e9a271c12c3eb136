// Forward projector, row-vector form: eight projection rows per CTA.
//
// Reference: VoxelProjector3D.projectJosephPartial (TomoJ_Base/.../projectors/
// VoxelProjector3D.java:671-821) and the sampler TomoReconstruction2.getPixel
// (TomoReconstruction2.java:154-190).
//
// With a vertical tilt axis every row of a tilt samples the same (x, z) positions, so a
// position, its interpolation weight and its shared-memory address serve all rows.  A CTA
// owns eight consecutive rows; a plane is staged transposed, [column][8 rows], and a lane
// holds one ray with all eight: four 128-bit shared loads (columns floor(x) and floor(x) + 1,
// two halves of four rows) feed eight samples with packed FP32x2 arithmetic.
//
// What bounds it: the shared-memory data path (a sample is 8 bytes, 16 samples per 128-byte
// wavefront without conflicts), then issue slots.  Odd lanes load the halves in the other
// order, so a quarter-warp's load covers both halves of a 32-byte column with four rays each,
// and is free of conflicts when those four rays start in different columns mod 4.  Rays sit
// 1/cos(theta) columns apart, so neighbours collide; kRayModes picks per tilt which rays
// share a quarter-warp and which of them load column floor(x) + 1 first.
//
// Work split: a CTA covers 8 rows x a run of planes (segment) x a window of columns x a
// group of tilts.  Its rays (blocks of 32, up to kSlots blocks per warp) keep their sums in
// registers while chunks of ZC planes pass through shared memory: bulk copies bring a
// chunk's rows while the chunk before is sampled; each warp transposes its share when it has
// sampled its rays, one barrier per chunk.  Segment
// sums go to part[segment][tilt][row][column]; fp_finish adds them in segment order, so a
// row's result does not depend on how rows, tilts or launches are grouped.
//
// Measured (with fp_finish) against the one-row kernel of fp_kernel.cuh: 512 x 256 x 512, 7
// evenly spread tilts 192 us, 213 us on average over the subsets of an iteration (246), 41 tilts
// 1.04 ms (1.37); 2048 x 512 x 2048, 121 tilts 97 ms (140); 333 x 67 x 150, one tilt 20 us (43).
// 14 samples per wavefront (8.8 there); the data path is 60 % busy over a 7-tilt launch, the
// rest is latency of the loads at 16 warps per SM and the chunk barriers.
#pragma once
#include <climits>
#include <type_traits>

#include "device_util.cuh"
#include "tomo_internal.h"
#include "vol_storage.cuh"

namespace tomo {
namespace fpr {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kSlots = kFprSlots;                    // ray blocks per warp and pass
constexpr int kCap = kWarps * kSlots;         // ray blocks per CTA and pass
constexpr int kRays = 32;                     // rays per block (one per lane)
constexpr int kMaxNB = 4096 / kRays;          // ray blocks of a detector row (w <= 4096)
constexpr uint32_t kWaitTries = 1u << 24;

// Shared memory: barrier | a column of zeros | per-slot info | block lists | two plane buffers.
constexpr int kZeroOff = 32;                                    // float [8]
constexpr int kInfoOff = 64;                                    // BlockInfo [kCap]
constexpr int kZabOff = kInfoOff + kCap * 32;                   // int [kCap][32] plane intervals
constexpr int kStepOff = kZabOff + kCap * 128;                  // long long [kFprMaxTilts]
constexpr int kTiltOff = kStepOff + kFprMaxTilts * 8;          // int [kFprMaxTilts] tilt index
constexpr int kModeOff = kTiltOff + kFprMaxTilts * 4;           // int [kFprMaxTilts]
constexpr int kCntOff = kModeOff + kFprMaxTilts * 4;            // int [kFprMaxTilts + 1]
constexpr int kWidthOff = kCntOff + (kFprMaxTilts + 4) * 4;     // int [kFprMaxTilts] columns a block spans
constexpr int kRowOff = kWidthOff + kFprMaxTilts * 4;           // int [8] rows, float [8] weights, int [2] span
constexpr int kChunkOff = kRowOff + 80;                         // int4 [kFprMaxChunks]
constexpr int kListOff = kChunkOff + kFprMaxChunks * 16;                         // uint16 [kFprMaxTilts][kMaxNB]
constexpr int kBufOff = (kListOff + kFprMaxTilts * kMaxNB * 2 + 127) & ~127;
static_assert(kBufOff <= kFprFixedSmem, "fixed part of the shared memory");

// A block of 32 rays of a tilt: steps from plane to plane (one, and ZC - 1 planes).
struct alignas(16) BlockInfo {
    long long step, span;
    int id;    // tilt slot << 16 | block
    int mode;  // ray_mode
    int pad[2];
};

extern __shared__ __align__(128) unsigned char fsm[];

// How the lanes of a warp share the 32 rays of a block.  A quarter-warp's load is one
// wavefront when the four rays of its even lanes start in different columns mod 4, and those
// of its odd lanes too.  bits 0-3: ray k of a set of four loads column floor(x) + 1 first;
// bits 4-5: log2 of the distance between a set's rays; bits 6-7: which sets are the even and
// odd lanes of one quarter-warp (neighbours, two apart, four apart).
// kRayModes[i]: the mode with the fewest wavefronts per load, averaged over ray offsets, at a
// ray spacing of 1 + i / 64 columns (an exhaustive search over 72 modes): 1.25 on average over
// tilts of 0..60 degrees, against 1.8 for lane order; worst 1.6 near 52 degrees.
__constant__ uint8_t kRayModes[129] = {
    0x00, 0x00, 0x00, 0x80, 0x80, 0x80, 0x4a, 0x4a, 0x4a, 0x4a, 0x4a, 0x8a, 0x8a, 0x0a, 0x0a, 0x0a,
    0x20, 0x0a, 0x0a, 0x0a, 0x8a, 0x0a, 0x0a, 0x4a, 0x4a, 0x4a, 0x0a, 0x8a, 0x8a, 0x0a, 0x0a, 0x10,
    0x10, 0x10, 0x10, 0x90, 0x90, 0x90, 0x8a, 0x44, 0x42, 0x42, 0x42, 0x84, 0x82, 0x02, 0x20, 0x20,
    0x20, 0x20, 0x06, 0x06, 0x86, 0x86, 0x46, 0x46, 0x46, 0x46, 0x46, 0x06, 0x86, 0x06, 0x06, 0x06,
    0x06, 0x06, 0x06, 0x86, 0x86, 0x86, 0x46, 0x46, 0x46, 0x46, 0x46, 0x86, 0x86, 0x20, 0x20, 0x20,
    0x20, 0x20, 0x20, 0xa0, 0x80, 0x80, 0x40, 0x40, 0xa0, 0x40, 0x50, 0x90, 0x90, 0x90, 0x10, 0x10,
    0x10, 0x10, 0x10, 0x90, 0x90, 0x90, 0x50, 0x50, 0xa0, 0x48, 0x48, 0x88, 0x88, 0xa0, 0x20, 0x20,
    0x20, 0x20, 0x20, 0x20, 0x80, 0x80, 0x40, 0x40, 0x40, 0x40, 0x40, 0x80, 0x80, 0x80, 0x00, 0x00,
    0x00,
};
__device__ __forceinline__ int ray_mode(float s) {
    const int i = (int)((s - 1.0f) * 64.0f + 0.5f);
    return s <= 1.0f || i > 128 ? 0 : kRayModes[i];
}
__device__ __forceinline__ int ray_of(int mode, int lane) {
    const int k = (lane >> 1) & 3, quarter = lane >> 3, odd = lane & 1, pair = (mode >> 6) & 3, q = (mode >> 4) & 3;
    const int set = pair == 0 ? 2 * quarter + odd : pair == 1 ? (quarter & 1) + 4 * (quarter >> 1) + 2 * odd : quarter + 4 * odd;
    return q == 0 ? 4 * set + k : q == 1 ? (set & 1) + 8 * (set >> 1) + 2 * k : (set & 3) + 16 * (set >> 2) + 4 * k;
}

__device__ __forceinline__ float4 lds4(unsigned off) { return *reinterpret_cast<const float4*>(fsm + off); }

// Sums of a chunk for the lane's eight rows: p[0..1] the half it loads first (rows 4h .. 4h+3,
// h = lane & 1), p[2..3] the other.  fl: floor-voxel sums of rows without interpolation.
struct Sums {
    float2 p[4];
    float fl[8];
};

// One sample of the eight rows.  a0, b0: columns A and B of the half loaded first; a1, b1: of
// the other.  A is column floor(x) and B the next one (flip: the reverse); g is B's weight.
// Samples with in == false add nothing.
// FL 0: no row without interpolation; 1: row 7 is one (the volume's last row); 2: any may be.
template <int FL, bool FIRST>
__device__ __forceinline__ void add_tap(Sums& s, unsigned a0, unsigned b0, unsigned a1, unsigned b1, float g, bool flip,
                                        int h, bool in) {
    const float2 n = make_float2(-1.0f, -1.0f), gg = make_float2(g, g);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const float4 A = lds4(q ? a1 : a0), B = lds4(q ? b1 : b0);
        const float2 A01 = make_float2(A.x, A.y), A23 = make_float2(A.z, A.w);
        const float2 d01 = __ffma2_rn(A01, n, make_float2(B.x, B.y));
        const float2 d23 = __ffma2_rn(A23, n, make_float2(B.z, B.w));
        const float2 t01 = __ffma2_rn(gg, d01, A01), t23 = __ffma2_rn(gg, d23, A23);
        if (FIRST) {
            s.p[2 * q] = t01;
            s.p[2 * q + 1] = t23;
        } else if (in) {
            s.p[2 * q] = __fadd2_rn(s.p[2 * q], t01);
            s.p[2 * q + 1] = __fadd2_rn(s.p[2 * q + 1], t23);
        }
        if (FL == 1 && h != q && in) s.fl[7] += flip ? B.w : A.w;
        if (FL == 2 && in) {
            s.fl[4 * q] += flip ? B.x : A.x;
            s.fl[4 * q + 1] += flip ? B.y : A.y;
            s.fl[4 * q + 2] += flip ? B.z : A.z;
            s.fl[4 * q + 3] += flip ? B.w : A.w;
        }
    }
}

// Rows without interpolation take their floor sums.  flatmask: bit c = the lane's c-th row.
template <int FL>
__device__ __forceinline__ void settle(Sums& s, int flatmask, int h) {
    if (FL == 1) {
        if (h) s.p[1].y = s.fl[7];
        else s.p[3].y = s.fl[7];
    }
    if (FL == 2) {
#pragma unroll
        for (int c = 0; c < 8; c++)
            if (flatmask >> c & 1) (c & 1 ? s.p[c >> 1].y : s.p[c >> 1].x) = s.fl[c];
    }
}

struct Rows8 {
    float2 p[4];
};

struct Chunk {
    int z0, zc;       // first plane, planes
    int cb, ncols;    // first staged column, staged columns
    int ca, cw;       // first column and columns as stored
};

// A chunk that some ray of the warp enters or leaves, or that ends with the volume's last
// plane: the same sums in the same order, each sample with the reference's inside decision
// (the ray's plane interval) and its raw-voxel rules.  Branch-free, addresses clamped into the
// staged columns; about a fifth dearer per plane than a full chunk.  One in ten chunks of a
// 512 x 512 plane and one in three at 128 x 128 come here, so it is written for speed, and out
// of line to keep the ray blocks' loop short.
template <int ZC, int FL, bool BLEND>
__device__ __noinline__ Rows8 partial_chunk(unsigned buf, int pitch, Chunk c, long long x, long long step, int zab,
                                            int flip, int W, int D, int flatmask, int h) {
    Sums s;
#pragma unroll
    for (int q = 0; q < 4; q++) s.p[q] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int q = 0; q < 8; q++) s.fl[q] = 0.0f;
    const int z1 = (zab & 0xFFFF) - c.z0;
    const unsigned cnt = (unsigned)zab >> 16, most = (unsigned)max(c.ncols - 2, 0);
    const unsigned h0 = buf + (h << 4), h1 = buf + 16 - (h << 4);
#pragma unroll
    for (int zz = 0; zz < ZC; zz++, x += step) {
        int hi = (int)(x >> 32);
        // raw voxels: the last plane, the last column and beside the volume
        const bool raw = c.z0 + zz == D - 1 || (unsigned)hi >= (unsigned)(W - 1);
        if (BLEND && hi >= W - 1) hi = W;  // column W holds the last column's unblended voxel
        const bool in = (unsigned)(zz - z1) < cnt;
        float g = fix_one_plus_frac((uint32_t)x);
        g = flip ? 2.0f - g : g - 1.0f;
        if (raw) g = 1.0f;
        const unsigned o = ((unsigned)(zz * pitch) + min((unsigned)(hi - c.cb), most)) << 5;
        // a raw voxel v is 0 + 1 (v - 0): exact, and no other column can make it NaN
        const unsigned oa = raw ? kZeroOff - buf : o + (flip ? 32u : 0u), ob = o + (flip || raw ? 0u : 32u);
        add_tap<FL, false>(s, h0 + oa, h0 + ob, h1 + oa, h1 + ob, g, flip || raw, h, in);
    }
    settle<FL>(s, flatmask, h);
    return Rows8{{s.p[0], s.p[1], s.p[2], s.p[3]}};
}

template <int VT>
__device__ __forceinline__ float load_voxel(const void* p, size_t o) {
    if (VT == kVolF32) return static_cast<const float*>(p)[o];
    return vol_load16<VT>(static_cast<const uint16_t*>(p)[o]);
}

__device__ __forceinline__ void cp_async4(unsigned dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(fsm) + dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One CTA's work.  jb: first of the eight projection rows; seg, win, g0: plane segment,
// column window and first tilt.  Returns false when a bounded wait ran out (recorded in the
// status word; nothing in flight).  `retire` as in fp_body.
// EB: bytes of a stored voxel (4: FP32, 2: BF16 or FP16).
template <int ZC, int EB, bool BLEND>
__device__ __forceinline__ bool fpr_body(const FpLaunch& a, const int g0, const int jb, const int seg, const int win,
                                         const bool retire = false) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int half = lane & 1;
    const int W = a.W, H = a.H, D = a.D, w = a.w;
    const int TG = min(a.tilts_per_cta, a.T - g0);
    const int NB = (w + kRays - 1) / kRays;
    const int pitch = a.rv.pitch;
    const int z_lo = seg * a.rv.seg, z_hi = min(D, z_lo + a.rv.seg);
    const int zm = (z_lo + z_hi) >> 1;
    const int nch = (z_hi - z_lo + ZC - 1) / ZC;
    BlockInfo* s_info = reinterpret_cast<BlockInfo*>(fsm + kInfoOff);
    int* s_zab = reinterpret_cast<int*>(fsm + kZabOff);
    long long* s_step = reinterpret_cast<long long*>(fsm + kStepOff);
    int* s_tilt = reinterpret_cast<int*>(fsm + kTiltOff);
    int* s_mode = reinterpret_cast<int*>(fsm + kModeOff);
    int* s_cnt = reinterpret_cast<int*>(fsm + kCntOff);
    int* s_width = reinterpret_cast<int*>(fsm + kWidthOff);
    int* s_row = reinterpret_cast<int*>(fsm + kRowOff);
    float* s_yf = reinterpret_cast<float*>(fsm + kRowOff + 32);
    int* s_base = reinterpret_cast<int*>(fsm + kRowOff + 64);
    uint16_t* s_list = reinterpret_cast<uint16_t*>(fsm + kListOff);
    uint64_t* bar = reinterpret_cast<uint64_t*>(fsm);
    // two chunks of transposed planes [ZC][pitch][8 rows], and the coming chunk's rows as stored
    const unsigned bufbytes = (unsigned)(ZC * pitch) << 5;
    const unsigned raw = kBufOff + 2 * bufbytes;
    constexpr int AL = 16 / EB;
    const int use_tma = a.rv.bulk;
    const int use_async = !use_tma && EB == 4;

    const size_t plane = (size_t)H * W;
    const int r0 = jb - a.row_off;  // whole rows: r0 .. r0 + 7; the lane's first four start at half * 4
    if (BLEND && tid < 8) {
        const int j = jb + tid;
        const int r = (j >= a.j0 && j < a.j1) ? a.rowmap[j] : -1;
        s_row[tid] = max(r, 0);
        s_yf[tid] = (r >= 0 && r < H - 1) ? a.rowyf[j] : 0.0f;
        // volume rows the group reads: [rb, rb + nr) (rows outside the volume read row 0's place)
        int lo = r >= 0 ? r : INT_MAX, hi = r;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffu, hi, o));
        }
        if (lo > hi) lo = hi = 0;
        s_row[tid] = max(r, lo) - lo;
        if (tid == 0) {
            s_base[0] = lo;
            s_base[1] = min(min(hi + 1, H - 1) - lo + 1, a.rv.rawrows);
        }
    }
    if (tid < 8) *reinterpret_cast<float*>(fsm + kZeroOff + 4 * tid) = 0.0f;
    if (use_tma && tid == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    // volume rows staged: rb .. rb + nr - 1
    const int rb = BLEND ? s_base[0] : r0, nr = BLEND ? s_base[1] : 8;
    const int rawrows = a.rv.rawrows;
    auto stage = [&](const Chunk& k, bool held) {
        const int ca = k.ca, cw = k.cw;
        if (use_tma) {
            // spread over the warps: a bulk copy takes tens of issue cycles
            const uint32_t nb = (uint32_t)cw * EB;
            const int n = nr * k.zc, per = (n + kWarps - 1) / kWarps;
            if (lane < per || tid == 0) fence_proxy_async();
            if (tid == 0) mbar_arrive_expect_tx(bar, nb * (uint32_t)n);
            for (int e = warp * per + lane; e < min((warp + 1) * per, n) && nb > 0 && !held; e += 32) {
                const int zz = e / nr, q = e - zz * nr;
                const int r = min(max(rb + q, 0), H - 1);
                const size_t o = ((size_t)(k.z0 + zz) * plane + (size_t)r * W + ca) * EB;
                tma_load_1d(fsm + raw + (unsigned)((zz * rawrows + q) * pitch) * EB,
                            static_cast<const unsigned char*>(a.vol) + o, nb, bar);
            }
        } else if (use_async) {
            for (int e = warp; e < nr * k.zc; e += kWarps) {
                const int zz = e / nr, q = e - zz * nr;
                const int r = min(max(rb + q, 0), H - 1);
                const float* src = static_cast<const float*>(a.vol) + (size_t)(k.z0 + zz) * plane + (size_t)r * W + ca;
                const unsigned dst = raw + (unsigned)((zz * rawrows + q) * pitch) * 4u;
                for (int x = lane; x < cw; x += 32) cp_async4(dst + 4u * x, src + x);
            }
        }
    };
    // the first chunk's copies go out at once where its columns are known (no windows): they
    // cover the block lists' global loads
    const bool hold0 = a.hold_first_copy != 0;
    if (a.rv.nwin == 1) stage(Chunk{z_lo, min(ZC, z_hi - z_lo), -1, W + 3, 0, W}, hold0);
    // --- ray blocks of this segment and window, one warp per tilt --------------------------
    const int wlo = win == 0 ? INT_MIN : win * a.rv.xw;
    const int whi = win == a.rv.nwin - 1 ? INT_MAX : (win + 1) * a.rv.xw;
    if (warp < TG) {
        const int tilt = a.tilts[g0 + warp];
        const long long step = a.ftilt[tilt].step;
        const long long first = a.rays[(size_t)tilt * w].X0, last = a.rays[(size_t)tilt * w + w - 1].X0;
        const long long space = w > 1 ? (last - first) / (w - 1) : 0, span = (kRays - 1) * space;
        const long long sa = min(step * z_lo, step * (z_hi - 1)), sb = max(step * z_lo, step * (z_hi - 1));
        int n = 0;
        for (int b0 = 0; b0 < NB; b0 += 32) {
            // (positions to a few units of 2^-32 column: the tests have a column to spare)
            const int b = b0 + lane;
            const long long x0 = first + (long long)(kRays * b) * space, x1 = x0 + span;
            const int xm = (int)((x0 + step * zm) >> 32);
            const int lo = (int)((min(x0, x1) + sa) >> 32), hi = (int)((max(x0, x1) + sb) >> 32);
            const bool in = b < NB && xm >= wlo && xm < whi && hi >= -2 && lo <= W + 1;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (in) s_list[warp * kMaxNB + n + __popc(m & ((1u << lane) - 1))] = (uint16_t)b;
            n += __popc(m);
        }
        if (lane == 0) {
            s_step[warp] = step;
            s_tilt[warp] = tilt;
            s_mode[warp] = ray_mode(fabsf((float)space * (1.0f / 4294967296.0f)));
            s_width[warp] = (int)(span >> 32);
            s_cnt[warp] = n;
        }
    }
    __syncthreads();
    if (tid == 0) {
        int run = 0;
        for (int t = 0; t < TG; t++) {
            const int n = s_cnt[t];
            s_cnt[t] = run;
            run += n;
        }
        s_cnt[TG] = run;
    }
    // columns of every chunk: staged [cb, cb + ncols), as stored [ca, ca + cw) (bulk copies on
    // 16-byte boundaries)
    int4* s_chunk = reinterpret_cast<int4*>(fsm + kChunkOff);
    if (tid < nch) {
        const int z0 = z_lo + tid * ZC, zc = min(ZC, z_hi - z0);
        int cb = -1, ncols = W + 3;
        if (a.rv.nwin > 1) {
            long long lo = LLONG_MAX, hi = LLONG_MIN;
            int wneg = 0, wpos = 0;
            for (int t = 0; t < TG; t++) {
                const long long m0 = (z0 - zm) * s_step[t], m1 = (z0 + zc - 1 - zm) * s_step[t];
                lo = min(lo, min(m0, m1));
                hi = max(hi, max(m0, m1));
                wneg = min(wneg, s_width[t] - 1);
                wpos = max(wpos, s_width[t] + 1);
            }
            cb = win == 0 ? -1 : min(max(-1, wlo + (int)(lo >> 32) + wneg - 1), W);
            const int ce = win == a.rv.nwin - 1 ? W + 1 : min(W + 1, whi + (int)(hi >> 32) + wpos + 2);
            ncols = min(max(ce - cb + 1, 0), pitch);
        }
        const int al = use_tma ? AL - 1 : 0, ca = max(cb, 0) & ~al;
        s_chunk[tid] = make_int4(cb, ncols, ca, max(min(W, (cb + ncols + al) & ~al) - ca, 0));
    }
    int flatmask = 0;
    bool any_flat = false;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int j = jb + q;
        const int r = BLEND ? (j >= a.j0 && j < a.j1 ? a.rowmap[j] : -1) : r0 + q;
        if (r == H - 1) {
            any_flat = true;
            flatmask |= 1 << (q ^ (half << 2));
        }
    }
    __syncthreads();

    auto chunk_of = [&](int c) {
        const int4 q = s_chunk[c];
        const int z0 = z_lo + c * ZC;
        return Chunk{z0, min(ZC, z_hi - z0), q.x, q.y, q.z, q.w};
    };
    const int nblk = s_cnt[TG];
    if (nblk == 0) {  // no ray comes near: the first chunk's copies, if any, land before the CTA ends
        bool ok = true;
        if (a.rv.nwin == 1) {
            if (use_async) cp_async_wait_all();
            if (use_tma && !hold0) ok = mbar_wait_bounded(bar, 0, kWaitTries);
        }
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicOr(a.status, kStatusTimeout);
            return false;
        }
        if (retire && use_tma && tid == 0) mbar_inval(bar);
        return true;
    }
    if (a.rv.nwin > 1) stage(chunk_of(0), hold0);
    // raw rows -> [plane][column][8 rows]; a thread writes four rows of a column in every plane
    auto transpose = [&](const Chunk& k, unsigned buf) {
        const int ca = k.ca;
        auto column = [&](int col, int z0, int z1) {
            const int xc = k.cb + col, x = min(max(xc, 0), W - 1);
            unsigned dst = buf + ((unsigned)(z0 * pitch + col) << 5) + half * 16;
            if (BLEND) {
                for (int zz = z0; zz < z1; zz++, dst += (unsigned)pitch << 5) {
                    const bool flat = xc >= W || k.z0 + zz == D - 1;
                    float v[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const float yf = s_yf[half * 4 + c];
                        const float* p = reinterpret_cast<const float*>(fsm + raw) +
                                         (zz * rawrows + s_row[half * 4 + c]) * pitch + (x - ca);
                        v[c] = p[0];
                        if (yf != 0.0f && !flat) v[c] = __fadd_rn(v[c], __fmul_rn(yf, __fsub_rn(p[pitch], v[c])));
                    }
                    *reinterpret_cast<float4*>(fsm + dst) = make_float4(v[0], v[1], v[2], v[3]);
                }
            } else if (use_tma || use_async) {
                const unsigned rp = (unsigned)pitch * EB;
                const unsigned src = raw + (unsigned)(z0 * 8 + half * 4) * rp + (unsigned)(x - ca) * EB;
                auto planes = [&](auto vtc) {
                    constexpr int VT = decltype(vtc)::value;
                    unsigned so = src, d = dst;
#pragma unroll 4
                    for (int zz = z0; zz < z1; zz++, d += (unsigned)pitch << 5, so += 8 * rp) {
                        const float v0 = load_voxel<VT>(fsm + so, 0), v1 = load_voxel<VT>(fsm + so + rp, 0);
                        const float v2 = load_voxel<VT>(fsm + so + 2 * rp, 0), v3 = load_voxel<VT>(fsm + so + 3 * rp, 0);
                        *reinterpret_cast<float4*>(fsm + d) = make_float4(v0, v1, v2, v3);
                    }
                };
                if (EB == 4) planes(std::integral_constant<int, kVolF32>{});
                else if (a.vtype == kVolBF16) planes(std::integral_constant<int, kVolBF16>{});
                else planes(std::integral_constant<int, kVolF16>{});
            } else if (EB == 2) {  // rows off 16-byte boundaries: read where they are used
                for (int zz = z0; zz < z1; zz++, dst += (unsigned)pitch << 5) {
                    float v[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const int r = min(max(r0 + half * 4 + c, 0), H - 1);
                        v[c] = vol_load16_rt(a.vtype, static_cast<const uint16_t*>(a.vol)[(size_t)(k.z0 + zz) * plane + (size_t)r * W + x]);
                    }
                    *reinterpret_cast<float4*>(fsm + dst) = make_float4(v[0], v[1], v[2], v[3]);
                }
            }
        };
        // the columns inside the volume, then the repeated ones at its edges (spread over the
        // planes: there are at most three)
        const int in0 = max(k.cb, 0) - k.cb, in1 = min(k.ncols, W - k.cb);
        for (int col = in0 + (tid >> 1); col < in1; col += kThreads / 2) column(col, 0, k.zc);
        const int edges = in0 + max(k.ncols - in1, 0);
        for (int e = tid >> 1; e < edges * k.zc; e += kThreads / 2) {
            const int n = e / k.zc, zz = e - n * k.zc;
            column(n < in0 ? n : in1 + n - in0, zz, zz + 1);
        }
    };
    uint32_t phase = 0;  // chunks staged so far, over all passes

    for (int p0 = 0; p0 < nblk; p0 += kCap) {
        // --- this pass's blocks: slot k of a warp is block p0 + k * kWarps + warp -----------
        const int np = min(kCap, nblk - p0);
        // slot k of warp v: neighbouring blocks leave the volume together, so the warps' order
        // rotates from slot to slot
        for (int e = tid; e < kCap; e += kThreads) {
            const int k = e / kWarps, q = p0 + min(k * kWarps + ((e + 5 * k) & (kWarps - 1)), np - 1);
            int t = 0;
            while (t + 1 < TG && s_cnt[t + 1] <= q) t++;
            const int b = s_list[t * kMaxNB + q - s_cnt[t]];
            BlockInfo bi;
            bi.step = s_step[t];
            bi.span = s_step[t] * (ZC - 1);
            bi.id = (t << 16) | b;
            bi.mode = s_mode[t];
            s_info[e] = bi;
        }
        __syncthreads();
        float2 acc[kSlots][4];
        long long X[kSlots];  // position at the current chunk's first plane
        unsigned flips = 0;   // bit k: the lane's ray of slot k loads column floor(x) + 1 first
        // slots in use: only the last row of blocks can be short
        int ns = 0;
#pragma unroll
        for (int k = 0; k < kSlots; k++) ns += k * kWarps + ((warp + 5 * k) & (kWarps - 1)) < np;
        const BlockInfo* info = s_info + warp;
        int* zabs = s_zab + warp * 32 + lane;
#pragma unroll
        for (int k = 0; k < kSlots; k++) {
#pragma unroll
            for (int c = 0; c < 4; c++) acc[k][c] = make_float2(0.0f, 0.0f);
            // (every slot loads: one past the warp's last repeats a block; rays past the
            // detector's last column repeat it)
            const BlockInfo& bi = info[k * kWarps];
            const int t = bi.id >> 16, i = min(kRays * (bi.id & 0xFFFF) + ray_of(bi.mode, lane), w - 1);
            const FpRay ray = a.rays[(size_t)s_tilt[t] * w + i];
            X[k] = ray.X0 + bi.step * z_lo;
            zabs[k * kThreads] = ray.zab;  // read back by this lane only
            flips |= (unsigned)((bi.mode >> ((lane >> 1) & 3)) & 1) << k;
        }
        const bool held = hold0 && p0 == 0;
        // the coming chunk's rows have landed and every thread may read them
        auto arrived = [&](bool hold) -> bool {
            bool ok = true;
            if (use_tma) ok = mbar_wait_bounded(bar, phase & 1, hold ? kHoldWaitTries : kWaitTries);
            else if (use_async) {
                cp_async_wait_all();
                __syncthreads();
            }
            phase++;
            return ok;
        };
        auto give_up = [&](bool hold) {
            if (tid == 0) atomicOr(a.status, kStatusTimeout);
            // let any copy still in flight land before the CTA's shared memory is released
            if (!hold) mbar_wait_bounded(bar, (phase - 1) & 1, kWaitTries);
        };
        Chunk cur = chunk_of(0);
        if (p0 > 0) stage(cur, false);
        bool ok = arrived(held);
        if (ok) transpose(cur, kBufOff);
        if (__syncthreads_or(!ok)) {
            give_up(held);
            return false;
        }
        if (nch > 1) stage(chunk_of(1), false);
        // --- chunks: sample, then transpose the next one into the other buffer (a warp that is
        // done early starts on it while others sample) and issue the copies of the one after --
        for (int c = 0; c < nch; c++) {
            const unsigned buf = kBufOff + (c & 1 ? bufbytes : 0u);
            // floors of full-chunk samples: [Lb, Lb + Lw), both columns staged and inside; the
            // volume's last plane (raw voxels) is left to partial_chunk
            const int Lb = max(cur.cb, 1);
            const unsigned Lw = cur.z0 + ZC < D ? (unsigned)max(min(cur.cb + cur.ncols - 1, W - 1) - Lb, 0) : 0u;
            const unsigned base = buf - ((unsigned)cur.cb << 5), base0 = base + (half << 4), base1 = base + 16 - (half << 4);
            auto slot = [&](int k, auto flc) {
                constexpr int FL = decltype(flc)::value;
                const BlockInfo& bi = info[k * kWarps];
                const long long step = bi.step, x0 = X[k], x1 = x0 + bi.span;
                X[k] = x1 + step;
                const int h0 = (int)(x0 >> 32), h1 = (int)(x1 >> 32);
                const bool full = (unsigned)(h0 - Lb) < Lw && (unsigned)(h1 - Lb) < Lw;
                const int flip = (flips >> k) & 1;
                if (__all_sync(0xffffffffu, full)) {
                    const unsigned fa = flip * 32, fb = 32 - fa;
                    const unsigned a0 = base0 + fa, b0 = base0 + fb, a1 = base1 + fa, b1 = base1 + fb;
                    const float sg = flip ? -1.0f : 1.0f, cg = flip ? 2.0f : -1.0f;
                    Sums s;
#pragma unroll
                    for (int q = 0; q < 8; q++) s.fl[q] = 0.0f;
                    const long long sp = step + ((long long)pitch << 32);
                    long long x = x0;
#pragma unroll
                    for (int zz = 0; zz < ZC; zz++, x += sp) {
                        const unsigned o = (unsigned)(x >> 32) << 5;
                        const float g = fmaf(fix_one_plus_frac((uint32_t)x), sg, cg);
                        if (zz == 0) add_tap<FL, true>(s, a0 + o, b0 + o, a1 + o, b1 + o, g, flip, half, true);
                        else add_tap<FL, false>(s, a0 + o, b0 + o, a1 + o, b1 + o, g, flip, half, true);
                    }
                    settle<FL>(s, flatmask, half);
#pragma unroll
                    for (int q = 0; q < 4; q++) acc[k][q] = __fadd2_rn(acc[k][q], s.p[q]);
                } else if (!__all_sync(0xffffffffu, (h0 < -1 && h1 < -1) || (h0 > W && h1 > W))) {
                    const Rows8 s = partial_chunk<ZC, FL, BLEND>(buf, pitch, cur, x0, step, zabs[k * kThreads], flip, W,
                                                                 D, flatmask, half);
#pragma unroll
                    for (int q = 0; q < 4; q++) acc[k][q] = __fadd2_rn(acc[k][q], s.p[q]);
                }
            };
            auto run = [&](auto flc) {
#pragma unroll
                for (int k = 0; k < kSlots; k++) {
                    if (k >= ns) break;
                    slot(k, flc);
                }
            };
            if (!any_flat) run(std::integral_constant<int, 0>{});
            else run(std::integral_constant<int, BLEND ? 2 : 1>{});
            if (c + 1 < nch) {
                cur = chunk_of(c + 1);
                ok = arrived(false);
                if (ok) transpose(cur, kBufOff + (c & 1 ? 0u : bufbytes));
            }
            if (__syncthreads_or(!ok)) {
                give_up(false);
                return false;
            }
            if (c + 2 < nch) stage(chunk_of(c + 2), false);
        }
        // --- segment sums -------------------------------------------------------------------
#pragma unroll
        for (int k = 0; k < kSlots; k++) {
            if (k >= ns) break;
            const BlockInfo& bi = info[k * kWarps];
            const int t = bi.id >> 16, i = kRays * (bi.id & 0xFFFF) + ray_of(bi.mode, lane);
            if (i >= w) continue;
            float* o = a.part + (((size_t)seg * a.T + g0 + t) * a.h) * w + i;
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const int q = c ^ (half << 2), j = jb + q;
                const bool ok = j >= a.j0 && j < a.j1 && (BLEND || (unsigned)(r0 + q) < (unsigned)H);
                if (ok) o[(size_t)j * w] = c & 1 ? acc[k][c >> 1].y : acc[k][c >> 1].x;
            }
        }
        __syncthreads();  // the block lists are free for the next pass
    }
    if (retire && use_tma && tid == 0) mbar_inval(bar);  // every phase has completed
    return true;
}

// CTA order: the tilt groups of a (window, row group, segment) side by side, so that its
// columns are read from L2 by all but the first.
template <int ZC, int EB, bool BLEND>
__global__ void __launch_bounds__(kThreads, 1) fpr_kernel(const __grid_constant__ FpLaunch a) {
    const int ntg = gridDim.x / a.rv.nwin, win = blockIdx.x / ntg, tg = blockIdx.x - win * ntg;
    fpr_body<ZC, EB, BLEND>(a, tg * a.tilts_per_cta, a.rv.jfirst + 8 * blockIdx.y, blockIdx.z, win);
}

// Batched form: CTA b works on item {problem, first tilt | window << 16, first row, segment}.
template <int ZC, int EB>
__global__ void __launch_bounds__(kThreads, 1)
    fpr_kernel_batch(const FpLaunch* __restrict__ descs, const int4* __restrict__ items) {
    const int4 it = items[blockIdx.x];
    fpr_body<ZC, EB, false>(descs[it.x], it.y & 0xFFFF, it.z, it.w, it.y >> 16);
}

// Persistent batched form: resident CTAs take items in list order through an atomic cursor
// until the list runs out, whatever the members' chunk depths.  A bounded wait that runs
// out ends the CTA (recorded in the problem's status word).
template <int ZC, int EB>
__device__ __noinline__ bool fpr_item(const FpLaunch* a, int4 it) {
    return fpr_body<ZC, EB, false>(*a, it.y & 0xFFFF, it.z, it.w, it.y >> 16, true);
}

template <int ZC, int EB, bool BLEND>
cudaError_t attr_one() {
    return cudaFuncSetAttribute(fpr_kernel<ZC, EB, BLEND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFprSmemMax);
}

template <int ZC>
cudaError_t attr_zc() {
    cudaError_t e;
    if ((e = attr_one<ZC, 4, false>()) != cudaSuccess) return e;
    if ((e = attr_one<ZC, 4, true>()) != cudaSuccess) return e;
    if ((e = attr_one<ZC, 2, false>()) != cudaSuccess) return e;
    const int m = (int)kFprSmemMax;
    if ((e = cudaFuncSetAttribute(fpr_kernel_batch<ZC, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, m)) != cudaSuccess)
        return e;
    return cudaFuncSetAttribute(fpr_kernel_batch<ZC, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
}

template <int ZC>
cudaError_t launch_zc(const FpLaunch& a, dim3 grid, size_t smem, cudaStream_t s) {
    if (a.two_rows) fpr_kernel<ZC, 4, true><<<grid, kThreads, smem, s>>>(a);
    else if (a.vtype == kVolF32) fpr_kernel<ZC, 4, false><<<grid, kThreads, smem, s>>>(a);
    else fpr_kernel<ZC, 2, false><<<grid, kThreads, smem, s>>>(a);
    return cudaGetLastError();
}

template <int ZC>
cudaError_t launch_batch_zc(int eb, const FpLaunch* descs, const int4* items, int n, size_t smem, cudaStream_t s) {
    if (eb == 4) fpr_kernel_batch<ZC, 4><<<n, kThreads, smem, s>>>(descs, items);
    else fpr_kernel_batch<ZC, 2><<<n, kThreads, smem, s>>>(descs, items);
    return cudaGetLastError();
}

}  // namespace fpr
}  // namespace tomo

// One translation unit per chunk depth defines these entry points.
#define TOMO_FPR_INSTANTIATE(ZC)                                                                            \
    namespace tomo {                                                                                        \
    cudaError_t fpr_attr_z##ZC() { return fpr::attr_zc<ZC>(); }                                             \
    cudaError_t fpr_launch_z##ZC(const FpLaunch& a, dim3 grid, size_t smem, cudaStream_t s) {               \
        return fpr::launch_zc<ZC>(a, grid, smem, s);                                                        \
    }                                                                                                       \
    cudaError_t fpr_batch_z##ZC(int eb, const FpLaunch* d, const int4* it, int n, size_t smem, cudaStream_t s) { \
        return fpr::launch_batch_zc<ZC>(eb, d, it, n, smem, s);                                             \
    }                                                                                                       \
    }
