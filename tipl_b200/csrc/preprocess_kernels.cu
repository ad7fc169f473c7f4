// Subject preprocessing of the mm_reg pipeline on the device (reg/mm_reg.hpp:14-20,
// subject_image_pre): the separable [1 2 1] Gaussian (filter/gaussian.hpp:18-88), the
// Otsu threshold histogram, the order-preserving selection of the voxels above it,
// chunked median selection (numerical/statistics.hpp:343-363) and the final
// normalisation to uint8 (numerical/otsu.hpp:110-136).
//
// Every float expression keeps the reference's evaluation order; the device build
// does not contract multiply-adds, so results are bit-identical.
#include <algorithm>
#include "kernels.h"
#include "voxel.cuh"

namespace regb {

namespace {

// ------------------------------------------------------------------ Gaussian
// One round of the reference's x, y, z passes fused in one kernel, from any storage type.  A
// warp owns 32 columns of four rows and walks WALK planes: a plane's six rows (a halo row
// on either side) are loaded one plane ahead, x neighbours come by shuffles (the two columns
// beside the tile from lanes 0 and 31), the y pass adds rows of the thread's registers, and
// the z pass the last three planes.  Halo and edge samples come from clamped coordinates,
// which is exactly the reference's "repeat the edge sample" rule for every pass (the x pass of
// a clamped row is the x pass of the edge row).  With mm the round also finds the smallest and
// largest result.
//
// Bound by issue (some 40 instructions a voxel) and by the loads one plane ahead.  uint16
// 256x256x200 with smallest and largest value: 92 us as a widening pass, a shared-memory tile
// with three barriers and a pass for the extremes, 34 so; two planes ahead or rows by six or
// eight gave no more (48, 38, 33).
constexpr int kGx = 32, kGRows = 4, kGWarps = 4, kGThreads = 32 * kGWarps;

__device__ __forceinline__ float tap3(float l, float c, float r)
{
    // (a[left] + (a[i] + a[i])) + a[right], filter/gaussian.hpp:45-48
    return __fadd_rn(__fadd_rn(l, __fadd_rn(c, c)), r);
}

template <int DT, int WALK>
__global__ void __launch_bounds__(kGThreads) gaussian_round_kernel(const void* __restrict__ in,
                                                                   float* __restrict__ out, int w, int h, int d,
                                                                   float scale, int apply_scale,
                                                                   unsigned* __restrict__ mm)
{
    constexpr int kRows = kGRows + 2;
    const int lane = threadIdx.x & 31;
    const int x0 = blockIdx.x * kGx, y0 = (blockIdx.y * kGWarps + (threadIdx.x >> 5)) * kGRows, z0 = blockIdx.z * WALK;
    if (y0 >= h)
        return;
    const int x = x0 + lane, xc = min(x, w - 1), xh = lane == 0 ? max(x0 - 1, 0) : min(x0 + kGx, w - 1);
    const bool edge = lane == 0 || lane == 31;
    const long long wh = (long long)w * h;
    int row[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
        row[r] = min(max(y0 - 1 + r, 0), h - 1) * w;
    float c[kRows], e[kRows];
    auto load = [&](int z) {
        const void* const plane = (const char*)in + min(max(z, 0), d - 1) * wh * (DT == 0 ? 1 : DT == 1 ? 4 : 2);
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            c[r] = load_as_float<DT>(plane, (unsigned)(row[r] + xc));
            e[r] = edge ? load_as_float<DT>(plane, (unsigned)(row[r] + xh)) : 0.0f;
        }
    };
    float ring[3][kGRows];
    auto pass = [&](float (&yp)[kGRows]) {
        float xp[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            float l = __shfl_up_sync(0xffffffffu, c[r], 1), g = __shfl_down_sync(0xffffffffu, c[r], 1);
            l = lane == 0 ? e[r] : l;
            g = lane == 31 ? e[r] : g;
            xp[r] = tap3(l, c[r], g);
        }
#pragma unroll
        for (int r = 0; r < kGRows; ++r)
            yp[r] = tap3(xp[r], xp[r + 1], xp[r + 2]);
    };
    unsigned lo = 0xffffffffu, hi = 0u;
    load(z0 - 1);
    pass(ring[0]);
    load(z0);
    pass(ring[1]);
    load(z0 + 1);
    // by threes, so that the ring of planes stays in registers
    static_assert(WALK % 3 == 0, "whole turns");
    for (int k0 = 0; k0 < WALK; k0 += 3) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int z = z0 + k0 + j;
            if (z >= d)
                break;
            pass(ring[(j + 2) % 3]);
            load(z + 2);
#pragma unroll
            for (int r = 0; r < kGRows; ++r) {
                float v = tap3(ring[j][r], ring[(j + 1) % 3][r], ring[(j + 2) % 3][r]);
                if (apply_scale)
                    v = __fmul_rn(v, scale);
                if (x < w && y0 + r < h) {
                    out[z * wh + (y0 + r) * w + x] = v;
                    // (the keys of values that cannot be negative are in the order of their bits)
                    const unsigned k = DT == 0 || DT == 2 ? __float_as_uint(v) : key_of(v);
                    lo = min(lo, k);
                    hi = max(hi, k);
                }
            }
        }
    }
    if (mm) {
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) {
            constexpr unsigned sign = DT == 0 || DT == 2 ? 0x80000000u : 0u;
            atomicMin(mm, lo | sign);
            atomicMax(mm + 1, hi | sign);
        }
    }
}

// ------------------------------------------------------------------ Otsu histogram
constexpr int kPThreads = 256;

// f of every element of v, eight loads in flight; a warp's lanes take neighbours.
template <typename F>
__device__ __forceinline__ void for_each_float(const float* __restrict__ v, long long n, F f)
{
    constexpr int kLoads = 8;
    for (long long b = (long long)blockIdx.x * kLoads * kPThreads; b < n; b += (long long)gridDim.x * kLoads * kPThreads) {
        float x[kLoads];
        const long long i = b + threadIdx.x;
#pragma unroll
        for (int k = 0; k < kLoads; ++k)
            x[k] = i + k * kPThreads < n ? __ldg(v + i + k * kPThreads) : 0.0f;
#pragma unroll
        for (int k = 0; k < kLoads; ++k)
            if (i + k * kPThreads < n)
                f(x[k]);
    }
}

// hist[clamp(floor((v - mn) * range), 0, 255)]++ over the image (numerical/basic_op.hpp:
// 1293-1311), mn and mx from their keys; exact integer counts, per-block shared histograms.
// Nothing when mn < mx does not hold.
__global__ void __launch_bounds__(kPThreads) otsu_hist_kernel(const float* __restrict__ v, long long n,
                                                               const unsigned* __restrict__ mm,
                                                               unsigned* __restrict__ hist)
{
    __shared__ unsigned sh[256];
    sh[threadIdx.x] = 0u;
    __syncthreads();
    const float mn = float_of(mm[0]), mx = float_of(mm[1]);
    if (!(mn < mx))
        return;
    const float width = __fsub_rn(mx, mn), range = __fdiv_rn(256.0f, width == 0.0f ? 1.0f : width);
    for_each_float(v, n, [&](float x) {
        int b = (int)floorf(__fmul_rn(__fsub_rn(x, mn), range));
        b = b < 0 ? 0 : (b > 255 ? 255 : b);
        atomicAdd(&sh[b], 1u);
    });
    __syncthreads();
    if (sh[threadIdx.x])
        atomicAdd(&hist[threadIdx.x], sh[threadIdx.x]);
}

// ------------------------------------------------------------------ compaction
// The voxels above the threshold, in voxel order (otsu.hpp:91-95), in three steps:
// per-tile counts, an exclusive scan of the counts, and an ordered scatter.  A warp takes
// kSpan values in a row, all its loads in flight at once (256x256x200: a load at a time with
// three barriers for each 256 values 15 + 40 us, 10 + 15 so).
constexpr int kTile = 4096, kSpan = kTile / (kPThreads / 32);

// The calling thread's values of its warp's span: lane l has l, l + 32, ...; bit k of the
// result: value k is above ot.
__device__ __forceinline__ unsigned span_above(const float* __restrict__ v, long long n, float ot,
                                               float (&x)[kSpan / 32])
{
    const long long b = (long long)blockIdx.x * kTile + (threadIdx.x >> 5) * kSpan + (threadIdx.x & 31);
    unsigned keep = 0u;
#pragma unroll
    for (int k = 0; k < kSpan / 32; ++k)
        x[k] = b + 32 * k < n ? __ldg(v + b + 32 * k) : 0.0f;
#pragma unroll
    for (int k = 0; k < kSpan / 32; ++k)
        keep |= b + 32 * k < n && x[k] > ot ? 1u << k : 0u;
    return keep;
}

__global__ void __launch_bounds__(kPThreads) above_count_kernel(const float* __restrict__ v, long long n, float ot,
                                                                 unsigned* __restrict__ counts)
{
    float x[kSpan / 32];
    const unsigned c = __reduce_add_sync(0xffffffffu, (unsigned)__popc(span_above(v, n, ot, x)));
    __shared__ unsigned red[kPThreads / 32];
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned s = 0;
        for (int k = 0; k < kPThreads / 32; ++k)
            s += red[k];
        counts[blockIdx.x] = s;
    }
}

// One block: counts[i] -> exclusive prefix (in place); total in counts[nt].
__global__ void __launch_bounds__(1024) exclusive_scan_kernel(unsigned* __restrict__ counts, int nt)
{
    __shared__ unsigned carry;
    __shared__ unsigned wsum[32];
    if (threadIdx.x == 0)
        carry = 0u;
    __syncthreads();
    for (int base = 0; base < nt; base += 1024) {
        const int i = base + threadIdx.x;
        const unsigned v = i < nt ? counts[i] : 0u;
        unsigned x = v;  // inclusive warp scan
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if ((threadIdx.x & 31) >= o)
                x += y;
        }
        if ((threadIdx.x & 31) == 31)
            wsum[threadIdx.x >> 5] = x;
        __syncthreads();
        if (threadIdx.x < 32) {
            unsigned ws = wsum[threadIdx.x];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, ws, o);
                if (threadIdx.x >= o)
                    ws += y;
            }
            wsum[threadIdx.x] = ws;
        }
        __syncthreads();
        const unsigned before = carry + ((threadIdx.x >> 5) ? wsum[(threadIdx.x >> 5) - 1] : 0u) + x - v;
        if (i < nt)
            counts[i] = before;
        __syncthreads();
        if (threadIdx.x == 1023)
            carry = before + v;
        __syncthreads();
    }
    if (threadIdx.x == 0)
        counts[nt] = carry;
}

// Ordered scatter: tile b writes its values above ot from offset[b] on, in order.
__global__ void __launch_bounds__(kPThreads) above_scatter_kernel(const float* __restrict__ v, long long n, float ot,
                                                                   const unsigned* __restrict__ offset,
                                                                   float* __restrict__ out)
{
    __shared__ unsigned count[kPThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned at = offset[blockIdx.x];
    float x[kSpan / 32];
    const unsigned keep = span_above(v, n, ot, x);
    const unsigned c = __reduce_add_sync(0xffffffffu, (unsigned)__popc(keep));
    if (lane == 0)
        count[wid] = c;
    __syncthreads();
    for (int k = 0; k < wid; ++k)
        at += count[k];
#pragma unroll
    for (int k = 0; k < kSpan / 32; ++k) {
        const bool mine = keep >> k & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (mine)
            out[at + __popc(m & ((1u << lane) - 1u))] = x[k];
        at += __popc(m);
    }
}

// ------------------------------------------------------------------ chunk medians
// median(container) (numerical/statistics.hpp:343-363) over m >= 2048 values: chunk c
// of 256 is [c*cs + min(c, rem), +cs + (c < rem)); its middle is the (len/2)-th
// smallest.  One block per chunk selects it exactly by radix selection on
// order-preserving keys: all of them lie between those of the threshold and of the largest
// value, so the 2048 bins of the first pass split that range, and those of the next the bin
// found, until a bin is one key (256x256x200: over the whole key range, where the values of
// an image crowd into few bins, 55 us, 16 so).
constexpr int kMThreads = 1024, kMBins = 2048, kMLoads = 8;

__global__ void __launch_bounds__(kMThreads) chunk_median_kernel(const float* __restrict__ v,
                                                                  const unsigned* __restrict__ count, float ot,
                                                                  const unsigned* __restrict__ max_key,
                                                                  float* __restrict__ med)
{
    __shared__ unsigned hist[kMBins], part[32];
    __shared__ unsigned sel_bin, sel_rank;
    const long long m = *count;
    if (m < 2048)
        return;
    const long long cs = m / 256, rem = m % 256, c = blockIdx.x;
    const long long len = cs + (c < rem ? 1 : 0);
    const float* __restrict__ const mine = v + c * cs + (c < rem ? c : rem);
    const int t = threadIdx.x, lane = t & 31;
    unsigned rank = (unsigned)(len / 2);  // 0-based rank sought
    unsigned lo = key_of(ot);             // the keys left: lo + [0, width]
    unsigned width = *max_key - lo;
    for (;;) {
        const int shift = max(0, 32 - __clz(width) - 11);
        hist[t] = hist[t + kMThreads] = 0u;
        __syncthreads();
        for (long long i0 = t; i0 < len; i0 += kMLoads * kMThreads) {
            unsigned k[kMLoads];
#pragma unroll
            for (int j = 0; j < kMLoads; ++j)
                k[j] = i0 + j * kMThreads < len ? key_of(__ldg(mine + i0 + j * kMThreads)) - lo : 0xffffffffu;
#pragma unroll
            for (int j = 0; j < kMLoads; ++j)
                if (i0 + j * kMThreads < len && k[j] <= width)
                    atomicAdd(&hist[k[j] >> shift], 1u);
        }
        __syncthreads();
        // the bin of the sought rank: thread t owns bins 2t and 2t + 1
        const unsigned a = hist[2 * t], own = a + hist[2 * t + 1];
        unsigned x = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            x += lane >= o ? y : 0u;
        }
        if (lane == 31)
            part[t >> 5] = x;
        __syncthreads();
        if (t < 32) {
            unsigned s = part[t];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
                s += lane >= o ? y : 0u;
            }
            part[t] = s;
        }
        __syncthreads();
        const unsigned before = (t >> 5 ? part[(t >> 5) - 1] : 0u) + x - own;
        if (before <= rank && rank < before + own) {
            const bool second = rank >= before + a;
            sel_bin = 2 * t + second;
            sel_rank = rank - before - (second ? a : 0u);
        }
        __syncthreads();
        lo += sel_bin << shift;
        rank = sel_rank;
        if (shift == 0)
            break;
        width = (1u << shift) - 1u;
    }
    if (t == 0)
        med[c] = float_of(lo);
}

// ------------------------------------------------------------------ normalisation
// count of voxels with v * s > 0 (normalize_otsu_median's majority test)
__global__ void __launch_bounds__(kPThreads) positive_count_kernel(const float* __restrict__ v, long long n, float s,
                                                                    unsigned long long* __restrict__ cnt)
{
    unsigned c = 0;
    for_each_float(v, n, [&](float x) { c += __fmul_rn(x, s) > 0.0f ? 1u : 0u; });
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c)
        atomicAdd(cnt, (unsigned long long)c);
}

// out = uint8(clamp(v * s - (shift ? c : 0), 0, upper)) (otsu.hpp:126-135, then the
// float -> uint8 conversion of subject_image_pre); shift: most voxels counted in cnt, if any
__global__ void __launch_bounds__(kPThreads) otsu_normalize_kernel(const float* __restrict__ v, long long n, float s,
                                                                    const unsigned long long* __restrict__ cnt, float c,
                                                                    float upper, uint8_t* __restrict__ out)
{
    const bool shift = cnt && (double)*cnt > 0.5 * (double)n;
    auto value = [&](float x) {
        x = __fmul_rn(x, s);
        if (shift)
            x = __fsub_rn(x, c);
        x = x > upper ? upper : (x < 0.0f ? 0.0f : x);
        return (unsigned)(uint8_t)(unsigned)x;
    };
    // four voxels a thread, one store where out allows it
    const bool words = (reinterpret_cast<uintptr_t>(out) & 3) == 0;
    const float4* const q = reinterpret_cast<const float4*>(v);
    for (long long i = (long long)blockIdx.x * kPThreads + threadIdx.x; i < n / 4; i += (long long)gridDim.x * kPThreads) {
        const float4 a = __ldg(q + i);
        const unsigned b[4] = {value(a.x), value(a.y), value(a.z), value(a.w)};
        if (words)
            reinterpret_cast<unsigned*>(out)[i] = b[0] | b[1] << 8 | b[2] << 16 | b[3] << 24;
        else
            for (int k = 0; k < 4; ++k)
                out[4 * i + k] = (uint8_t)b[k];
    }
    const long long t = n / 4 * 4 + threadIdx.x;
    if (blockIdx.x == 0 && t < n)
        out[t] = (uint8_t)value(v[t]);
}

// A launch with WALK planes a warp.
template <int WALK>
cudaError_t gaussian_launch(const void* in, int dtype, float* out, int w, int h, int d, float scale, int apply_scale,
                            unsigned* mm, cudaStream_t st)
{
    const int rows = kGRows * kGWarps;
    const dim3 grid((w + kGx - 1) / kGx, (h + rows - 1) / rows, (d + WALK - 1) / WALK);
    switch (dtype) {
    case 0: gaussian_round_kernel<0, WALK><<<grid, kGThreads, 0, st>>>(in, out, w, h, d, scale, apply_scale, mm); break;
    case 1: gaussian_round_kernel<1, WALK><<<grid, kGThreads, 0, st>>>(in, out, w, h, d, scale, apply_scale, mm); break;
    case 2: gaussian_round_kernel<2, WALK><<<grid, kGThreads, 0, st>>>(in, out, w, h, d, scale, apply_scale, mm); break;
    case 3: gaussian_round_kernel<3, WALK><<<grid, kGThreads, 0, st>>>(in, out, w, h, d, scale, apply_scale, mm); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

int pgrid(long long n)
{
    return (int)std::min<long long>(std::max<long long>(n / (4 * kPThreads), 1), 148LL * 8);
}

}  // namespace

// Small volumes walk fewer planes, so that a launch is not a chain of 15 on a few SMs: 3 while
// that makes no more than three blocks an SM, 6 while no more than four.  With 3 / 6 / 15 planes:
// 16^3 to 64^3 3.1 / 4.0 / 6.7 us, 100^3 6.4 / 6.2 / 8.0, 160^3 14.0 / 12.0 / 11.9, 182x218x182
// 24.9 / 21.1 / 19.1.
cudaError_t launch_gaussian_round(const void* in, int dtype, float* out, int w, int h, int d, float scale,
                                  int apply_scale, unsigned* mm, cudaStream_t st)
{
    const long long columns = (long long)((w + kGx - 1) / kGx) * ((h + kGRows * kGWarps - 1) / (kGRows * kGWarps));
    auto launch = columns * ((d + 2) / 3) <= 148 * 3   ? gaussian_launch<3>
                  : columns * ((d + 5) / 6) <= 148 * 4 ? gaussian_launch<6>
                                                       : gaussian_launch<15>;
    return launch(in, dtype, out, w, h, d, scale, apply_scale, mm, st);
}

cudaError_t launch_otsu_hist(const float* v, long long n, const unsigned* mm, unsigned* hist, cudaStream_t st)
{
    otsu_hist_kernel<<<pgrid(n), kPThreads, 0, st>>>(v, n, mm, hist);
    return cudaGetLastError();
}

long long compact_tiles(long long n) { return (n + kTile - 1) / kTile; }

cudaError_t launch_compact_above(const float* v, long long n, float ot, unsigned* counts, float* out, cudaStream_t st)
{
    const long long nt = compact_tiles(n);
    if (nt > 0x7fffffffLL)
        return cudaErrorInvalidValue;
    above_count_kernel<<<(unsigned)nt, kPThreads, 0, st>>>(v, n, ot, counts);
    exclusive_scan_kernel<<<1, 1024, 0, st>>>(counts, (int)nt);
    above_scatter_kernel<<<(unsigned)nt, kPThreads, 0, st>>>(v, n, ot, counts, out);
    return cudaGetLastError();
}

cudaError_t launch_chunk_medians(const float* v, const unsigned* count, float ot, const unsigned* max_key, float* med,
                                 cudaStream_t st)
{
    chunk_median_kernel<<<256, kMThreads, 0, st>>>(v, count, ot, max_key, med);
    return cudaGetLastError();
}

cudaError_t launch_positive_count(const float* v, long long n, float s, unsigned long long* cnt, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess)
        return e;
    positive_count_kernel<<<pgrid(n), kPThreads, 0, st>>>(v, n, s, cnt);
    return cudaGetLastError();
}

cudaError_t launch_otsu_normalize(const float* v, long long n, float s, const unsigned long long* cnt, float c,
                                  float upper, uint8_t* out, cudaStream_t st)
{
    otsu_normalize_kernel<<<pgrid(n), kPThreads, 0, st>>>(v, n, s, cnt, c, upper, out);
    return cudaGetLastError();
}

}  // namespace regb
