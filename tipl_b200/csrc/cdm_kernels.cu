// CDM nonlinear registration passes (reg/cdm.hpp) and the displacement algebra
// they use (numerical/dif.hpp), as segment kernels: a launch covers one or more job
// levels (CdmSeg entries), each owning nblk consecutive blocks of a 1-D grid that
// stride over its voxels.
//
// One iteration of a level (reg/cdm.hpp:418-470) is the launch sequence
//   gradient (+ loop decisions in its last block) -> 12 Poisson sweeps -> theta, on a
//   level's first iteration only -> accumulate -> smooth and compose
// with a compose launch of its own ahead of the first iteration, and one ahead of the
// gradient of each further modality.  The reference's host-side decisions (cost
// bookkeeping, cdm_improved, the smoothing schedule, best_d save/restore, theta, the
// iteration cap) run on the device against CdmCtl, so a level runs without any host round
// trip; every kernel of an iteration reads ctl->done and returns once a level has left its
// loop.  best_d's save and restore move no data: the field has two buffers, and CdmCtl says
// which one holds the best field and which the current one (128^3: the copies took up to 40
// us of an iteration of 330).
#include <algorithm>
#include <atomic>
#include <cfloat>
#include "common.cuh"
#include "stats.h"

namespace regb {

constexpr int kCdmThreads = 256;

int cdm_blocks_for(long long nvox)
{
    long long b = (nvox + kCdmThreads - 1) / kCdmThreads;
    if (b > 148 * 8)
        b = 148 * 8;
    return (int)(b < 1 ? 1 : b);
}

// The segment entry a block of a launch over nseg entries works on: the last one
// whose first block <= blockIdx.x.  Every warp finds it on its own with one ballot per 32
// entries (all lanes active: this runs first in each kernel); a launch of one entry
// reads nothing to find it.
// FIRST: the numbering of the launch's grid.
template <int CdmSeg::*FIRST>
__device__ __forceinline__ int seg_of_block(const CdmSeg* __restrict__ segs, int nseg)
{
    if (nseg <= 1)
        return 0;
    const int b = (int)blockIdx.x, lane = threadIdx.x & 31;
    int k = 0;
    for (int base = 0; base < nseg; base += 32) {
        const int i = base + lane;
        const unsigned m = __ballot_sync(0xffffffffu, i < nseg && segs[i].*FIRST <= b);
        k += __popc(m);
        if (m != 0xffffffffu)
            break;
    }
    return k - 1;
}

// MULTI: the kernel's instantiation for launches over several entries; a launch of one
// entry takes the other, which has no lookup in its code at all and the entry as a kernel
// argument (`one`): a trip to memory less before its first load, 0.3 us of a launch.
// The standalone compose and accumulate read the entry from memory all the same: what their long
// loops use of it is in registers then (512x512x400 compose 1010 / 938 us, accumulate 2365 /
// 2150), and the trip counts for nothing.
#define SEG_ARGS const CdmSeg *__restrict__ segs, int nseg, const __grid_constant__ CdmSeg one
#define SEG_OF(blk0) (MULTI ? segs[seg_of_block<&CdmSeg::blk0>(segs, nseg)] : one)
#define SEG_BEGIN                                                  \
    const CdmSeg& S = SEG_OF(blk0);                               \
    SEG_LOOP
#define SEG_LOOP                                                   \
    const int blk = (int)blockIdx.x - (MULTI ? S.blk0 : 0);        \
    if (blk >= S.nblk)                                             \
        return;                                                    \
    const Dim3 D{S.w, S.h, S.d};                                   \
    const long long n = D.n();                                     \
    const long long stride = (long long)S.nblk * blockDim.x;       \
    const long long first = (long long)blk * blockDim.x + threadIdx.x;

// Where voxel i's x component sits in the fields (field, new_d, aux_d, tmp_d): component
// planes of padded rows, or interleaved xyz; y and z follow at a stride of update_comp.
__device__ __forceinline__ long long update_index(const CdmSeg& S, long long i)
{
    if (!S.planar)
        return 3 * i;
    return i + (long long)((unsigned)i / (unsigned)S.w) * (S.ppitch - S.w);
}
// the same of voxel x of row r = z * h + y
__device__ __forceinline__ long long update_index(const CdmSeg& S, long long r, int x)
{
    return S.planar ? r * S.ppitch + x : 3 * (r * S.w + x);
}
__device__ __forceinline__ long long update_comp(const CdmSeg& S) { return S.planar ? S.pplane : 1; }

// Fields whose offsets in bytes fit 32 bits and whose coordinates are exact floats: the
// sampling loops then need one add an address, and no conversion unit.
__device__ __forceinline__ bool narrow(const CdmSeg& S)
{
    return S.pplane < (1LL << 30) && max(S.w, max(S.h, S.d)) < (1 << 22);
}
// The cell of a point inside such a field: f[axis] = its two corners' coordinates, the weights
// as trilinear_cell forms them; returns its first corner's offset in rows of `pitch`.
__device__ __forceinline__ unsigned narrow_cell(float x, float y, float z, unsigned pitch, unsigned h, float (&f)[3][2],
                                                float (&r)[8])
{
    int ix, iy, iz;
    f[0][0] = floor_pos(x, ix);
    f[1][0] = floor_pos(y, iy);
    f[2][0] = floor_pos(z, iz);
#pragma unroll
    for (int k = 0; k < 3; ++k)
        f[k][1] = f[k][0] + 1.0f;
    const float p0 = x - f[0][0], p1 = y - f[1][0], p2 = z - f[2][0];
    const float n0 = 1.0f - p0, n1 = 1.0f - p1, n2 = 1.0f - p2;
    const float n0n1 = n0 * n1, p0n1 = p0 * n1, n0p1 = n0 * p1, p0p1 = p0 * p1;
    r[0] = n0n1 * n2;
    r[1] = p0n1 * n2;
    r[2] = n0p1 * n2;
    r[3] = p0p1 * n2;
    r[4] = n0n1 * p2;
    r[5] = p0n1 * p2;
    r[6] = n0p1 * p2;
    r[7] = p0p1 * p2;
    return ((unsigned)iz * h + (unsigned)iy) * pitch + (unsigned)ix;
}

// ------------------------------------------------------------------ compose
// compose_displacement (numerical/dif.hpp:90-107, 260-285): Js = Is[mod] where the
// displacement is exactly zero, else the trilinear sample at x + d; failed
// samples are 0.  2-D: vector<2> field, bilinear sample at (x + dx, y + dy).
template <typename T>
__device__ __forceinline__ T compose_moved(const T* __restrict__ Is, const Dim3& D, int ndim, int x, int y, int z, float dx,
                                           float dy, float dz)
{
    const float px = (float)x + dx, py = (float)y + dy;
    T v = T(0);
    if (ndim == 2) {
        Cell2 c;
        if (bilinear_cell(D, px, py, c))
            v = assign_pix<T>(cell_sum2(Is, D, c));
    } else {
        Cell c;
        if (trilinear_cell(D, px, py, (float)z + dz, c))
            v = assign_pix<T>(cell_sum(Is, D, c));
    }
    return v;
}
template <typename T>
__device__ __forceinline__ T compose_pixel(const T* __restrict__ Is, const Dim3& D, int ndim, int i, int x, int y, int z,
                                           float dx, float dy, float dz)
{
    if (dx == 0.0f && dy == 0.0f && (ndim == 2 || dz == 0.0f))
        return __ldg(Is + i);
    return compose_moved(Is, D, ndim, x, y, z, dx, dy, dz);
}

// The same in 3-D for a voxel of a narrow() level.
__device__ __forceinline__ float pix_float(const uint8_t* p) { return u8_to_f(__ldg(p)); }
__device__ __forceinline__ float pix_float(const float* p) { return __ldg(p); }
template <typename T>
__device__ __forceinline__ T compose_narrow(const T* __restrict__ Is, const SampleGeo& G, unsigned i, int x, int y, int z,
                                            float dx, float dy, float dz)
{
    if (dx == 0.0f && dy == 0.0f && dz == 0.0f)
        return __ldg(Is + i);
    const float px = u8_to_f(x) + dx, py = u8_to_f(y) + dy, pz = u8_to_f(z) + dz;
    if ((px < 0.0f || py < 0.0f || pz < 0.0f) || !(px < G.wl && py < G.hl && pz < G.dl))
        return T(0);
    float f[3][2], r[8], acc = 0.0f;
    const unsigned b = narrow_cell(px, py, pz, (unsigned)G.w, (unsigned)G.h, f, r);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const unsigned off = (b + (k >> 1 & 1) * G.w + (k >> 2) * G.wh) * (unsigned)sizeof(T);
        const float v = pix_float((const T*)((const char*)Is + off) + (k & 1));
        acc = k ? acc + v * r[k] : v * r[k];
    }
    return assign_pix<T>(acc);
}

// PLANAR: the field's layout, known here to keep its index arithmetic out of the loop, as the
// dimension is (interleaved, 2048x2048x1: 24.5 us with both looked up for each voxel, 18.7 so;
// 256x256x200 127 / 119).
template <typename T, bool MULTI, bool PLANAR>
__global__ void __launch_bounds__(kCdmThreads) cdm_compose_kernel(SEG_ARGS, int mod)
{
    const CdmSeg& S = segs[MULTI ? seg_of_block<&CdmSeg::blk0>(segs, nseg) : 0];
    SEG_LOOP
    if (S.ctl->done || mod >= max(S.nmod, 1))
        return;
    const T* __restrict__ Is = (const T*)S.Is[mod];
    T* __restrict__ Js = (T*)S.Js;
    const float* __restrict__ f = S.field[S.ctl->cur];
    const long long cs = PLANAR ? S.pplane : 1;
    auto pixels = [&](int ndim) {
        for (long long i = first; i < n; i += stride) {
            const long long o = PLANAR ? update_index(S, i) : 3 * i;
            const float dx = f[o], dy = f[o + cs], dz = ndim == 2 ? 0.0f : f[o + 2 * cs];
            T v;
            if (dx == 0.0f && dy == 0.0f && dz == 0.0f)
                v = Is[i];
            else {
                int x, y, z;
                unflat((int)i, D, x, y, z);
                v = compose_moved(Is, D, ndim, x, y, z, dx, dy, dz);
            }
            Js[i] = v;
        }
    };
    if (S.ndim == 2)
        pixels(2);
    else
        pixels(3);
}

__device__ void control_block(const CdmSeg& S, int mod);
__device__ __forceinline__ bool last_block_of_segment(const CdmSeg& S);

// ------------------------------------------------------------------ gradient
// x / m rounded like the division, for the window sizes m <= 125 and r = RN(1 / m): the
// quotient from the reciprocal, corrected twice by its exact remainder.  With r correctly
// rounded and the first correction within an ulp, the second rounds correctly (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).  An
// infinite x makes the remainder NaN; the division itself settles those.
__device__ __forceinline__ double div_window(double x, double m, double r)
{
    double q = x * r;
    q = __fma_rn(__fma_rn(-q, m, x), r, q);
    q = __fma_rn(__fma_rn(-q, m, x), r, q);
    return q == q ? q : x / m;
}

// The regression of the clipped 5^3 window's sums (numerical/statistics.hpp:694-713).
struct Reg {
    float a, b, r2;
};

__device__ __forceinline__ void regress_finish(double sx, double sy, double sxx, double syy, double sxy, int m,
                                               Reg& r)
{
    const double dn = (double)m, rn = 1.0 / dn;
    const double mx = div_window(sx, dn, rn), my = div_window(sy, dn, rn);
    const double xv = div_window(sxx, dn, rn) - mx * mx;
    const double yv = div_window(syy, dn, rn) - my * my;
    if (xv == 0.0 || yv == 0.0) {
        r.a = 0.0f;
        r.b = (float)my;
        r.r2 = 0.0f;
        return;
    }
    const double cov = div_window(sxy, dn, rn) - mx * my;
    r.a = (float)(cov / xv);
    r.b = (float)(my - (double)r.a * mx);  // b uses the float-rounded slope
    r.r2 = (float)(cov * cov / xv / yv);
}

template <typename T>
__device__ __forceinline__ float pix_diff(T a, T b)
{
    return (float)(a - b);
}
template <>
__device__ __forceinline__ float pix_diff<uint8_t>(uint8_t a, uint8_t b)
{
    return (float)((int)a - (int)b);
}

// gradient_at (numerical/numerical.hpp:102-109)
template <typename T>
__device__ __forceinline__ float3 grad_at(const T* __restrict__ I, const Dim3& D, int x, int y, int z, long long i)
{
    float3 g;
    const long long w = D.w, wh = D.wh();
    g.x = (x + 1 < D.w && x) ? pix_diff(I[i + 1], I[i - 1]) : 0.0f;
    g.y = (y + 1 < D.h && y) ? pix_diff(I[i + w], I[i - w]) : 0.0f;
    g.z = (z + 1 < D.d && z) ? pix_diff(I[i + wh], I[i - wh]) : 0.0f;
    return g;
}

// Stores modality mod's gradient term dd = 0 + g at q, its components cs apart: new_d = dd
// for the first modality, new_d += dd for the others (reg/cdm.hpp:430-433).
__device__ __forceinline__ void store_term(float* __restrict__ q, long long cs, float3 out, int mod)
{
    if (mod) {
        out.x = q[0] + out.x;
        out.y = q[cs] + out.y;
        out.z = q[2 * cs] + out.z;
    }
    q[0] = out.x;
    q[cs] = out.y;
    q[2 * cs] = out.z;
}

// cdm_get_gradient_d_imp (reg/cdm.hpp:46-78) of modality mod: the term is 0 + gradient
// term; the cost of every voxel is summed per block in double.
template <typename T, bool MULTI>
__global__ void __launch_bounds__(kCdmThreads) cdm_gradient_d_kernel(SEG_ARGS, int mod)
{
    SEG_BEGIN
    if (S.ctl->done || mod >= max(S.nmod, 1))
        return;
    const T* __restrict__ Js = (const T*)S.Js;
    const T* __restrict__ It = (const T*)S.It[mod];
    float* __restrict__ nd = S.new_d;
    double csum = 0.0;
    for (long long i = first; i < n; i += stride) {
        int x, y, z;
        unflat((int)i, D, x, y, z);
        float3 g = grad_at(Js, D, x, y, z, i);
        const float dif = pix_diff(Js[i], It[i]);
        g.x *= dif;
        g.y *= dif;
        g.z *= dif;
        store_term(nd + update_index(S, i), update_comp(S), make_float3(0.0f + g.x, 0.0f + g.y, 0.0f + g.z), mod);
        csum += (double)(dif * dif);
    }
    __shared__ double red[32];
    csum = block_sum(csum, red);
    if (threadIdx.x == 0)
        S.cost_part[blk] = csum;
    if (last_block_of_segment(S))
        control_block(S, mod);
}

// Tiled uint8 'r' gradient.  For integer pixels the regression's window sums (sum Js,
// sum It, sum Js^2, sum It^2, sum Js*It over the clipped 5^3 window) are exact integers, so
// they are formed here as separable 5-tap box sums over a tile staged as bytes (zero outside
// the volume, the window size m from the clipped extents) -- the same integers the
// reference sums voxel by voxel, hence bit-identical results at a fraction of the work.
//
// Along x a thread forms the sums of four neighbours from two words a row with byte dot
// products, along y it adds a run of 8 rows in registers, and the plane sums of the five
// quantities go to shared memory as one uint4 a voxel (sum Js and sum It share a word: 125
// pixels of 255 fit 16 bits); along z each thread slides the window over its (x, y) column.
// Bound by latency at two blocks an SM (128 registers, 60 KB): at 128^3 issue 41 %, FP64 pipe and
// conversion unit 21 and 18 %, and a warp waits 2.5 cycles an issue for its own last result.
// Launches, per-tap byte loads and sums of 32-bit words before, so after: 157x189x155 236 / 99
// us, 91x109x91 58.7 / 33.5, 46x55x46 17.8 / 14.7, 23x28x23 15.8 / 9.8.
constexpr int kUX = 32, kUY = 8, kUThreads = 256;
constexpr int kUHX = 40, kUHY = kUY + 4;  // staged rows: 36 bytes used
struct WinSum {
    uint32_t s, xx, yy, xy;  // sum Js | sum It << 16, sum Js^2, sum It^2, sum Js*It
};
__device__ __forceinline__ void operator+=(WinSum& a, const WinSum& b)
{
    a.s += b.s, a.xx += b.xx, a.yy += b.yy, a.xy += b.xy;
}
__device__ __forceinline__ void operator-=(WinSum& a, const WinSum& b)
{
    a.s -= b.s, a.xx -= b.xx, a.yy -= b.yy, a.xy -= b.xy;
}

template <int TZ>
constexpr int box_smem()  // bytes: both staged tiles, then the plane sums
{
    return 2 * (TZ + 4) * kUHY * kUHX + (TZ + 4) * kUY * kUX * 16;
}

template <int TZ>
__device__ __forceinline__ double gradient_box_u8(const CdmSeg& S, int blk, int mod, unsigned char* __restrict__ smem)
{
    constexpr int HZ = TZ + 4, kRows = HZ * kUHY;
    static_assert(16 * HZ <= kUThreads && kUX * kUY == kUThreads, "threads of the two passes");
    uint8_t* const sj = smem;
    uint8_t* const si = smem + kRows * kUHX;
    uint4* const sum = reinterpret_cast<uint4*>(smem + 2 * kRows * kUHX);
    const Dim3 D{S.w, S.h, S.d};
    const uint8_t* __restrict__ Js = (const uint8_t*)S.Js;
    const uint8_t* __restrict__ It = (const uint8_t*)S.It[mod];
    float* __restrict__ nd = S.new_d;
    const int ntx = (D.w + kUX - 1) / kUX, nty = (D.h + kUY - 1) / kUY, ntz = (D.d + TZ - 1) / TZ;
    const long long ntiles = (long long)ntx * nty * ntz;
    const long long wl = D.w, whl = D.wh();
    const int tid = threadIdx.x, lane = tid & 31;
    double csum = 0.0;
    for (long long tile = blk; tile < ntiles; tile += S.nblk) {
        const int x0 = (int)(tile % ntx) * kUX, y0 = (int)(tile / ntx % nty) * kUY, z0 = (int)(tile / ((long long)ntx * nty)) * TZ;
        __syncthreads();  // the previous tile's readers are done with the buffers
        // rows by warps: bytes 0..31 of one row, then the last 4 bytes of 8 rows at a time;
        // the loads of a thread's rows are in flight together
        auto stage = [&](int r, int hx, bool on, uint8_t& a, uint8_t& b) {
            const int gx = x0 + hx - 2, gy = y0 + r % kUHY - 2, gz = z0 + r / kUHY - 2;
            a = b = 0;
            if (on && gx >= 0 && gy >= 0 && gz >= 0 && gx < D.w && gy < D.h && gz < D.d) {
                const long long gi = gz * whl + gy * wl + gx;
                a = __ldg(Js + gi);
                b = __ldg(It + gi);
            }
        };
        constexpr int kPer = (kRows + 7) / 8, kTail = (kRows + 63) / 64;
        constexpr int kBatch = kPer % 9 == 0 ? 9 : kPer;
        for (int q0 = 0; q0 < kPer; q0 += kBatch) {
            uint8_t a[kBatch], b[kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const int r = (tid >> 5) + 8 * (q0 + q);
                stage(r, lane, r < kRows, a[q], b[q]);
            }
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const int r = (tid >> 5) + 8 * (q0 + q);
                if (r < kRows) {
                    sj[r * kUHX + lane] = a[q];
                    si[r * kUHX + lane] = b[q];
                }
            }
        }
        {
            uint8_t a[kTail], b[kTail];
#pragma unroll
            for (int q = 0; q < kTail; ++q) {
                const int r = (tid >> 2) + 64 * q;
                stage(r, kUX + (tid & 3), r < kRows, a[q], b[q]);
            }
#pragma unroll
            for (int q = 0; q < kTail; ++q) {
                const int r = (tid >> 2) + 64 * q;
                if (r < kRows) {
                    sj[r * kUHX + kUX + (tid & 3)] = a[q];
                    si[r * kUHX + kUX + (tid & 3)] = b[q];
                }
            }
        }
        __syncthreads();
        if (tid < 16 * HZ) {
            // x and y sums: 4 voxels in x, 4 in y (8 rows) of plane zz
            const int quad = tid & 7, half = (tid >> 3) & 1, zz = tid >> 4;
            const int o = (zz * kUHY + 4 * half) * kUHX + 4 * quad;
            WinSum row[8][4];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const uint32_t* pj = reinterpret_cast<const uint32_t*>(sj + o + r * kUHX);
                const uint32_t* pi = reinterpret_cast<const uint32_t*>(si + o + r * kUHX);
                const uint32_t j0 = pj[0], j1 = pj[1], t0 = pi[0], t1 = pi[1];
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    // bytes v .. v + 3 and v + 4
                    const uint32_t ja = __funnelshift_r(j0, j1, 8 * v), ta = __funnelshift_r(t0, t1, 8 * v);
                    const uint32_t jb = (j1 >> (8 * v)) & 0xffu, tb = (t1 >> (8 * v)) & 0xffu;
                    row[r][v].s = __dp4a(ja, 0x01010101u, jb) + (__dp4a(ta, 0x01010101u, tb) << 16);
                    row[r][v].xx = __dp4a(ja, ja, jb * jb);
                    row[r][v].yy = __dp4a(ta, ta, tb * tb);
                    row[r][v].xy = __dp4a(ja, ta, jb * tb);
                }
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                WinSum w = row[0][v];
#pragma unroll
                for (int r = 1; r < 5; ++r)
                    w += row[r][v];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    sum[(zz * kUY + 4 * half + r) * kUX + 4 * quad + v] = make_uint4(w.s, w.xx, w.yy, w.xy);
                    if (r < 3) {
                        w += row[r + 5][v];
                        w -= row[r][v];
                    }
                }
            }
        }
        __syncthreads();
        const int xo = lane, yo = tid >> 5, x = x0 + xo, y = y0 + yo;
        if (x >= D.w || y >= D.h)
            continue;
        const int mxy = (min(D.w - 1, x + 2) - max(0, x - 2) + 1) * (min(D.h - 1, y + 2) - max(0, y - 2) + 1);
        auto plane = [&](int z) {
            const uint4 q = sum[(z * kUY + yo) * kUX + xo];
            return WinSum{q.x, q.y, q.z, q.w};
        };
        WinSum w = plane(0);
#pragma unroll
        for (int z = 1; z < 4; ++z)
            w += plane(z);
#pragma unroll 1
        for (int zo = 0; zo < TZ; ++zo) {
            const int z = z0 + zo;
            if (z >= D.d)
                break;
            w += plane(zo + 4);
            const uint8_t* const pj = sj + ((zo + 2) * kUHY + yo + 2) * kUHX + xo + 2;
            const int js = *pj, it = si[pj - sj];
            float3 out = make_float3(0.0f, 0.0f, 0.0f);
            if (!(js == 0 || it == 0)) {
                const int m = mxy * (min(D.d - 1, z + 2) - max(0, z - 2) + 1);
                Reg r;
                regress_finish((double)(int)(w.s & 0xffffu), (double)(int)(w.s >> 16), (double)(int)w.xx,
                               (double)(int)w.yy, (double)(int)w.xy, m, r);
                if (r.a > 0.0f) {
                    // gradient_at from the tile (neighbours are inside the halo)
                    float3 g;
                    g.x = (x + 1 < D.w && x) ? (float)((int)pj[1] - (int)pj[-1]) : 0.0f;
                    g.y = (y + 1 < D.h && y) ? (float)((int)pj[kUHX] - (int)pj[-kUHX]) : 0.0f;
                    g.z = (z + 1 < D.d && z) ? (float)((int)pj[kUHX * kUHY] - (int)pj[-kUHX * kUHY]) : 0.0f;
                    const float sc = r.r2 * ((float)js * r.a + r.b - (float)it);
                    g.x *= sc;
                    g.y *= sc;
                    g.z *= sc;
                    out.x = 0.0f + g.x;
                    out.y = 0.0f + g.y;
                    out.z = 0.0f + g.z;
                    csum += (double)-r.r2;
                }
            }
            store_term(nd + update_index(S, (long long)z * D.h + y, x), update_comp(S), out, mod);
            w -= plane(zo);
        }
    }
    return csum;
}

template <bool MULTI>
__global__ void __launch_bounds__(kUThreads) cdm_gradient_box_u8_kernel(SEG_ARGS,
                                                                         int mod)
{
    const CdmSeg& S = SEG_OF(blk0);
    const int blk = (int)blockIdx.x - (MULTI ? S.blk0 : 0);
    if (blk >= S.nblk)
        return;
    if (S.ctl->done || mod >= max(S.nmod, 1))
        return;
    extern __shared__ __align__(16) unsigned char smraw[];
    const double cs = S.shallow ? gradient_box_u8<2>(S, blk, mod, smraw) : gradient_box_u8<8>(S, blk, mod, smraw);
    __shared__ double red[32];
    const double csum = block_sum(cs, red);
    if (threadIdx.x == 0)
        S.cost_part[blk] = csum;
    if (last_block_of_segment(S))
        control_block(S, mod);
}

// Asynchronous copy of a float from global to shared memory, +0 instead where !ok: all of a
// tile's loads are in flight together.
__device__ __forceinline__ void copy_async_f32(float* to, const float* from, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from),
                 "r"(ok ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Tiled float 'r' gradient (cdm_get_gradient_r_imp, reg/cdm.hpp:46-78).  Float pixels: the
// window sums of linear_regression over the clipped 5^3 window (numerical/window.hpp:92-110,
// numerical/statistics.hpp:694-713) are double sums in the reference's visiting order
// (offsets 0, 1, 2, -1, -2 per axis, z outermost), sxy of float products.  Double sums do
// not reassociate, so every voxel adds its own 125 taps in that order; taps outside the
// volume are zeros of the staged tile, which change no sum.  What neighbouring voxels share
// is the taps' widening to double and their products, so a thread takes V voxels in x:
// with V = 4 a window row is 8 values, widened once (24 conversions) for 20 taps.  A square
// of a widened float is exact, so adding it by a fused multiply-add rounds like the sum.
// Bound by latency at 24 warps an SM (80 registers): at 128^3 with every voxel inside the counters
// read FP64 pipe 61 %, conversion unit 55 %, issue 60 %, and a warp waits 2.0 cycles an issue for
// its own last result and 1.4 for the FP64 pipe.  The tile's loads are all in flight at once.
// 157x189x155 launch: 305 us with one voxel a thread reading global memory, 235 so;
// 91x109x91: 87 / 66; 64^3: 50 / 32; 23x28x23: 25 / 14.6.
constexpr int kFX = 32, kFY = 8, kFThreads = 256, kFHX = kFX + 4, kFHY = kFY + 4, kFMaxV = 4;

template <int V>
__device__ __forceinline__ double gradient_r_f32(const CdmSeg& S, int blk, int mod, float* __restrict__ smem)
{
    constexpr int kTX = kFX / V, kHZ = V + 4;  // the tile is 32 x 8 x V voxels
    static_assert((V == 2 || V == 4) && kTX * kFY * V == kFThreads, "one thread per V voxels of the tile");
    float* const sj = smem;
    float* const si = smem + kHZ * kFHY * kFHX;
    const Dim3 D{S.w, S.h, S.d};
    const float* __restrict__ Js = (const float*)S.Js;
    const float* __restrict__ It = (const float*)S.It[mod];
    float* __restrict__ nd = S.new_d;
    const int ntx = (D.w + kFX - 1) / kFX, nty = (D.h + kFY - 1) / kFY, ntz = (D.d + V - 1) / V;
    const long long ntiles = (long long)ntx * nty * ntz;
    const long long wl = D.w, whl = D.wh();
    const int xo = V * (threadIdx.x % kTX), yo = threadIdx.x / kTX % kFY, zo = threadIdx.x / (kTX * kFY);
    const int lane = threadIdx.x & 31;
    double csum = 0.0;
    for (long long tile = blk; tile < ntiles; tile += S.nblk) {
        const int x0 = (int)(tile % ntx) * kFX, y0 = (int)(tile / ntx % nty) * kFY, z0 = (int)(tile / ((long long)ntx * nty)) * V;
        __syncthreads();  // the previous tile's readers are done with the buffers
        for (int r = threadIdx.x >> 5; r < kFHY * kHZ; r += kFThreads / 32) {
            const int gy = y0 + r % kFHY - 2, gz = z0 + r / kFHY - 2;
            const bool row = gy >= 0 && gz >= 0 && gy < D.h && gz < D.d;
            const long long gi = gz * whl + gy * wl + x0 - 2;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int hx = lane + 32 * k, gx = x0 + hx - 2;
                if (hx < kFHX) {
                    const bool ok = row && gx >= 0 && gx < D.w;
                    copy_async_f32(sj + r * kFHX + hx, ok ? Js + gi + hx : Js, ok);
                    copy_async_f32(si + r * kFHX + hx, ok ? It + gi + hx : It, ok);
                }
            }
        }
        copy_async_wait();
        __syncthreads();
        const int y = y0 + yo, z = z0 + zo;
        if (x0 + xo >= D.w || y >= D.h || z >= D.d)
            continue;
        const long long i0 = z * whl + y * wl + x0 + xo;
        const float* const cj = sj + ((zo + 2) * kFHY + yo + 2) * kFHX + xo + 2;  // the first voxel in the tile
        const float* const ci = si + (cj - sj);
        bool any = false;
#pragma unroll
        for (int v = 0; v < V; ++v)
            any = any || !(cj[v] == 0.0f || ci[v] == 0.0f);
        double sx[V] = {}, sy[V] = {}, sxx[V] = {}, syy[V] = {}, sxy[V] = {};
        if (any) {
#pragma unroll 1
            for (int row = 0; row < 25; ++row) {
                const int a = row / 5, b = row % 5;  // offsets 0, 1, 2, -1, -2
                const int o = ((zo + 2 + (a < 3 ? a : 2 - a)) * kFHY + yo + 2 + (b < 3 ? b : 2 - b)) * kFHX + xo;
                float fj[V + 4], ft[V + 4];
#pragma unroll
                for (int k = 0; k < V + 4; k += V) {
                    if constexpr (V == 4) {
                        const float4 p = *reinterpret_cast<const float4*>(sj + o + k), q = *reinterpret_cast<const float4*>(si + o + k);
                        fj[k] = p.x, fj[k + 1] = p.y, fj[k + 2] = p.z, fj[k + 3] = p.w;
                        ft[k] = q.x, ft[k + 1] = q.y, ft[k + 2] = q.z, ft[k + 3] = q.w;
                    } else {
                        const float2 p = *reinterpret_cast<const float2*>(sj + o + k), q = *reinterpret_cast<const float2*>(si + o + k);
                        fj[k] = p.x, fj[k + 1] = p.y;
                        ft[k] = q.x, ft[k + 1] = q.y;
                    }
                }
                // one quantity after the other: 8 widened values at a time
                constexpr int kOrd[5] = {2, 3, 4, 1, 0};
                double q[V + 4];
#pragma unroll
                for (int k = 0; k < V + 4; ++k)
                    q[k] = (double)fj[k];
#pragma unroll
                for (int c = 0; c < 5; ++c)
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        sx[v] += q[v + kOrd[c]];
                        sxx[v] = __fma_rn(q[v + kOrd[c]], q[v + kOrd[c]], sxx[v]);
                    }
#pragma unroll
                for (int k = 0; k < V + 4; ++k)
                    q[k] = (double)ft[k];
#pragma unroll
                for (int c = 0; c < 5; ++c)
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        sy[v] += q[v + kOrd[c]];
                        syy[v] = __fma_rn(q[v + kOrd[c]], q[v + kOrd[c]], syy[v]);
                    }
#pragma unroll
                for (int k = 0; k < V + 4; ++k)
                    q[k] = (double)__fmul_rn(fj[k], ft[k]);
#pragma unroll
                for (int c = 0; c < 5; ++c)
#pragma unroll
                    for (int v = 0; v < V; ++v)
                        sxy[v] += q[v + kOrd[c]];
            }
        }
        const int myz = (min(D.h - 1, y + 2) - max(0, y - 2) + 1) * (min(D.d - 1, z + 2) - max(0, z - 2) + 1);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int x = x0 + xo + v;
            if (x >= D.w)
                break;
            float3 out = make_float3(0.0f, 0.0f, 0.0f);
            const float js = cj[v], it = ci[v];
            if (!(js == 0.0f || it == 0.0f)) {
                Reg r;
                regress_finish(sx[v], sy[v], sxx[v], syy[v], sxy[v],
                               (min(D.w - 1, x + 2) - max(0, x - 2) + 1) * myz, r);
                if (r.a > 0.0f) {
                    // gradient_at from the tile (neighbours are inside the halo)
                    const float* const p = cj + v;
                    float3 g;
                    g.x = (x + 1 < D.w && x) ? p[1] - p[-1] : 0.0f;
                    g.y = (y + 1 < D.h && y) ? p[kFHX] - p[-kFHX] : 0.0f;
                    g.z = (z + 1 < D.d && z) ? p[kFHX * kFHY] - p[-kFHX * kFHY] : 0.0f;
                    const float s = r.r2 * (js * r.a + r.b - it);
                    g.x *= s;
                    g.y *= s;
                    g.z *= s;
                    out.x = 0.0f + g.x;
                    out.y = 0.0f + g.y;
                    out.z = 0.0f + g.z;
                    csum += (double)-r.r2;
                }
            }
            store_term(nd + update_index(S, (long long)z * D.h + y, x), update_comp(S), out, mod);
        }
    }
    return csum;
}

// The same a voxel a thread, from global memory: for the volumes of cdm_gradient_each.
__device__ __forceinline__ double gradient_r_f32_each(const CdmSeg& S, int blk, int mod)
{
    const Dim3 D{S.w, S.h, S.d};
    const float* __restrict__ Js = (const float*)S.Js;
    const float* __restrict__ It = (const float*)S.It[mod];
    float* __restrict__ nd = S.new_d;
    const long long n = D.n(), w = D.w, wh = D.wh();
    double csum = 0.0;
    for (long long i = blk * (long long)kFThreads + threadIdx.x; i < n; i += (long long)S.nblk * kFThreads) {
        int x, y, z;
        unflat((int)i, D, x, y, z);
        float3 out = make_float3(0.0f, 0.0f, 0.0f);
        const float js = Js[i], it = It[i];
        if (!(js == 0.0f || it == 0.0f)) {
            const int xu = min(D.w - x - 1, 2), yu = min(D.h - y - 1, 2), zu = min(D.d - z - 1, 2);
            const int xl = min(x, 2), yl = min(y, 2), zl = min(z, 2);
            double sx = 0.0, sy = 0.0, sxx = 0.0, syy = 0.0, sxy = 0.0;
            auto add = [&](long long k) {
                const float j = Js[k], t = It[k];
                const double dj = j, dt = t;
                sx += dj;
                sy += dt;
                sxx = __fma_rn(dj, dj, sxx);
                syy = __fma_rn(dt, dt, syy);
                sxy += (double)__fmul_rn(j, t);
            };
            for (int a = 0; a <= zu + zl; ++a) {  // offsets 0, 1, 2, -1, -2 where they are inside
                const long long zi = i + (a <= zu ? a : zu - a) * wh;
                for (int b = 0; b <= yu + yl; ++b) {
                    const long long yi = zi + (b <= yu ? b : yu - b) * w;
                    if (w < 4)  // one loop (3x300x300 59 / 45 us), two from there on (4x300x300 89 / 73)
                        for (int c = 0; c <= xu + xl; ++c)
                            add(yi + (c <= xu ? c : xu - c));
                    else {
                        for (int c = 0; c <= xu; ++c)
                            add(yi + c);
                        for (int c = 1; c <= xl; ++c)
                            add(yi - c);
                    }
                }
            }
            Reg r;
            regress_finish(sx, sy, sxx, syy, sxy, (xu + xl + 1) * (yu + yl + 1) * (zu + zl + 1), r);
            if (r.a > 0.0f) {
                const float3 g = grad_at(Js, D, x, y, z, i);
                const float s = r.r2 * (js * r.a + r.b - it);
                out.x = 0.0f + g.x * s;
                out.y = 0.0f + g.y * s;
                out.z = 0.0f + g.z * s;
                csum += (double)-r.r2;
            }
        }
        store_term(nd + update_index(S, i), update_comp(S), out, mod);
    }
    return csum;
}

template <bool MULTI>
__global__ void __launch_bounds__(kFThreads, 3) cdm_gradient_r_f32_kernel(SEG_ARGS,
                                                                          int mod)
{
    const CdmSeg& S = SEG_OF(blk0);
    const int blk = (int)blockIdx.x - (MULTI ? S.blk0 : 0);
    if (blk >= S.nblk)
        return;
    if (S.ctl->done || mod >= max(S.nmod, 1))
        return;
    __shared__ __align__(16) float smem[2 * (kFMaxV + 4) * kFHY * kFHX];
    // Small levels take two voxels a thread: a tile's time is its 25 rows' latency there, and
    // there are not enough tiles of four to fill the chip (91x109x91: 71.0 us with two, 65.6
    // with four; 64^3: 32.0 / 30.1; 46x55x46: 25.3 / 27.4; 23x28x23: 14.8 / 20.6).
    const long long n = (long long)S.w * S.h * S.d;
    const double cs = MULTI && S.each ? gradient_r_f32_each(S, blk, mod)
                      : n < 200000    ? gradient_r_f32<2>(S, blk, mod, smem)
                                      : gradient_r_f32<4>(S, blk, mod, smem);
    __shared__ double red[32];
    const double csum = block_sum(cs, red);
    if (threadIdx.x == 0)
        S.cost_part[blk] = csum;
    if (last_block_of_segment(S))
        control_block(S, mod);
}

// One level of that form: 64 registers, four blocks an SM instead of the three of the tiles.
__global__ void __launch_bounds__(kFThreads) cdm_gradient_r_f32_each_kernel(SEG_ARGS, int mod)
{
    const CdmSeg& S = one;
    const int blk = (int)blockIdx.x;
    if (S.ctl->done || mod >= max(S.nmod, 1))
        return;
    __shared__ double red[32];
    const double csum = block_sum(gradient_r_f32_each(S, blk, mod), red);
    if (threadIdx.x == 0)
        S.cost_part[blk] = csum;
    if (last_block_of_segment(S))
        control_block(S, mod);
}

// ------------------------------------------------------------------ control
// cdm_improved (reg/cdm.hpp:19-34): regression of the last costs on their index
// (int x, float y; statistics.hpp:694-713); a positive slope means "not improved".
__device__ bool cdm_improved_dev(CdmCtl* c)
{
    const int n = c->ncost;
    if (n > 5) {
        long long sx = 0, sxx = 0;
        double sy = (double)c->cost[0], syy = 0.0, sxy = (double)(0.0f * c->cost[0]);
        for (int i = 0; i < n; ++i) {
            sx += i;
            sxx += (long long)i * i;
        }
        for (int i = 1; i < n; ++i) {
            sy += (double)c->cost[i];
            sxy += (double)((float)i * c->cost[i]);
        }
        for (int i = 0; i < n; ++i) {
            const double t = c->cost[i];
            syy += t * t;
        }
        const double mx = (double)sx / n, my = sy / n;
        const double xv = (double)sxx / n - mx * mx, yv = syy / n - my * my;
        float a = 0.0f;
        if (!(xv == 0.0 || yv == 0.0))
            a = (float)((sxy / n - mx * my) / xv);
        if (a > 0.0f)
            return false;
        if (n > 7) {
            for (int i = 1; i < n; ++i)
                c->cost[i - 1] = c->cost[i];
            c->ncost = n - 1;
        }
    }
    return true;
}

// Mean of the per-block cost partials, summed in a fixed order.
__device__ float seg_cost_mean(const CdmSeg& S)
{
    __shared__ double red[32];
    double s = 0.0;
    for (int k = threadIdx.x; k < S.nblk; k += blockDim.x)
        s += S.cost_part[k];
    s = block_sum(s, red);
    __shared__ float out;
    if (threadIdx.x == 0)
        out = (float)(s / (double)((long long)S.w * S.h * S.d));
    __syncthreads();
    return out;
}

// The body of the reference's iteration loop between the gradient and the
// Poisson solve (reg/cdm.hpp:418-460), run by one block of the segment (the
// gradient kernel's last block).  Each modality's launch keeps its mean cost; the
// last modality's sums them in modality order (float), failing the level as soon
// as a partial sum is exactly zero, and records sum / nmod.
__device__ void control_step(CdmCtl* c, int nm, int mod, float mean_cost)
{
    c->mod_cost[mod] = mean_cost;
    if (mod + 1 < nm)
        return;
    if (c->index >= c->max_iter) {
        c->done = 1;
        return;
    }
    float sum_cost = 0.0f;
    for (int k = 0; k < nm; ++k) {
        sum_cost += c->mod_cost[k];
        if (sum_cost == 0.0f) {
            c->last_cost = sum_cost;
            c->done = 2;
            return;
        }
    }
    c->last_cost = sum_cost;
    c->cost[c->ncost++] = sum_cost / (float)nm;
    const float cur = c->cost[c->ncost - 1];
    if (cur < c->best_cost) {
        c->best_cost = cur;
        if (c->index)
            c->best = c->cur;
    }
    if (!cdm_improved_dev(c)) {
        if (c->cur_smoothing <= c->smoothing) {
            c->done = 1;
            ++c->iters_run;
            return;
        }
        c->cur = c->best;
        c->cur_smoothing *= 0.5f;
        c->ncost = 0;
    }
    // this iteration's field goes where the best one is not; without smoothing the field
    // stays what it is
    c->from = c->cur;
    if (c->cur_smoothing != 0.0f)
        c->cur = 1 - c->best;
    ++c->index;
    ++c->iters_run;
}

// The block works on a copy of the control block in shared memory: one thread takes the
// decisions, some thirty dependent loads and stores, each of which would cost a trip to L2
// (16^3 uint8 gradient launch: 15.5 us with the control block in global memory, 14.7 so).
__device__ void control_block(const CdmSeg& S, int mod)
{
    constexpr int kWords = sizeof(CdmCtl) / 4;
    static_assert(sizeof(CdmCtl) % 4 == 0, "copied by words");
    __shared__ CdmCtl c;
    uint32_t* const g = reinterpret_cast<uint32_t*>(S.ctl);
    uint32_t* const l = reinterpret_cast<uint32_t*>(&c);
    for (int i = threadIdx.x; i < kWords; i += blockDim.x)
        l[i] = g[i];
    const float mean_cost = seg_cost_mean(S);  // (its barriers order the copy too)
    if (threadIdx.x == 0)
        control_step(&c, S.nmod > 1 ? S.nmod : 1, mod, mean_cost);
    __syncthreads();
    for (int i = threadIdx.x; i < kWords; i += blockDim.x)
        g[i] = l[i];
}

// Completion ticket of a segment's blocks: true in the one block that finishes
// last (all other blocks' global writes are visible to it).
__device__ __forceinline__ bool last_block_of_segment(const CdmSeg& S)
{
    __shared__ unsigned int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = (atomicAdd(&S.ctl->ticket, 1u) == (unsigned)S.nblk - 1u);
        if (last)
            S.ctl->ticket = 0u;
    }
    __syncthreads();
    if (last)
        __threadfence();
    return last;
}

// ------------------------------------------------------------------ Poisson
// cdm_solve_poisson (reg/cdm.hpp:158-253): s0 = new_d * (-1/6); then 12 Jacobi sweeps
// s' = (new_d - s[-1] - s[+1] - s[-w] - s[+w] - s[-wh] - s[+wh]) * (-1/6) with the
// neighbours taken by flat index, bounds on the flat index only (2-D: -1/4 and no
// +-wh taps).
//
// The components are planes of their own here, rows padded to 16 bytes (CdmSeg::ppitch).
// In units of float4 the padded component is a line on which every tap is a fixed offset: a
// row's ends meet the rows before and after it and a plane's the neighbouring planes, as the
// flat taps want, except that a row's last voxels may share their float4 with padding.  So
// the threads of a block take consecutive float4 of a plane whatever rows they belong to, and
// walk a few planes: the z taps are the thread's registers, x taps too but for a shuffle a
// side, the rows above and below are loads that the block's walk has just brought to L1.
// Positions outside the field count as +0, whose subtraction changes nothing, like the taps
// the reference skips.
//
// Bound by L2 (and its latency): a sweep with a thread per float of the interleaved field (nine
// scalar loads each, the neighbouring rows and planes from L2), and so: 91x109x91 11.4 / 6.5 us,
// 128^3 22.7 / 10.7, 182x218x182 103 / 53.  Levels of up to 64 planes of 1024 columns take the
// clusters below instead (46x55x46, 12 sweeps: 49 / 40 / 17.6).
constexpr int kPThreads = 256, kFlat = 4;
constexpr int kPSweeps = 12;  // reg/cdm.hpp:165
static_assert(kPSweeps % 2 == 0, "the result lands in aux_d");
// The tail launches (accumulate, smooth and compose): a block takes kTile positions of a
// component, whatever rows and planes they belong to.
constexpr int kTThreads = 128, kTile = 4 * kTThreads, kAVox = 2;

// The clusters of small levels (below): a block's columns are a plane's, and its planes few.
constexpr int kPCluster = 16, kPClusterThreads = 1024, kPClusterPlanes = 4;
static bool cluster_holds(long long pitch, int h, int d)
{
    return pitch / 4 * h <= kPClusterThreads && d <= kPCluster * kPClusterPlanes;
}

// Planes a thread of the sweeps walks, and their grids, for a launch of n levels.  The fewest
// that let the whole launch be resident at once keep every SM busy to its end; levels that would
// take more than 12 have several waves anyway and walk 8, which reads a plane of the input 1.25
// times (a sweep of 91x109x91: 7.3 us with 8, 6.5 with 5, 7.9 with 4, whose blocks are 1.2
// waves; 128^3: 12.3 / 10.7 with 11; 100x100x120 8.7 / 7.8 with 7; 182x218x182 the same from 7
// to 14).
//
// Planes that leave more than a fifth of their blocks' threads without a column, and single
// planes, are not walked: the threads take the component's float4 one after the other, the z taps
// from L1 (12 sweeps walked / so: 4x4x20000 744 / 46 us, 16x16x1500 90 / 52, 36x32x400, 56 % of
// the threads, 75 / 59; 28x28x700, 77 %, the same; 44x44x300, 95 %, 66 / 69).
void cdm_set_walk(CdmSeg* s, int n)
{
    constexpr long long kResident = 148 * 4;
    auto blocks_of = [](long long items) { return (items + kPThreads - 1) / kPThreads; };
    auto whole = [&](const CdmSeg& e) {
        const long long cols = e.ppitch / 4 * e.h;
        return (e.ppitch & 3) || e.d == 1 || 5 * cols < 4 * blocks_of(cols) * kPThreads;
    };
    auto blocks = [&](const CdmSeg& e, int dz) {
        if (e.ppitch & 3)
            return 3 * blocks_of((e.pplane + kFlat - 1) / kFlat);
        return 3 * (whole(e) ? blocks_of(e.pplane / 4) : blocks_of(e.ppitch / 4 * e.h) * ((e.d + dz - 1) / dz));
    };
    int walk = 8;
    for (int dz = 1; dz <= 12; ++dz) {
        long long total = 0;
        for (int k = 0; k < n; ++k)
            total += blocks(s[k], dz);
        if (total <= kResident) {
            walk = dz;
            break;
        }
    }
    for (int k = 0; k < n; ++k) {
        s[k].pdz = whole(s[k]) ? 0 : walk;
        s[k].pnb = (int)blocks(s[k], walk);
    }
}

// Whether the float 'r' gradient takes a voxel a thread: for volumes of few voxels on an axis,
// which fill little of a tile and have few of the window's taps inside.  The lower of two
// estimates in us: each voxel its taps, against the tiles, of which small levels have more than
// blocks.  Launches in tiles / so: 1x300x300 290 / 15.7 us, 3x300x300 202 / 59, 7x300x300 203 /
// 119, 1024x1024x1 168 / 60, 300x2x300 51 / 26, 8x60x60 32 / 21; and where tiles are kept:
// 9x300x300 206 / 187, 300x300x3 36 / 47, 33x33x33 21 / 23, 91x109x91 80 / 183.
static int gradient_each(int w, int h, int d)
{
    auto taps = [](int n) { return n < 4 ? n : 5.0 - 6.0 / n; };  // inside, on average
    const long long n = (long long)w * h * d;
    const int v = n < 200000 ? 2 : 4;
    const long long tiles = (long long)((w + kFX - 1) / kFX) * ((h + kFY - 1) / kFY) * ((d + v - 1) / v);
    const double t = taps(w) * taps(h) * taps(d);
    const int blocks = cdm_blocks_for(n);
    const double each = std::max(9.0 + 0.09 * t, 2.1e-6 * (double)n * (t + 14.0));
    return each < (v == 2 ? 7.0 + 7.2 * (double)((tiles + blocks - 1) / blocks) : 0.06 * (double)tiles);
}

// Whether the uint8 'r' gradient's tiles are 2 planes deep, not 8: where there are no more planes
// (1024x1024x1 63 / 89 us), and on levels whose tiles of 8 would leave most SMs idle (23x28x23
// 9.8 / 14.0; 64^3 20.1 / 19.6), unless a block has several of them in turn (short rows or
// columns: 300x2x300 35.5 / 28.8).
static int gradient_shallow(int w, int h, int d)
{
    const long long n = (long long)w * h * d;
    const long long tiles = (long long)((w + kUX - 1) / kUX) * ((h + kUY - 1) / kUY) * ((d + 1) / 2);
    return d <= 2 || (n < 200000 && tiles <= 3 * std::min(cdm_blocks_for(n), 148 * 3));
}

// Launch shapes that follow from a level's dims alone.
void cdm_set_dims(CdmSeg& s, int w, int h, int d)
{
    s.w = w;
    s.h = h;
    s.d = d;
    s.nblk = cdm_blocks_for((long long)w * h * d);
    // component planes of the fields: rows padded to 4 voxels, unless that doubles them (rows of
    // one or two voxels; not where the sweeps then run in clusters) or costs memory that counts
    // (other short rows of a huge volume).  12 sweeps with padded rows / so: 1x200000x1 86 / 44
    // us, 2x200000x1 86 / 74, 2x300x300 50 / 42; 9x1280x1200 1449 / 1600.
    const long long rows = (long long)h * d, padded = (w + 3LL) / 4 * 4;
    const bool pad = 4 * padded <= 5LL * w || cluster_holds(padded, h, d) ||
                     (padded < 2LL * w && padded * rows < (1LL << 24));
    s.ppitch = pad ? padded : w;
    s.pplane = s.ppitch * rows;
    cdm_set_walk(&s, 1);
    s.each = gradient_each(w, h, d);
    s.shallow = gradient_shallow(w, h, d);
    s.tnb = (int)((s.pplane + kTile - 1) / kTile);
}

// inv_d2 = -0.5 / dimension (reg/cdm.hpp:163,175): -1/6 in 3-D, -1/4 in 2-D.  A 2-D
// level's plane is the whole image (d == 1), so its +-wh taps fall outside the flat
// index range and drop out, as the reference's 2-D stencil has none.
__device__ __forceinline__ float poisson_weight(const CdmSeg& S)
{
    return S.ndim == 2 ? -0.5f / 2.0f : -0.5f / 3.0f;
}

// A load the compiler leaves where it stands; zeros where !ok.
__device__ __forceinline__ float4 load_now(const float4* __restrict__ p, bool ok)
{
    float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (ok)
        asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w) : "l"(p));
    return f;
}

__device__ __forceinline__ float load_now(const float* __restrict__ p, bool ok)
{
    float f = 0.0f;
    if (ok)
        asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(f) : "l"(p));
    return f;
}

// One block's part of a sweep: float4 column q of a plane, planes [z0, z1).  FIRST: the input
// is the right-hand side times c6.  EDGE: some tap of the block may lie outside the field.  WHOLE:
// float4 q of the component instead, for planes [0, 1).
template <bool FIRST, bool EDGE, bool WHOLE = false>
__device__ __forceinline__ void poisson_walk(const CdmSeg& S, const float4* __restrict__ in, const float4* __restrict__ rhs,
                                             float4* __restrict__ out, unsigned q, int z0, int z1, int done)
{
    const unsigned P = (unsigned)(S.ppitch / 4), plane = P * (unsigned)S.h, total = plane * (unsigned)S.d;
    const float c6 = poisson_weight(S);
    const int rem = S.w & 3, lane = threadIdx.x & 31;
    const unsigned xq = q % P;
    const unsigned span = WHOLE ? total : plane;
    const bool on = q < span, row_end = xq == P - 1;
    const bool fix1 = row_end && rem == 1, fix2 = row_end && rem == 2, fix3 = row_end && rem == 3;
    unsigned i = (unsigned)z0 * plane + q;
    auto inside = [&](unsigned k) { return on && (!EDGE || k < total); };
    auto value = [&](float4 f, unsigned k) {
        return FIRST && inside(k) ? make_float4(f.x * c6, f.y * c6, f.z * c6, f.w * c6) : f;
    };
    auto at = [&](unsigned k) {
        float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (inside(k))
            f = __ldg(in + k);
        return value(f, k);
    };
    auto one = [&](long long k) {
        float f = 0.0f;
        if (on && (!EDGE || (k >= 0 && k < 4LL * total))) {
            f = __ldg(reinterpret_cast<const float*>(in) + k);
            if (FIRST)
                f *= c6;
        }
        return f;
    };
    // the first plane's loads go out before the loop flag is waited for
    float4 down = load_now(in + (i - plane), inside(i - plane)), cur = load_now(in + i, on),
           up = load_now(in + (i + plane), inside(i + plane)), b = load_now(rhs + i, on);
    if (done)
        return;
    down = value(down, i - plane);
    cur = value(cur, i);
    up = value(up, i + plane);
    for (int z = z0; z < z1; ++z, i += plane) {
        const float4 ya = at(i - P), yb = at(i + P);
        if (z > z0)
            b = on ? __ldg(rhs + i) : b;
        float4 next = up;
        if (z + 1 < z1)
            next = at(i + 2 * plane);
        // a row's last voxel is where the padding begins
        const float tail = fix1 ? cur.x : fix2 ? cur.y : fix3 ? cur.z : cur.w;
        float xl = __shfl_up_sync(0xffffffffu, tail, 1), xr = __shfl_down_sync(0xffffffffu, cur.x, 1);
        if (lane == 0)
            xl = one(4LL * i - 1 - (xq == 0 && rem ? 4 - rem : 0));
        if (lane == 31 || q + 1 == span)
            xr = one(4LL * i + 4);
        const float n1 = fix1 ? xr : cur.y, n2 = fix2 ? xr : cur.z, n3 = fix3 ? xr : cur.w;
        float4 v;
        v.x = ((((((b.x - xl) - n1) - ya.x) - yb.x) - down.x) - up.x) * c6;
        v.y = ((((((b.y - cur.x) - n2) - ya.y) - yb.y) - down.y) - up.y) * c6;
        v.z = ((((((b.z - cur.y) - n3) - ya.z) - yb.z) - down.z) - up.z) * c6;
        v.w = ((((((b.w - cur.z) - xr) - ya.w) - yb.w) - down.w) - up.w) * c6;
        if (on)
            out[i] = v;
        down = cur;
        cur = up;
        up = next;
    }
}

// The part of block b in a sweep over unpadded rows: kFlat runs of a float a thread, whose taps
// are all on their way before the first is used (12 sweeps of 2x2000x5000: 3247 us a float after
// the other, 2281 so; 9x1280x1200 2350 / 1600; 2x300x300 48 / 42).
template <bool FIRST>
__device__ __forceinline__ void poisson_flat(const CdmSeg& S, const float* __restrict__ in, const float* __restrict__ rhs,
                                             float* __restrict__ out, unsigned b)
{
    const unsigned w = (unsigned)S.w, wh = w * (unsigned)S.h, n = wh * (unsigned)S.d;
    const float c6 = poisson_weight(S);
    auto at = [&](unsigned k) { return FIRST ? __ldg(in + k) * c6 : __ldg(in + k); };
    const unsigned first = b * (kFlat * kPThreads), p0 = first + threadIdx.x;
    if (first >= wh && first + kFlat * kPThreads + wh <= n) {  // every tap is inside
        float t[kFlat][7];
#pragma unroll
        for (int k = 0; k < kFlat; ++k) {
            const unsigned p = p0 + k * kPThreads, i[6] = {p - 1, p + 1, p - w, p + w, p - wh, p + wh};
            t[k][6] = __ldg(rhs + p);
#pragma unroll
            for (int j = 0; j < 6; ++j)
                t[k][j] = at(i[j]);
        }
#pragma unroll
        for (int k = 0; k < kFlat; ++k) {
            float acc = t[k][6];
#pragma unroll
            for (int j = 0; j < 6; ++j)
                acc -= t[k][j];
            out[p0 + k * kPThreads] = acc * c6;
        }
        return;
    }
    for (int k = 0; k < kFlat; ++k) {
        const unsigned p = p0 + k * kPThreads;
        if (p >= n)
            return;
        float acc = __ldg(rhs + p);
        if (p >= 1) acc -= at(p - 1);
        if (p < n - 1) acc -= at(p + 1);
        if (p >= w) acc -= at(p - w);
        if (p < n - w) acc -= at(p + w);
        if (p >= wh) acc -= at(p - wh);
        if (p < n - wh) acc -= at(p + wh);
        out[p] = acc * c6;
    }
}

// One sweep.  FIRST: its input is new_d * (-1/6) formed on the fly (the same float product
// the reference stores), its output tmp_d.  Otherwise parity picks aux_d -> tmp_d or
// tmp_d -> aux_d (the last sweep).
template <bool FIRST, bool MULTI>
__global__ void __launch_bounds__(kPThreads, 4) cdm_poisson_kernel(SEG_ARGS, int parity)
{
    const CdmSeg& S = SEG_OF(pblk0);
    const int tile = (int)blockIdx.x - (MULTI ? S.pblk0 : 0);
    if (tile >= S.pnb)
        return;
    const int done = S.ctl->done;
    // component slowest, then z chunks: the blocks in flight share planes
    const int per = S.pnb / 3, comp = tile / per, t = tile % per;
    const float* const rhs = S.new_d + comp * S.pplane;
    const float* const in = FIRST ? rhs : (parity ? S.tmp_d : S.aux_d) + comp * S.pplane;
    float* const out = (FIRST || !parity ? S.tmp_d : S.aux_d) + comp * S.pplane;
    if (MULTI && (S.ppitch & 3)) {
        if (!done)
            poisson_flat<FIRST>(S, in, rhs, out, (unsigned)t);
    } else {
        const float4* const in4 = reinterpret_cast<const float4*>(in);
        const float4* const rhs4 = reinterpret_cast<const float4*>(rhs);
        float4* const out4 = reinterpret_cast<float4*>(out);
        if (S.pdz == 0) {
            const unsigned q = (unsigned)t * kPThreads + threadIdx.x;
            poisson_walk<FIRST, true, true>(S, in4, rhs4, out4, q, 0, 1, done);
            return;
        }
        const int nz = (S.d + S.pdz - 1) / S.pdz, nq = per / nz;
        const int z0 = t / nq * S.pdz, z1 = min(S.d, z0 + S.pdz);
        const unsigned q = (unsigned)(t % nq) * kPThreads + threadIdx.x;
        if (z0 == 0 || z1 == S.d)  // (a plane below and above covers the rows and voxels beside)
            poisson_walk<FIRST, true>(S, in4, rhs4, out4, q, z0, z1, done);
        else
            poisson_walk<FIRST, false>(S, in4, rhs4, out4, q, z0, z1, done);
    }
}

// One level of unpadded rows.
template <bool FIRST>
__global__ void __launch_bounds__(kPThreads, 4) cdm_poisson_flat_kernel(SEG_ARGS, int parity)
{
    const CdmSeg& S = one;
    const int done = S.ctl->done;
    const int per = S.pnb / 3, comp = (int)blockIdx.x / per, t = (int)blockIdx.x % per;
    const float* const rhs = S.new_d + comp * S.pplane;
    const float* const in = FIRST ? rhs : (parity ? S.tmp_d : S.aux_d) + comp * S.pplane;
    float* const out = (FIRST || !parity ? S.tmp_d : S.aux_d) + comp * S.pplane;
    if (!done)
        poisson_flat<FIRST>(S, in, rhs, out, (unsigned)t);
}

// ---- the 12 sweeps of a small level in one launch ----
// A cluster of kPCluster blocks holds one component in shared memory: a block owns K planes and
// a halo plane on either side, a thread a float4 column of them with its right-hand side in
// registers.  A sweep reads one copy of the planes and writes the other; the outer planes also
// go to the neighbouring blocks' halos over distributed shared memory, and a cluster barrier
// ends it.  Taps, padding and arithmetic are poisson_walk's; a halo outside the field stays
// zero.
//
// Bound by the barrier and the exchange (0.6 us a sweep at 16^3) on the smallest, then by issue.
// Twelve launches of a sweep before, one so: 23x28x23 25 / 8.4 us, 32^3 24.6 / 10.9, 46x55x46
// 40 / 17.6, 64^3 40 / 29, and the gaps between the launches.
// Larger levels do not fit: a plane has to be a block's columns, 16 blocks hold 64 planes.
__device__ __forceinline__ void cluster_barrier()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of p (shared memory of this block) in block `rank` of the cluster, and a store there.
__device__ __forceinline__ unsigned remote_address(const float4* p, int rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void store_remote(unsigned address, float4 v)
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(address), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// The sweeps of a block with NZ planes from z0 on.  K: the planes of a full block, which place
// the upper halo of the block below.  PAD: rows end within a float4.
template <int NZ, bool PAD>
__device__ __forceinline__ void poisson_block(const CdmSeg& S, float4* planes, int K, int rank, int comp)
{
    const unsigned P = (unsigned)(S.ppitch / 4), plane = P * (unsigned)S.h, copy = (K + 2) * plane;
    const float c6 = poisson_weight(S);
    const int z0 = rank * K, rem = S.w & 3, lane = threadIdx.x & 31;
    // threads past the plane go through the last column's motions and store nothing
    const unsigned q = min(threadIdx.x, plane - 1), xq = q % P;
    const bool on = threadIdx.x < plane, row_end = PAD && xq == P - 1, first = lane == 0, last = lane == 31 || q + 1 == plane;
    const bool fix1 = row_end && rem == 1, fix2 = row_end && rem == 2, fix3 = row_end && rem == 3;
    const int left = -1 - (PAD && xq == 0 && rem ? 4 - rem : 0);
    const bool push_low = on && rank > 0, push_high = on && z0 + NZ < S.d;
    const unsigned low = remote_address(planes + (K + 1) * plane + q, max(rank - 1, 0)),
                   high = remote_address(planes + q, rank + (z0 + NZ < S.d ? 1 : 0));
    const float4* const rhs = reinterpret_cast<const float4*>(S.new_d + comp * S.pplane) + (unsigned)z0 * plane + q;
    float4* const out = reinterpret_cast<float4*>(S.aux_d + comp * S.pplane) + (unsigned)z0 * plane + q;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto scaled = [&](float4 f) { return make_float4(f.x * c6, f.y * c6, f.z * c6, f.w * c6); };
    float4 b[NZ], v[NZ];
#pragma unroll
    for (int k = 0; k < NZ; ++k)
        b[k] = __ldg(rhs + k * plane);
    const float4 below = rank > 0 ? scaled(__ldg(rhs - plane)) : zero;
    const float4 above = z0 + NZ < S.d ? scaled(__ldg(rhs + NZ * plane)) : zero;
#pragma unroll
    for (int k = 0; k < NZ; ++k)
        v[k] = scaled(b[k]);
    if (on) {  // the second copy's halos outside the field stay zero
        planes[q] = below;
        planes[(NZ + 1) * plane + q] = above;
        planes[copy + q] = zero;
        planes[copy + (NZ + 1) * plane + q] = zero;
#pragma unroll
        for (int k = 0; k < NZ; ++k)
            planes[(k + 1) * plane + q] = v[k];
    }
    cluster_barrier();
    auto sweep = [&](unsigned from, unsigned to, bool end) {
        const float4* p = planes + from + plane + q;
        float4* t = planes + to + plane + q;
        float4 down = *(p - plane);
        const float4 top = *(p + NZ * plane);
#pragma unroll
        for (int k = 0; k < NZ; ++k) {
            const float4 cur = v[k], ya = *(p - P), yb = *(p + P), up = k + 1 < NZ ? v[k + 1 < NZ ? k + 1 : k] : top;
            const float tail = fix1 ? cur.x : fix2 ? cur.y : fix3 ? cur.z : cur.w;
            float xl = __shfl_up_sync(0xffffffffu, tail, 1), xr = __shfl_down_sync(0xffffffffu, cur.x, 1);
            if (first)
                xl = *(reinterpret_cast<const float*>(p) + left);
            if (last)
                xr = *(reinterpret_cast<const float*>(p) + 4);
            const float n1 = fix1 ? xr : cur.y, n2 = fix2 ? xr : cur.z, n3 = fix3 ? xr : cur.w;
            float4 n;
            n.x = ((((((b[k].x - xl) - n1) - ya.x) - yb.x) - down.x) - up.x) * c6;
            n.y = ((((((b[k].y - cur.x) - n2) - ya.y) - yb.y) - down.y) - up.y) * c6;
            n.z = ((((((b[k].z - cur.y) - n3) - ya.z) - yb.z) - down.z) - up.z) * c6;
            n.w = ((((((b[k].w - cur.z) - xr) - ya.w) - yb.w) - down.w) - up.w) * c6;
            down = cur;
            v[k] = n;
            if (end) {
                if (on)
                    out[k * plane] = n;
            } else {
                if (on)
                    *t = n;
                if (k == 0 && push_low)
                    store_remote(low + 16 * to, n);
                if (k + 1 == NZ && push_high)
                    store_remote(high + 16 * to, n);
            }
            p += plane;
            t += plane;
        }
    };
#pragma unroll 1
    for (int k = 0; k + 1 < kPSweeps; ++k) {
        sweep(k & 1 ? copy : 0, k & 1 ? 0 : copy, false);
        cluster_barrier();
    }
    sweep(kPSweeps & 1 ? 0 : copy, 0, true);
}

// Three clusters an entry.
template <bool PAD, bool MULTI>
__global__ void __launch_bounds__(kPClusterThreads) cdm_poisson_cluster_kernel(const CdmSeg* __restrict__ segs,
                                                                               const __grid_constant__ CdmSeg one)
{
    extern __shared__ float4 planes[];  // two copies of K + 2 planes
    const CdmSeg& S = MULTI ? segs[blockIdx.x / (3 * kPCluster)] : one;
    if (S.ctl->done)
        return;
    const int rank = (int)blockIdx.x % kPCluster, comp = (int)blockIdx.x / kPCluster % 3;
    const int K = (S.d + kPCluster - 1) / kPCluster;
    static_assert(kPClusterPlanes == 4, "one case for each number of planes");
    switch (max(0, min(K, S.d - rank * K))) {  // the same for every thread of the block
    case 4: poisson_block<4, PAD>(S, planes, K, rank, comp); break;
    case 3: poisson_block<3, PAD>(S, planes, K, rank, comp); break;
    case 2: poisson_block<2, PAD>(S, planes, K, rank, comp); break;
    case 1: poisson_block<1, PAD>(S, planes, K, rank, comp); break;
    default:
        for (int k = 0; k < kPSweeps; ++k)
            cluster_barrier();
    }
}

struct ClusterLaunch {
    cudaLaunchAttribute attr{};
    cudaLaunchConfig_t cfg{};
    ClusterLaunch(int n, unsigned cols, unsigned planes, cudaStream_t st)
    {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kPCluster;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(3 * kPCluster * n);
        cfg.blockDim = dim3((cols + 31) / 32 * 32);
        cfg.dynamicSmemBytes = 2 * (planes + 2) * cols * sizeof(float4);
        cfg.stream = st;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
};

// Lets the cluster kernels have their shared memory and cluster size on the current device;
// whether it can hold a whole cluster.
bool clusters_fit()
{
    static std::atomic<unsigned long long> asked{0}, fits{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(asked.load() & bit)) {
        const ClusterLaunch most(1, kPClusterThreads, kPClusterPlanes, nullptr);
        bool ok = true;
        auto kernels = {cdm_poisson_cluster_kernel<false, false>, cdm_poisson_cluster_kernel<true, false>,
                        cdm_poisson_cluster_kernel<true, true>};
        for (auto k : kernels) {
            int clusters = 0;
            ok = ok &&
                 cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most.cfg.dynamicSmemBytes) ==
                     cudaSuccess &&
                 cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                 cudaOccupancyMaxActiveClusters(&clusters, k, &most.cfg) == cudaSuccess && clusters > 0;
        }
        if (ok)
            fits.fetch_or(bit);
        else
            (void)cudaGetLastError();  // a "no" is an answer: the next launch is not to report it
        asked.fetch_or(bit);
    }
    return fits.load() & bit;
}

bool cdm_poisson_small(const CdmSeg& s)
{
    return s.ppitch % 4 == 0 && cluster_holds(s.ppitch, s.h, s.d) && clusters_fit();
}

// The sweeps of L's first L.small entries.
cudaError_t launch_poisson_clusters(const CdmSegs& L, cudaStream_t st)
{
    unsigned cols = 0, planes = 0;
    for (int k = 0; k < L.small; ++k) {
        const CdmSeg& s = L.host[k];
        cols = std::max(cols, (unsigned)(s.ppitch / 4 * s.h));
        planes = std::max(planes, (unsigned)((s.d + kPCluster - 1) / kPCluster));
    }
    const ClusterLaunch launch(L.small, cols, planes, st);
    auto kernel = L.small > 1         ? cdm_poisson_cluster_kernel<true, true>
                  : L.host->w % 4 == 0 ? cdm_poisson_cluster_kernel<false, false>
                                       : cdm_poisson_cluster_kernel<true, false>;
    const cudaError_t e = cudaLaunchKernelEx(&launch.cfg, kernel, L.dev, *L.host);
    if (e == cudaSuccess)
        count_launch();
    return e;
}

// An interleaved xyz field to the component planes of a segment's scratch, and back.
__global__ void __launch_bounds__(kCdmThreads) planes_from_xyz_kernel(const float* __restrict__ xyz, Dim3 D,
                                                                      long long pitch, long long plane,
                                                                      float* __restrict__ planes)
{
    const long long n = D.n();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long r = (unsigned)i / (unsigned)D.w, o = r * pitch + (i - r * D.w);
#pragma unroll
        for (int c = 0; c < 3; ++c)
            planes[o + c * plane] = __ldg(xyz + 3 * i + c);
    }
}

__global__ void __launch_bounds__(kCdmThreads) xyz_from_planes_kernel(const float* __restrict__ planes, Dim3 D,
                                                                      long long pitch, long long plane,
                                                                      float* __restrict__ xyz)
{
    const long long n = D.n();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long r = (unsigned)i / (unsigned)D.w, o = r * pitch + (i - r * D.w);
#pragma unroll
        for (int c = 0; c < 3; ++c)
            xyz[3 * i + c] = __ldg(planes + o + c * plane);
    }
}

cudaError_t launch_planes_from_xyz(const float* xyz, const CdmSeg& s, float* planes, cudaStream_t st)
{
    planes_from_xyz_kernel<<<cdm_blocks_for((long long)s.w * s.h * s.d), kCdmThreads, 0, st>>>(
        xyz, Dim3{s.w, s.h, s.d}, s.ppitch, s.pplane, planes);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_xyz_from_planes(const float* planes, const CdmSeg& s, float* xyz, cudaStream_t st)
{
    xyz_from_planes_kernel<<<cdm_blocks_for((long long)s.w * s.h * s.d), kCdmThreads, 0, st>>>(
        planes, Dim3{s.w, s.h, s.d}, s.ppitch, s.pplane, xyz);
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ theta
// cdm_max_displacement_length (reg/cdm.hpp:260-295), only while theta == 0 (the
// first iteration of a level); the last block sets theta and speed/theta, or
// leaves the loop when theta is 0 (reg/cdm.hpp:463-467).
template <bool MULTI>
__global__ void __launch_bounds__(kCdmThreads) cdm_theta_kernel(SEG_ARGS)
{
    SEG_BEGIN
    CdmCtl* c = S.ctl;
    if (c->done || c->theta != 0.0f)
        return;
    const float* __restrict__ d = S.aux_d;
    const long long cs = update_comp(S);
    float m = 0.0f;
    for (long long i = first; i < n; i += stride) {
        const long long o = update_index(S, i);
        const float x = d[o], y = d[o + cs], z = d[o + 2 * cs];
        const float l2 = x * x + y * y + z * z;
        const float l = (float)sqrt((double)l2);
        m = fmaxf(m, l);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0)
        atomicMax(&c->theta_bits, __float_as_uint(m));
    if (!last_block_of_segment(S) || threadIdx.x != 0)
        return;
    const float theta = __uint_as_float(atomicAdd(&c->theta_bits, 0u));
    c->theta = theta;
    if (theta == 0.0f)
        c->done = 1;
    else
        c->scale = c->speed / theta;
}

// ------------------------------------------------------------------ accumulate
// new_d *= speed/theta (reg/cdm.hpp:467) fused with accumulate_displacement
// (numerical/dif.hpp:166-186): out = (cur_d + id)(x + new_d) - x where new_d is
// non-zero and the sample lands inside, else cur_d.  The mapping cur_d + id is
// formed per corner exactly as displacement_to_mapping stores it.  The 2-D form is the
// bilinear sample of the mapping cur_d + (x, y); z stays 0.
struct Accumulate {
    const float *__restrict__ nd, *__restrict__ cd;
    float* __restrict__ out;
    Dim3 D;
    int ndim;
    float scale;
};
// One voxel whose x component sits at o; cs, sx, sy, sz: strides of a component, voxel, row
// and plane.
__device__ __forceinline__ void accumulate_voxel(const Accumulate& A, int x, int y, int z, long long o, long long cs, int sx,
                                                 long long sy, long long sz, float dx, float dy, float dz)
{
    dx *= A.scale;
    dy *= A.scale;
    dz = A.ndim == 2 ? 0.0f : dz * A.scale;
    bool ok = false;
    float ax = 0.0f, ay = 0.0f, az = 0.0f;
    if (dx != 0.0f || dy != 0.0f || dz != 0.0f) {
        dx += (float)x;
        dy += (float)y;
        dz += (float)z;
        const int bx = (int)dx, by = (int)dy, bz = (int)dz;
        const float fx[2] = {(float)bx, (float)(bx + 1)}, fy[2] = {(float)by, (float)(by + 1)};
        if (A.ndim == 2) {
            Cell2 cl;
            ok = bilinear_cell(A.D, dx, dy, cl);
            if (ok) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float* q = A.cd + (by + (k >> 1)) * sy + (long long)bx * sx + (k & 1) * sx;
                    const float mx = q[0] + fx[k & 1], my = q[cs] + fy[k >> 1];
                    ax = k ? ax + mx * cl.r[k] : mx * cl.r[k];
                    ay = k ? ay + my * cl.r[k] : my * cl.r[k];
                }
            }
        } else {
            Cell cl;
            ok = trilinear_cell(A.D, dx, dy, dz, cl);
            if (ok) {
                const float fz[2] = {(float)bz, (float)(bz + 1)};
                const float* const p = A.cd + bz * sz + by * sy + (long long)bx * sx;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float* q = p + (k >> 2) * sz + (k >> 1 & 1) * sy + (k & 1) * sx;
                    const float mx = q[0] + fx[k & 1], my = q[cs] + fy[k >> 1 & 1], mz = q[2 * cs] + fz[k >> 2];
                    ax = k ? ax + mx * cl.r[k] : mx * cl.r[k];
                    ay = k ? ay + my * cl.r[k] : my * cl.r[k];
                    az = k ? az + mz * cl.r[k] : mz * cl.r[k];
                }
            }
        }
    }
    A.out[o] = ok ? ax - (float)x : A.cd[o];
    A.out[o + cs] = ok ? ay - (float)y : A.cd[o + cs];
    A.out[o + 2 * cs] = A.ndim == 2 ? 0.0f : ok ? az - (float)z : A.cd[o + 2 * cs];
}

// Interleaved fields (one accumulate_displacement).
__global__ void __launch_bounds__(kCdmThreads) cdm_accumulate_xyz_kernel(SEG_ARGS)
{
    constexpr bool MULTI = false;
    const CdmSeg& S = segs[0];
    SEG_LOOP
    const CdmCtl* c = S.ctl;
    if (c->done)
        return;
    const Accumulate A{S.aux_d, S.field[c->from], S.tmp_d, D, S.ndim, c->scale};
    for (long long i = first; i < n; i += stride) {
        int x, y, z;
        unflat((int)i, D, x, y, z);
        const long long o = 3 * i;
        accumulate_voxel(A, x, y, z, o, 1, 3, 3LL * D.w, 3LL * D.wh(), A.nd[o], A.nd[o + 1], A.nd[o + 2]);
    }
}

// The voxel at position p of a component, and the one `step` positions on.
struct Place {
    int x, y, z;
    __device__ __forceinline__ Place(unsigned p, unsigned pitch, int h)
    {
        const unsigned r = p / pitch;
        x = (int)(p - r * pitch);
        z = (int)(r / (unsigned)h);
        y = (int)r - z * h;
    }
    __device__ __forceinline__ void advance(unsigned step, unsigned pitch, int h)
    {
        const unsigned rows = step / pitch;
        x += (int)(step - rows * pitch);
        y += (int)rows;
        if (x >= (int)pitch) {
            x -= (int)pitch;
            ++y;
        }
        for (; y >= h; y -= h)
            ++z;
    }
};

// Component planes: 24 gathers a voxel, whose lanes take neighbouring floats.  Bound by the
// chain flag -> update -> cell -> gathers and the L2 traffic of the corner planes; a block
// takes kTile positions, so that the last wave of a launch is short.
// 91x109x91: 14.5 us on interleaved fields with a grid-wide stride, 11.7 so; with 1 / 4 voxels
// a thread 14.9 / 12.4, 32^3 3.5 us against 2.8 / 6.0.
constexpr int kAThreads = kTile / kAVox, kABlocks = 1280 / kAThreads;
template <bool MULTI>
__global__ void __launch_bounds__(kAThreads, kABlocks) cdm_accumulate_kernel(SEG_ARGS)
{
    const CdmSeg& S = SEG_OF(tblk0);
    const int tile = (int)blockIdx.x - (MULTI ? S.tblk0 : 0);
    if (tile >= S.tnb)
        return;
    const CdmCtl* c = S.ctl;
    const Dim3 D{S.w, S.h, S.d};
    const unsigned pitch = (unsigned)S.ppitch, total = (unsigned)S.pplane;
    const unsigned p0 = (unsigned)tile * kTile + threadIdx.x;
    const long long cs = S.pplane;
    // the update's loads go out before the loop flag is waited for
    float n0[kAVox], n1[kAVox], n2[kAVox];
#pragma unroll
    for (int k = 0; k < kAVox; ++k) {
        const unsigned p = p0 + kAThreads * k;
        const float* const q = S.aux_d + p;
        n0[k] = load_now(q, p < total);
        n1[k] = load_now(q + cs, p < total);
        n2[k] = load_now(q + 2 * cs, p < total);
    }
    const int done = c->done, from = c->from;
    const float scale = c->scale;
    if (done)
        return;
    const float* __restrict__ const cd = S.field[from];
    if (S.ndim == 2 || !narrow(S)) {
        const Accumulate A{S.aux_d, cd, S.tmp_d, D, S.ndim, scale};
        for (unsigned p = p0; p < p0 - threadIdx.x + kTile; p += kAThreads) {
            const Place at(p, pitch, D.h);
            const float* const q = A.nd + p;
            if (p < total && at.x < D.w)
                accumulate_voxel(A, at.x, at.y, at.z, p, cs, 1, pitch, (long long)pitch * D.h, q[0], q[cs], q[2 * cs]);
        }
        return;
    }
    // below, offsets in bytes fit 32 bits and coordinates are exact floats
    const SampleGeo G{D.w, D.h, 0, (float)(D.w - 1), (float)(D.h - 1), (float)(D.d - 1)};
    const char* const base[3] = {(const char*)cd, (const char*)(cd + cs), (const char*)(cd + 2 * cs)};
    const unsigned plane = pitch * (unsigned)D.h;
    Place at(p0, pitch, D.h);
#pragma unroll
    for (int k = 0; k < kAVox; ++k) {
        const unsigned p = p0 + kAThreads * k;
        if (p < total && at.x < D.w) {
            const float dx = n0[k] * scale, dy = n1[k] * scale, dz = n2[k] * scale;
            const float X = u8_to_f(at.x), Y = u8_to_f(at.y), Z = u8_to_f(at.z), px = dx + X, py = dy + Y, pz = dz + Z;
            float* const o = S.tmp_d + p;
            if (!(dx == 0.0f && dy == 0.0f && dz == 0.0f) && !(px < 0.0f || py < 0.0f || pz < 0.0f) && px < G.wl &&
                py < G.hl && pz < G.dl) {
                float f[3][2], r[8];
                const unsigned b = 4u * narrow_cell(px, py, pz, pitch, (unsigned)D.h, f, r);
                float a[3];
#pragma unroll
                for (int v = 0; v < 8; ++v) {
                    const unsigned off = b + 4u * ((v >> 1 & 1) * pitch + (v >> 2) * plane);
#pragma unroll
                    for (int t = 0; t < 3; ++t) {
                        const float m = __ldg((const float*)(base[t] + off) + (v & 1)) + f[t][v >> t & 1];
                        a[t] = v ? a[t] + m * r[v] : m * r[v];
                    }
                }
                o[0] = a[0] - X;
                o[cs] = a[1] - Y;
                o[2 * cs] = a[2] - Z;
            } else {
                o[0] = __ldg(cd + p);
                o[cs] = __ldg(cd + p + cs);
                o[2 * cs] = __ldg(cd + p + 2 * cs);
            }
        }
        if (k + 1 < kAVox)
            at.advance(kAThreads, pitch, D.h);
    }
}

// ------------------------------------------------------------------ smooth
// cdm_smooth (reg/cdm.hpp:302-366): cur_d = d*(1-s) + (s/6) * (d[+1] + d[-1] +
// d[+w] + d[-w] + d[+wh] + d[-wh]) by flat index; s == 0 leaves cur_d as it is.
// 2-D: s/4 and four neighbours (the +-wh taps of a d == 1 level fall outside).
__device__ __forceinline__ float smooth_weight(const CdmSeg& S, float sm)
{
    return sm / (2.0f * (S.ndim == 2 ? 2.0f : 3.0f));  // smoothing / (2 * dimension)
}

// An interleaved field, a float a thread.
__global__ void __launch_bounds__(kCdmThreads) cdm_smooth_kernel(SEG_ARGS)
{
    constexpr bool MULTI = false;
    SEG_BEGIN
    const CdmCtl* c = S.ctl;
    if (c->done)
        return;
    const float sm = c->cur_smoothing;
    if (sm == 0.0f)
        return;
    const float w_6 = smooth_weight(S, sm), w_1 = 1.0f - sm;
    const float* __restrict__ d = S.tmp_d;
    float* __restrict__ dd = S.field[c->cur];
    const long long N3 = 3 * n, w3 = 3 * (long long)D.w, wh3 = 3 * (long long)D.wh();
    for (long long f = first; f < N3; f += stride) {
        float v = 0.0f;
        if (f + 3 < N3) v += d[f + 3];
        if (f >= 3) v += d[f - 3];
        if (f + w3 < N3) v += d[f + w3];
        if (f >= w3) v += d[f - w3];
        if (f + wh3 < N3) v += d[f + wh3];
        if (f >= wh3) v += d[f - wh3];
        v *= w_6;
        dd[f] = d[f] * w_1 + v;
    }
}

// An iteration's smoothing and the next one's compose of the first modality in one pass over
// the component planes: a thread smooths a float4 of each component (taps as in the Poisson
// sweeps), and a warp hands its 128 voxels over through shared memory to sample them 32
// neighbours at a time.  91x109x91 uint8: 17.9 us as two launches over interleaved fields
// (seven scalar loads a float), 11.8 so.
template <typename T, bool MULTI>
__global__ void __launch_bounds__(kTThreads) cdm_smooth_compose_kernel(SEG_ARGS)
{
    const CdmSeg& S = SEG_OF(tblk0);
    const int tile = (int)blockIdx.x - (MULTI ? S.tblk0 : 0);
    if (tile >= S.tnb)
        return;
    const CdmCtl* c = S.ctl;
    if (c->done)
        return;
    const float sm = c->cur_smoothing;
    const float w_6 = smooth_weight(S, sm), w_1 = 1.0f - sm;
    float* const dst = S.field[c->cur];
    const T* __restrict__ const Is = (const T*)S.Is[0];
    T* __restrict__ const Js = (T*)S.Js;
    const Dim3 D{S.w, S.h, S.d};
    const unsigned pitch = (unsigned)S.ppitch;
    const unsigned tp = (unsigned)tile * kTile;  // the tile's first position
    const int lane = threadIdx.x & 31, warp = threadIdx.x & ~31;
    __shared__ float4 field[3][kTThreads];
    if ((pitch & 3) == 0) {
        const unsigned P = pitch / 4, plane = P * (unsigned)D.h, total = plane * (unsigned)D.d;
        const unsigned i = tp / 4 + threadIdx.x, xq = i % P;
        const int rem = D.w & 3;
        const bool on = i < total, row_end = xq == P - 1;
        const bool fix1 = row_end && rem == 1, fix2 = row_end && rem == 2, fix3 = row_end && rem == 3;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float4* const in = reinterpret_cast<const float4*>(S.tmp_d + k * S.pplane);
            float4* const out = reinterpret_cast<float4*>(dst + k * S.pplane);
            auto at = [&](unsigned j) {
                return on && j < total ? __ldg(in + j) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            };
            auto one = [&](long long j) {
                return on && j >= 0 && j < 4LL * total ? __ldg(reinterpret_cast<const float*>(in) + j) : 0.0f;
            };
            float4 r;
            if (sm == 0.0f)
                r = on ? out[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            else {
                const float4 cur = at(i), ya = at(i - P), yb = at(i + P), down = at(i - plane), up = at(i + plane);
                const float tail = fix1 ? cur.x : fix2 ? cur.y : fix3 ? cur.z : cur.w;
                float xl = __shfl_up_sync(0xffffffffu, tail, 1), xr = __shfl_down_sync(0xffffffffu, cur.x, 1);
                if (lane == 0)
                    xl = one(4LL * i - 1 - (xq == 0 && rem ? 4 - rem : 0));
                if (lane == 31 || i + 1 == total)
                    xr = one(4LL * i + 4);
                const float n1 = fix1 ? xr : cur.y, n2 = fix2 ? xr : cur.z, n3 = fix3 ? xr : cur.w;
                r.x = cur.x * w_1 + ((((((0.0f + n1) + xl) + yb.x) + ya.x) + up.x) + down.x) * w_6;
                r.y = cur.y * w_1 + ((((((0.0f + n2) + cur.x) + yb.y) + ya.y) + up.y) + down.y) * w_6;
                r.z = cur.z * w_1 + ((((((0.0f + n3) + cur.y) + yb.z) + ya.z) + up.z) + down.z) * w_6;
                r.w = cur.w * w_1 + ((((((0.0f + xr) + cur.z) + yb.w) + ya.w) + up.w) + down.w) * w_6;
                if (on)
                    out[i] = r;
            }
            field[k][threadIdx.x] = r;
        }
    } else {  // unpadded rows: a float at a time
        const long long w = D.w, wh = D.wh(), n = D.n();
        for (int k = 0; k < 3; ++k)
            for (int j = 0; j < 4; ++j) {
                const int v = 4 * warp + 32 * j + lane;
                const long long i = (long long)tp + v;
                const float* __restrict__ const d = S.tmp_d + k * S.pplane;
                float* const out = dst + k * S.pplane;
                if (i >= n)
                    continue;
                float r;
                if (sm == 0.0f)
                    r = out[i];
                else {
                    float a = 0.0f;
                    if (i + 1 < n) a += d[i + 1];
                    if (i >= 1) a += d[i - 1];
                    if (i + w < n) a += d[i + w];
                    if (i >= w) a += d[i - w];
                    if (i + wh < n) a += d[i + wh];
                    if (i >= wh) a += d[i - wh];
                    a *= w_6;
                    r = d[i] * w_1 + a;
                    out[i] = r;
                }
                reinterpret_cast<float*>(field[k])[v] = r;
            }
    }
    __syncwarp();
    const bool fast = S.ndim != 2 && narrow(S);
    const SampleGeo G = sample_geo(D);
    const int v0 = 4 * warp + lane;
    Place at(tp + v0, pitch, D.h);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int v = v0 + 32 * k;
        const float dx = reinterpret_cast<const float*>(field[0])[v], dy = reinterpret_cast<const float*>(field[1])[v],
                    dz = reinterpret_cast<const float*>(field[2])[v];
        if (at.z < D.d && at.x < D.w) {
            const int j = (at.z * D.h + at.y) * D.w + at.x;
            Js[j] = fast ? compose_narrow(Is, G, (unsigned)j, at.x, at.y, at.z, dx, dy, dz)
                         : compose_pixel(Is, D, S.ndim, j, at.x, at.y, at.z, dx, dy, dz);
        }
        if (k < 3)
            at.advance(32, pitch, D.h);
    }
}

// ------------------------------------------------------------------ pyramid
// downsample_with_padding (numerical/resampling.hpp:575-603): 2x box mean; a
// missing +1 neighbour repeats the nearest present one; integer pixels sum in
// 16 bits and shift by 3, float pixels divide by 8.
template <typename T>
__global__ void downsample_kernel(const T* __restrict__ in, Dim3 di, T* __restrict__ out, Dim3 dout)
{
    const long long n = dout.n();
    const long long w = di.w, wh = (long long)di.wh();
    const long long shift[8] = {0, 1, w, 1 + w, wh, wh + 1, wh + w, wh + 1 + w};
    for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < n; o += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        unflat((int)o, dout, x, y, z);
        const int x2 = 2 * x, y2 = 2 * y, z2 = 2 * z;
        int has = 0;
        if (x2 + 1 < di.w) has += 1;
        if (y2 + 1 < di.h) has += 2;
        if (z2 + 1 < di.d) has += 4;
        const long long base = ((long long)z2 * di.h + y2) * di.w + x2;
        T buf[8];
        buf[0] = in[base];
        if constexpr (sizeof(T) == 1) {
            unsigned int acc = buf[0];
#pragma unroll
            for (int k = 1; k < 8; ++k) {
                const int h = has & k;
                buf[k] = (h == k) ? in[base + shift[k]] : buf[h];
                acc = (acc + buf[k]) & 0xffffu;
            }
            out[o] = (T)(acc >> 3);
        } else {
            T acc = buf[0];
#pragma unroll
            for (int k = 1; k < 8; ++k) {
                const int h = has & k;
                buf[k] = (h == k) ? in[base + shift[k]] : buf[h];
                acc += buf[k];
            }
            out[o] = acc / 8;
        }
    }
}

cudaError_t launch_downsample(const void* in, void* out, int w, int h, int d, int pix, cudaStream_t st)
{
    Dim3 di{w, h, d}, dout{(w + 1) / 2, (h + 1) / 2, (d + 1) / 2};
    int blocks = cdm_blocks_for(dout.n());
    if (pix == 0)
        downsample_kernel<uint8_t><<<blocks, kCdmThreads, 0, st>>>((const uint8_t*)in, di, (uint8_t*)out, dout);
    else
        downsample_kernel<float><<<blocks, kCdmThreads, 0, st>>>((const float*)in, di, (float*)out, dout);
    count_launch();
    return cudaGetLastError();
}

// best_d *= 2; upsample_with_padding (reg/cdm.hpp:402-403,
// numerical/resampling.hpp:849-891): out(x) = trilinear(2*in, x * 0.5), 0 where the
// sample fails.  The doubling is exact, so it is applied to the corner values.
__global__ void upsample_x2_kernel(const float* __restrict__ in, Dim3 di, float* __restrict__ out, Dim3 dout)
{
    const long long n = dout.n();
    for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < n; o += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        unflat((int)o, dout, x, y, z);
        float vx = (float)x, vy = (float)y, vz = (float)z;
        vx *= 0.5f;
        vy *= 0.5f;
        vz *= 0.5f;
        Cell c;
        float3 v = make_float3(0.f, 0.f, 0.f);
        if (trilinear_cell(di, vx, vy, vz, c)) {
            const int w = di.w, wh = di.wh(), b = c.base;
            const int off[8] = {0, 1, w, w + 1, wh, wh + 1, wh + w, wh + w + 1};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float* q = in + 3LL * (b + off[k]);
                const float qx = q[0] * 2.0f, qy = q[1] * 2.0f, qz = q[2] * 2.0f;
                if (k == 0) {
                    v.x = qx * c.r[0];
                    v.y = qy * c.r[0];
                    v.z = qz * c.r[0];
                } else {
                    v.x += qx * c.r[k];
                    v.y += qy * c.r[k];
                    v.z += qz * c.r[k];
                }
            }
        }
        out[3 * o] = v.x;
        out[3 * o + 1] = v.y;
        out[3 * o + 2] = v.z;
    }
}

// The 2-D form (vector<2> field of a d == 1 level): bilinear at (x, y) * 0.5; z is 0.
__global__ void upsample_x2_2d_kernel(const float* __restrict__ in, Dim3 di, float* __restrict__ out, Dim3 dout)
{
    const long long n = dout.n();
    for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < n; o += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(o % dout.w), y = (int)(o / dout.w);
        float vx = (float)x, vy = (float)y;
        vx *= 0.5f;
        vy *= 0.5f;
        Cell2 c;
        float2 v = make_float2(0.f, 0.f);
        if (bilinear_cell(di, vx, vy, c)) {
            const int w = di.w, b = c.base;
            const int off[4] = {0, 1, w, w + 1};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float* q = in + 3LL * (b + off[k]);
                const float qx = q[0] * 2.0f, qy = q[1] * 2.0f;
                if (k == 0) {
                    v.x = qx * c.r[0];
                    v.y = qy * c.r[0];
                } else {
                    v.x += qx * c.r[k];
                    v.y += qy * c.r[k];
                }
            }
        }
        out[3 * o] = v.x;
        out[3 * o + 1] = v.y;
        out[3 * o + 2] = 0.0f;
    }
}

cudaError_t launch_upsample_field_x2(const float* in, int iw, int ih, int id, float* out, int ow, int oh, int od,
                                     cudaStream_t st, int ndim)
{
    Dim3 di{iw, ih, id}, dout{ow, oh, od};
    if (ndim == 2)
        upsample_x2_2d_kernel<<<cdm_blocks_for(dout.n()), kCdmThreads, 0, st>>>(in, di, out, dout);
    else
        upsample_x2_kernel<<<cdm_blocks_for(dout.n()), kCdmThreads, 0, st>>>(in, di, out, dout);
    count_launch();
    return cudaGetLastError();
}

__global__ void field_xy_kernel(const float* __restrict__ xyz, long long n, float* __restrict__ xy)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        xy[2 * i] = xyz[3 * i];
        xy[2 * i + 1] = xyz[3 * i + 1];
    }
}

cudaError_t launch_field_xy(const float* xyz, long long n, float* xy, cudaStream_t st)
{
    if (n <= 0)
        return cudaSuccess;
    field_xy_kernel<<<cdm_blocks_for(n), kCdmThreads, 0, st>>>(xyz, n, xy);
    count_launch();
    return cudaGetLastError();
}

__global__ void cost_mean_kernel(const CdmSeg* __restrict__ segs, float* __restrict__ out)
{
    const float m = seg_cost_mean(segs[blockIdx.y]);
    if (threadIdx.x == 0)
        out[blockIdx.y] = m;
}

cudaError_t launch_cost_mean(const CdmSeg* segs, int nseg, float* out, cudaStream_t st)
{
    cost_mean_kernel<<<dim3(1, nseg), 256, 0, st>>>(segs, out);
    count_launch();
    return cudaGetLastError();
}

// done flags of many segments gathered into one array (one read-back per round)
__global__ void cdm_status_kernel(const CdmSeg* __restrict__ segs, int n, int* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = segs[i].ctl->done;
}

cudaError_t launch_cdm_status(const CdmSeg* segs, int nseg, int* out, cudaStream_t st)
{
    if (nseg <= 0)
        return cudaSuccess;
    cdm_status_kernel<<<(nseg + 127) / 128, 128, 0, st>>>(segs, nseg, out);
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ launchers
#define SEG_LAUNCH(multi, single, threads, smem, ...)                                      \
    do {                                                                                   \
        if (L.n > 1)                                                                       \
            multi<<<L.blocks, threads, smem, st>>>(L.dev, L.n, *L.host, ##__VA_ARGS__);    \
        else                                                                               \
            single<<<L.blocks, threads, smem, st>>>(L.dev, L.n, *L.host, ##__VA_ARGS__);   \
    } while (0)

cudaError_t launch_cdm_compose(const CdmSegs& L, int pix, cudaStream_t st, int mod)
{
    if (mod < 0 || mod >= kCdmMaxModalities)
        return cudaErrorInvalidValue;
    if (L.host->planar) {
        if (pix == 0)
            SEG_LAUNCH((cdm_compose_kernel<uint8_t, true, true>), (cdm_compose_kernel<uint8_t, false, true>), kCdmThreads,
                       0, mod);
        else
            SEG_LAUNCH((cdm_compose_kernel<float, true, true>), (cdm_compose_kernel<float, false, true>), kCdmThreads, 0,
                       mod);
    } else if (L.n == 1) {
        auto kernel = pix ? cdm_compose_kernel<float, false, false> : cdm_compose_kernel<uint8_t, false, false>;
        kernel<<<L.blocks, kCdmThreads, 0, st>>>(L.dev, L.n, *L.host, mod);
    } else
        return cudaErrorInvalidValue;
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_cdm_gradient(const CdmSegs& L, int pix, int gradient_type,
                                cudaStream_t st, int mod)
{
    if (mod < 0 || mod >= kCdmMaxModalities)
        return cudaErrorInvalidValue;
    if (pix == 0 && gradient_type == 'r') {
        static std::atomic<unsigned long long> attr_set{0};
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess)
            return e;
        const unsigned long long bit = 1ull << (dev & 63);
        if (!(attr_set.load() & bit)) {
            e = cudaFuncSetAttribute(cdm_gradient_box_u8_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     box_smem<8>());
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(cdm_gradient_box_u8_kernel<false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, box_smem<8>());
            if (e != cudaSuccess)
                return e;
            attr_set.fetch_or(bit);
        }
        SEG_LAUNCH(cdm_gradient_box_u8_kernel<true>, cdm_gradient_box_u8_kernel<false>, kUThreads,
                   box_smem<8>(), mod);
    } else if (gradient_type == 'r' && L.n == 1 && L.host->each)
        cdm_gradient_r_f32_each_kernel<<<L.blocks, kFThreads, 0, st>>>(L.dev, L.n, *L.host, mod);
    else if (gradient_type == 'r')
        SEG_LAUNCH(cdm_gradient_r_f32_kernel<true>, cdm_gradient_r_f32_kernel<false>, kFThreads, 0, mod);
    else if (pix == 0)
        SEG_LAUNCH((cdm_gradient_d_kernel<uint8_t, true>), (cdm_gradient_d_kernel<uint8_t, false>), kCdmThreads, 0, mod);
    else
        SEG_LAUNCH((cdm_gradient_d_kernel<float, true>), (cdm_gradient_d_kernel<float, false>), kCdmThreads, 0, mod);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_cdm_poisson(const CdmSegs& L, cudaStream_t st)
{
    if (L.small) {
        const cudaError_t e = launch_poisson_clusters(L, st);
        if (e != cudaSuccess)
            return e;
    }
    const int n = L.n - L.small;
    if (n == 0)
        return cudaSuccess;
    const bool flat = n == 1 && (L.host[L.small].ppitch & 3);
    for (int k = 0; k < kPSweeps; ++k) {
        auto kernel = n > 1  ? (k ? cdm_poisson_kernel<false, true> : cdm_poisson_kernel<true, true>)
                      : flat ? (k ? cdm_poisson_flat_kernel<false> : cdm_poisson_flat_kernel<true>)
                             : (k ? cdm_poisson_kernel<false, false> : cdm_poisson_kernel<true, false>);
        kernel<<<L.pblocks, kPThreads, 0, st>>>(L.dev + L.small, n, L.host[L.small], k & 1);
    }
    count_launch(kPSweeps);
    return cudaGetLastError();
}

cudaError_t launch_cdm_theta(const CdmSegs& L, cudaStream_t st)
{
    SEG_LAUNCH(cdm_theta_kernel<true>, cdm_theta_kernel<false>, kCdmThreads, 0);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_cdm_accumulate(const CdmSegs& L, cudaStream_t st)
{
    if (L.host->planar) {
        auto kernel = L.n > 1 ? cdm_accumulate_kernel<true> : cdm_accumulate_kernel<false>;
        kernel<<<L.tblocks, kAThreads, 0, st>>>(L.dev, L.n, *L.host);
    } else if (L.n == 1)
        cdm_accumulate_xyz_kernel<<<L.blocks, kCdmThreads, 0, st>>>(L.dev, L.n, *L.host);
    else
        return cudaErrorInvalidValue;
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_cdm_smooth(const CdmSegs& L, cudaStream_t st)
{
    if (L.n != 1 || L.host->planar)
        return cudaErrorInvalidValue;
    cdm_smooth_kernel<<<L.blocks, kCdmThreads, 0, st>>>(L.dev, L.n, *L.host);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_cdm_smooth_compose(const CdmSegs& L, int pix, cudaStream_t st)
{
    auto kernel = L.n > 1 ? (pix ? cdm_smooth_compose_kernel<float, true> : cdm_smooth_compose_kernel<uint8_t, true>)
                          : (pix ? cdm_smooth_compose_kernel<float, false> : cdm_smooth_compose_kernel<uint8_t, false>);
    kernel<<<L.tblocks, kTThreads, 0, st>>>(L.dev, L.n, *L.host);
    count_launch();
    return cudaGetLastError();
}

}  // namespace regb
