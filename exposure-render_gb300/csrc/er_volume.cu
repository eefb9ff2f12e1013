/*
 * er_volume.cu - per-volume pre-passes of the free-flight estimators.
 *
 *   k_brick_minmax : min and max voxel of every brick's footprint: voxels
 *                    b B .. (b + 1) B per axis, every corner a trilinear
 *                    lookup (Source/buffer3d.h:222-242) at local coordinates
 *                    in [b B, (b + 1) B] can blend with a nonzero weight (the
 *                    trackers clamp their lookups to that range,
 *                    er_path.cuh sigma_point_in_brick).
 *   k_rmq, k_rmq_tile, k_rmq_level : sparse table of running maxima over the
 *                    sigma table (sigma[I] = DensityScale * Opacity(I)).
 *   k_majorant     : majorant[brick] = DensityScale * max sigma[lo..hi].
 *   k_skip_x, _yz  : distances to the nearest non-empty brick.
 *   k_occupancy    : the empty bricks of the fixed-step march.
 *
 * A lookup inside a brick is a truncated trilinear blend of voxels in
 * [lo, hi]; float rounding of a blend (1 - t) a + t b can fall just below
 * min(a, b), which the truncation turns into one intensity less, so its
 * integer intensity lies in [lo - 1, hi] and its extinction
 * DensityScale * sigma[I] is bounded by the max over that range exactly
 * (max of the same floats, one multiply).  The CPU oracle builds the same grid by
 * brute force; the tests compare them bit for bit through the rendered paths.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <cstdio>
#include <type_traits>

#include "er_capi.h"
#include "er_kernels.h"

/* Min and max voxel of every brick's footprint, lo | hi << 16.

   Bound by the read of the volume.  A block owns one row of bricks in y, a
   range of bricks in z and BM_X voxels in x, and walks z plane by plane:
   each thread reduces the B + 1 rows of its VEC voxels in a plane (coalesced
   along x, rows of a plane independent loads), a plane that two bricks share
   in z is read once, and the rows that neighbouring blocks share in y come
   from L2.  When a brick's last plane is in, the per-x values go through
   shared memory and one thread per brick takes the B + 1 values of its x
   range.  One warp per brick, which it replaces, put 5 voxels of a row on 32
   lanes at 4^3 bricks and took 3.79 ms at 512^3; an edit of the transfer
   function of that volume with a one-sample picture went from 5.8 to 1.9 ms
   with this kernel, k_rmq and outward distance passes. */
#define BM_THREADS 160

template <int VEC>
__global__ void __launch_bounds__(BM_THREADS) k_brick_minmax(const uint16_t* __restrict__ vox, int rx, int ry, int rz, int B, int nbx,
                                                             int nby, int nbz, int xbricks, int zbricks, int xblocks,
                                                             uint32_t* __restrict__ minmax)
{
    /* per-x values of the open brick row: (lo, 65535 - hi) packed, so that one
       packed minimum serves both; two buffers, so that one barrier a brick suffices */
    __shared__ uint32_t cols[2][BM_THREADS * VEC];
    const unsigned row_id = blockIdx.x / (unsigned)xblocks;
    const int by = (int)(row_id % (unsigned)nby);
    const int bx0 = (int)(blockIdx.x % (unsigned)xblocks) * xbricks, bx1 = min(bx0 + xbricks, nbx);
    const int bz0 = (int)(row_id / (unsigned)nby) * zbricks, bz1 = min(bz0 + zbricks, nbz);
    const int xs = bx0 * B;
    const int xw = min(bx1 * B, rx - 1) - xs + 1;                 /* voxels of the block's rows */
    const int y0 = by * B, y1 = min(y0 + B, ry - 1);
    const int x = (int)threadIdx.x * VEC;
    const bool in = x < xw;
    /* a pair's second voxel may lie past the row's last used one but not past the row (rx is even then) */
    uint32_t open[VEC], plane[VEC];
#pragma unroll
    for (int v = 0; v < VEC; v++) open[v] = 0xffffffffu;
    int buf = 0;
    const int z_end = min(bz1 * B, rz - 1);
    int z = bz0 * B, bz = bz0;
    for (; z <= z_end; z++) {
#pragma unroll
        for (int v = 0; v < VEC; v++) plane[v] = 0xffffffffu;
        if (in) {
            const uint16_t* row = vox + ((size_t)z * ry + y0) * (size_t)rx + xs + x;
#pragma unroll 4
            for (int y = y0; y <= y1; y++, row += rx) {
                if (VEC == 2) {
                    const uint32_t w = __ldg((const uint32_t*)row);
                    const uint32_t a = w & 0xffffu, b = w >> 16;
                    plane[0] = __vminu2(plane[0], a | ((0xffffu ^ a) << 16));
                    plane[VEC - 1] = __vminu2(plane[VEC - 1], b | ((0xffffu ^ b) << 16));
                } else {
                    const uint32_t a = __ldg(row);
                    plane[0] = __vminu2(plane[0], a | ((0xffffu ^ a) << 16));
                }
            }
        }
#pragma unroll
        for (int v = 0; v < VEC; v++) open[v] = __vminu2(open[v], plane[v]);
        /* brick bz ends with plane (bz + 1) B, or with the volume */
        if (z == (bz + 1) * B || z == rz - 1) {
#pragma unroll
            for (int v = 0; v < VEC; v++) {
                cols[buf][x + v] = open[v];
                open[v] = plane[v];
            }
            __syncthreads();
            for (int b = bx0 + (int)threadIdx.x; b < bx1; b += BM_THREADS) {
                const int c0 = b * B - xs, c1 = min((b + 1) * B, rx - 1) - xs;
                uint32_t m = 0xffffffffu;
                for (int c = c0; c <= c1; c++) m = __vminu2(m, cols[buf][c]);
                minmax[((size_t)bz * nby + by) * (size_t)nbx + b] = m ^ 0xffff0000u;
            }
            buf ^= 1;
            bz++;
            /* the last voxel plane of a volume that bricks divide without a
               remainder plus one also closes the brick after it */
            if (z == rz - 1 && bz < bz1) {
                z--;
#pragma unroll
                for (int v = 0; v < VEC; v++) open[v] = 0xffffffffu;
            }
        }
    }
}

/* The sparse table of running maxima, level 0 a copy of the sigma table.  A
   level needs the one before it.  Short tables: one block makes all levels,
   each in a few of its iterations (a launch a level took 3 us each, 33 us at
   n = 2600).  Long ones: blocks of RMQ_TILE entries make the levels that reach
   no further than a tile from it, in shared memory, and the rest are a launch
   each.  A majorant grid of 64^3 voxels at n = 2600, 16384 and 65536, us: one
   block 21, 44 and 266, tiles 18, 32 and 42, a launch a level 57, 81 and 90. */
__global__ void __launch_bounds__(1024) k_rmq(const float* __restrict__ sigma, float* __restrict__ table, int n, int levels)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) table[i] = sigma[i];
    for (int k = 1; k < levels; k++) {
        __syncthreads();
        const float* prev = table + (size_t)(k - 1) * n;
        float* next = table + (size_t)k * n;
        const int half = 1 << (k - 1);
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float a = prev[i];
            const float b = (i + half < n) ? prev[i + half] : a;
            next[i] = b > a ? b : a;
        }
    }
}

#define RMQ_TILE 1024
#define RMQ_TILE_LEVELS 11      /* levels 0 .. 10 reach 1023 entries further */

__global__ void __launch_bounds__(RMQ_TILE) k_rmq_tile(const float* __restrict__ sigma, float* __restrict__ table, int n, int levels)
{
    __shared__ float v[2 * RMQ_TILE];
    const int t = threadIdx.x, i0 = blockIdx.x * RMQ_TILE;
    float a[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int p = t + j * RMQ_TILE;
        a[j] = i0 + p < n ? sigma[i0 + p] : 0.0f;
        v[p] = a[j];
    }
    if (i0 + t < n) table[i0 + t] = a[0];
    for (int k = 1; k < levels && k < RMQ_TILE_LEVELS; k++) {
        const int half = 1 << (k - 1);
        __syncthreads();
        float b[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int p = t + j * RMQ_TILE;
            b[j] = (p + half < 2 * RMQ_TILE && i0 + p + half < n) ? v[p + half] : a[j];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 2; j++) {
            a[j] = b[j] > a[j] ? b[j] : a[j];
            v[t + j * RMQ_TILE] = a[j];
        }
        if (i0 + t < n) table[(size_t)k * n + i0 + t] = a[0];
    }
}

__global__ void k_rmq_level(const float* __restrict__ prev, float* __restrict__ next, int n, int half)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float a = prev[i];
    const float b = (i + half < n) ? prev[i + half] : a;
    next[i] = b > a ? b : a;
}

static void launch_rmq(const float* sigma, float* table, int n, int levels, cudaStream_t s)
{
    if (n <= 4 * RMQ_TILE) {
        k_rmq<<<1, 1024, 0, s>>>(sigma, table, n, levels);
        return;
    }
    k_rmq_tile<<<(n + RMQ_TILE - 1) / RMQ_TILE, RMQ_TILE, 0, s>>>(sigma, table, n, levels);
    for (int k = RMQ_TILE_LEVELS; k < levels; k++)
        k_rmq_level<<<(n + 255) / 256, 256, 0, s>>>(table + (size_t)(k - 1) * n, table + (size_t)k * n, n, 1 << (k - 1));
}

__global__ void k_majorant(const uint32_t* __restrict__ minmax, const float* __restrict__ table, int n, int levels, float ds,
                           float* __restrict__ majorant, long long total)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const uint32_t mm = minmax[i];
    int lo = (int)(mm & 0xffffu) - 1, hi = (int)(mm >> 16);
    lo = lo < 0 ? 0 : (lo > n - 1 ? n - 1 : lo);
    hi = hi > n - 1 ? n - 1 : hi;
    const int len = hi - lo + 1;
    int k = 31 - __clz(len);
    k = k > levels - 1 ? levels - 1 : k;
    const float* lvl = table + (size_t)k * n;
    const float a = lvl[lo];
    const float b = lvl[hi - (1 << k) + 1];
    float m = b > a ? b : a;
    m = m > 0.0f ? m : 0.0f;
    majorant[i] = ds * m;
}

/* launches k_brick_minmax: blocks of at most BM_THREADS voxel pairs (or
   voxels, when the rows are not 4-byte aligned) in x, evenly filled, and z
   ranges short enough for about 16 blocks per SM (each range reads one plane
   more than its bricks) */
static void launch_minmax(const uint16_t* vox, const int res[3], int B, const int nb[3], uint32_t* minmax, cudaStream_t s)
{
    const bool pairs = (res[0] & 1) == 0 && ((uintptr_t)vox & 3u) == 0;
    const int most = (BM_THREADS * (pairs ? 2 : 1) - 1) / B;
    int xblocks = (nb[0] + most - 1) / most;
    int xbricks = (nb[0] + xblocks - 1) / xblocks;
    /* a pair starts at an even voxel: an even number of voxels per block */
    if (pairs && ((xbricks * B) & 1)) xbricks += xbricks < most ? 1 : -1;
    if (xbricks < 1) xbricks = 1;
    xblocks = (nb[0] + xbricks - 1) / xbricks;
    const long long rows = (long long)xblocks * nb[1];
    const long long want = 152ll * 16;
    int zblocks = rows >= want ? 1 : (int)((want + rows - 1) / rows);
    if (zblocks > nb[2]) zblocks = nb[2];
    const int zbricks = (nb[2] + zblocks - 1) / zblocks;
    zblocks = (nb[2] + zbricks - 1) / zbricks;
    const unsigned grid = (unsigned)(rows * zblocks);
    if (pairs)
        k_brick_minmax<2><<<grid, BM_THREADS, 0, s>>>(vox, res[0], res[1], res[2], B, nb[0], nb[1], nb[2], xbricks, zbricks, xblocks, minmax);
    else
        k_brick_minmax<1><<<grid, BM_THREADS, 0, s>>>(vox, res[0], res[1], res[2], B, nb[0], nb[1], nb[2], xbricks, zbricks, xblocks, minmax);
}

__global__ void k_sample_voxels(const uint16_t* __restrict__ vox, size_t n, int step, uint16_t* __restrict__ out)
{
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i * step < n; i += stride) out[i] = vox[i * step];
}

cudaError_t er_launch_sample_voxels(const uint16_t* vox, size_t n, int step, uint16_t* out, cudaStream_t s)
{
    k_sample_voxels<<<1216, 256, 0, s>>>(vox, n, step, out);
    return cudaGetLastError();
}

cudaError_t er_launch_majorant(const uint16_t* vox, const int res[3], int B, const int nb[3], const float* sigma, int n,
                               float* rmq, int levels, uint32_t* minmax, float density_scale, float* majorant, cudaStream_t s)
{
    const long long total = (long long)nb[0] * nb[1] * nb[2];
    launch_minmax(vox, res, B, nb, minmax, s);
    launch_rmq(sigma, rmq, n, levels, s);
    k_majorant<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(minmax, rmq, n, levels, density_scale, majorant, total);
    return cudaGetLastError();
}

/* Empty-space distances of a brick grid.  For an empty brick dist = min over
   non-empty bricks q of max_a |b_a - q_a| (Chebyshev distance in bricks),
   capped at ER_SKIP_CAP; computed exactly by three 1D passes (x: nearest
   non-empty along the row; y and z: min over offsets of max(offset, previous
   pass)).  A ray in a brick at distance dist knows every brick within dist-1
   of it is empty too (er_path.cuh dda_jump, march_skip).

   k_skip_x: a warp takes 32 bricks of a row; the occupancy of them and of the
   32 on either side are three ballots, and the nearest set bits give the
   distance (below 32, so the neighbours' words suffice).  k_skip_yz looks
   outwards and stops at the first offset that is no smaller than the best
   distance so far; four bricks of a row to a thread where the rows are whole
   words.  Loops over the 63 bricks of the cap's window took 94 us a pass at
   128^3 bricks, outward ones, a brick to a thread, 53 us. */
#define ER_SKIP_CAP 32

/* MARCH: `occ` holds k_occupancy's bytes (0: not empty); else a brick is empty
   where its majorant is not positive */
template <int MARCH>
__global__ void __launch_bounds__(256) k_skip_x(const float* __restrict__ majorant, const uint8_t* __restrict__ occ,
                                                uint8_t* __restrict__ out, int nbx, long long rows)
{
    const int lane = threadIdx.x & 31;
    const int words = (nbx + 31) / 32;
    const long long total = rows * words, stride = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < total; w += stride) {
        const long long row = (w / words) * nbx;
        const int x = (int)(w % words) * 32 + lane;
        auto full = [&](int c) -> bool {
            if (c < 0 || c >= nbx) return false;
            return MARCH ? occ[row + c] == 0 : majorant[row + c] > 0.0f;
        };
        const unsigned l = __ballot_sync(0xffffffffu, full(x - 32)), m = __ballot_sync(0xffffffffu, full(x)),
                       r = __ballot_sync(0xffffffffu, full(x + 32));
        if (x >= nbx) continue;
        /* bits of the bricks at and right of x (bit 0: x), and at and left of it (bit 31: x) */
        const unsigned right = __funnelshift_r(m, r, lane), left = __funnelshift_l(l, m, 31 - lane);
        const int dr = right ? __ffs(right) - 1 : ER_SKIP_CAP, dl = left ? __clz(left) : ER_SKIP_CAP;
        out[row + x] = (uint8_t)(dr < dl ? dr : dl);
    }
}

/* VEC bricks of a row per thread; the last pass of the delta trackers writes
   -dist into the empty bricks of the majorant grid, the march's its bytes */
template <int VEC>
__global__ void __launch_bounds__(256) k_skip_yz(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, float* __restrict__ majorant_out,
                                                 int n, long long step, long long total)
{
    typedef typename std::conditional<VEC == 4, uint32_t, uint8_t>::type Word;
    const long long stride = (long long)gridDim.x * blockDim.x * VEC;
    for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * VEC; i < total; i += stride) {
        const int c = (int)((i / step) % n);
        uint32_t best = *(const Word*)(in + i);
        /* largest of the VEC distances bounds the offsets to look at */
        for (int o = 1;; o++) {
            uint32_t most = best & 0xffu;
            if (VEC == 4) most = max(max(most, (best >> 8) & 0xffu), max((best >> 16) & 0xffu, best >> 24));
            if ((uint32_t)o >= most) break;
            const uint32_t oo = (uint32_t)o * (VEC == 4 ? 0x01010101u : 1u);
            if (c - o >= 0) best = __vminu4(best, __vmaxu4((uint32_t) * (const Word*)(in + i - o * step), oo));
            if (c + o < n) best = __vminu4(best, __vmaxu4((uint32_t) * (const Word*)(in + i + o * step), oo));
        }
        if (!majorant_out) {
            *(Word*)(out + i) = (Word)best;
        } else {
#pragma unroll
            for (int k = 0; k < VEC; k++)
                if (!(majorant_out[i + k] > 0.0f)) majorant_out[i + k] = -(float)((best >> (8 * k)) & 0xffu);
        }
    }
}

static cudaError_t launch_skip(int march, float* majorant, uint8_t* occ, const int nb[3], uint8_t* tmp, cudaStream_t s)
{
    const long long total = (long long)nb[0] * nb[1] * nb[2], rows = (long long)nb[1] * nb[2];
    const long long words = rows * ((nb[0] + 31) / 32);
    auto grid = [](long long threads) { const long long b = (threads + 255) / 256; return (unsigned)(b < 65536 ? b : 65536); };
    uint8_t *px = tmp, *py = tmp + total;
    /* whole words: rows of a multiple of four bricks, and aligned maps */
    const bool vec = (nb[0] & 3) == 0 && (((uintptr_t)px | (uintptr_t)py | (uintptr_t)occ) & 3u) == 0;
    if (march) k_skip_x<1><<<grid(words * 32), 256, 0, s>>>(nullptr, occ, px, nb[0], rows);
    else k_skip_x<0><<<grid(words * 32), 256, 0, s>>>(majorant, nullptr, px, nb[0], rows);
    float* mj = march ? nullptr : majorant;
    if (vec) {
        k_skip_yz<4><<<grid(total / 4), 256, 0, s>>>(px, py, nullptr, nb[1], nb[0], total);
        k_skip_yz<4><<<grid(total / 4), 256, 0, s>>>(py, occ, mj, nb[2], rows / nb[2] * nb[0], total);
    } else {
        k_skip_yz<1><<<grid(total), 256, 0, s>>>(px, py, nullptr, nb[1], nb[0], total);
        k_skip_yz<1><<<grid(total), 256, 0, s>>>(py, occ, mj, nb[2], rows / nb[2] * nb[0], total);
    }
    return cudaGetLastError();
}

cudaError_t er_launch_empty_skip(float* majorant, const int nb[3], uint8_t* tmp, cudaStream_t s)
{
    return launch_skip(0, majorant, nullptr, nb, tmp, s);
}

/* The empty-space map of the fixed-step march: dist bytes of bricks of
   2^shift voxels a side (launch_skip).  A brick is empty when sigma is
   exactly zero (of either sign) at every intensity a lookup in it can have,
   lo - 3 .. hi (each of the blend's three truncated lerps can round to one
   below its smaller end): a step there adds nothing to the march's sum, so
   the march may leave the lookup out.  A negative or NaN sigma counts as not
   empty. */
/* running count of the nonzero entries (n <= 65536): a warp's ballots of 32
   entries each, then a scan over those words, then the counts; loads and stores
   coalesced and independent (64 neighbouring entries to a thread took 95 of the
   235 us of a march tracer's edit and frame at n = 65536) */
__global__ void __launch_bounds__(1024) k_nonzero_prefix(const float* __restrict__ sigma, uint32_t* __restrict__ count, int n)
{
    __shared__ uint32_t word[2048], before[2048], part[32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
#pragma unroll 8
    for (int i0 = 0; i0 < n; i0 += 1024) {
        const int i = i0 + t;
        const uint32_t m = __ballot_sync(0xffffffffu, i < n && sigma[i] != 0.0f);
        if (lane == 0) word[(i0 >> 5) + w] = m;
    }
    const int words = (n + 1023) / 1024 * 32;
    __syncthreads();
    const uint32_t c0 = 2 * t < words ? __popc(word[2 * t]) : 0u, c1 = 2 * t + 1 < words ? __popc(word[2 * t + 1]) : 0u;
    uint32_t incl = c0 + c1;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) part[w] = incl;
    __syncthreads();
    uint32_t run = incl - c0 - c1;
    for (int k = 0; k < w; k++) run += part[k];
    before[2 * t] = run;
    before[2 * t + 1] = run + c0;
    __syncthreads();
#pragma unroll 8
    for (int i = t; i < n; i += 1024) count[i] = before[i >> 5] + (uint32_t)__popc(word[i >> 5] & (0xffffffffu >> (31 - (i & 31))));
}

__global__ void k_occupancy(const uint32_t* __restrict__ minmax, const uint32_t* __restrict__ count, int n, uint8_t* __restrict__ occ,
                            long long total)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const uint32_t mm = minmax[i];
    int lo = (int)(mm & 0xffffu) - 3, hi = (int)(mm >> 16);
    lo = lo < 0 ? 0 : (lo > n - 1 ? n - 1 : lo);
    hi = hi > n - 1 ? n - 1 : hi;
    const uint32_t below = lo > 0 ? count[lo - 1] : 0u;
    occ[i] = count[hi] == below ? ER_SKIP_CAP : 0;
}

cudaError_t er_launch_march_map(const uint16_t* vox, const int res[3], int shift, const int nb[3], const float* sigma, int n,
                                uint32_t* count, uint32_t* minmax, uint8_t* tmp, uint8_t* occ, cudaStream_t s)
{
    const long long total = (long long)nb[0] * nb[1] * nb[2];
    const long long want = (total + 255) / 256;
    launch_minmax(vox, res, 1 << shift, nb, minmax, s);
    k_nonzero_prefix<<<1, 1024, 0, s>>>(sigma, count, n);
    k_occupancy<<<(unsigned)want, 256, 0, s>>>(minmax, count, n, occ, total);
    return launch_skip(1, nullptr, occ, nb, tmp, s);
}

/* corner quads: for voxel (x, y, z) the intensities at (x, y), (x+1, y),
   (x, y+1), (x+1, y+1) of slice z, packed as two uint16 pairs, so that a
   trilinear lookup reads two 8-byte words instead of eight 2-byte ones;
   stored x fastest or in 8^3 bricks (quad_index, er_device.cuh).  This
   kernel writes the quads of the voxels in the box [lo, lo + n) (a region
   edit changes the quads of the voxels one below it in x and y as well) and
   finds the largest voxel value in the box. */
/* A warp takes a row of the box at a time (no division per voxel: one 64-bit
   remainder chain a voxel bounded the kernel before, 569 us at 512^3); a lane
   makes VEC neighbouring quads: with VEC 2 (x fastest, even rows) it reads
   three voxels of two rows as two words and stores both quads as 16 bytes. */
template <int VEC>
__global__ void __launch_bounds__(256) k_box_quads_max(const uint16_t* __restrict__ vox, int rx, int ry, int x0, int y0, int z0, int nx,
                                                       int ny, int nz, uint2* __restrict__ quad, int qb_nbx,
                                                       unsigned long long qb_slab, unsigned int* __restrict__ vmax)
{
    const long long rows = (long long)ny * nz;
    const long long stride = (long long)gridDim.x * (blockDim.x >> 5);
    const int lane = threadIdx.x & 31;
    unsigned int m = 0;
    for (long long r = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += stride) {
        const int y = y0 + (int)(r % ny), z = z0 + (int)(r / ny);
        const int y1 = y + 1 < ry ? y + 1 : ry - 1;
        const uint16_t* a = vox + ((size_t)z * ry + y) * (size_t)rx;
        const uint16_t* b = vox + ((size_t)z * ry + y1) * (size_t)rx;
        if (VEC == 2) {
#pragma unroll 2
            for (int x = x0 + 2 * lane; x < x0 + nx; x += 64) {
                const int x2 = x + 2 < rx ? x + 2 : rx - 1;
                const uint32_t wa = *(const uint32_t*)(a + x), wb = *(const uint32_t*)(b + x);
                const uint32_t na = a[x2], nb = b[x2];
                const uint32_t a1 = wa >> 16, b1 = wb >> 16;
                *(uint4*)(quad + ((size_t)z * ry + y) * (size_t)rx + x) = make_uint4(wa, wb, a1 | (na << 16), b1 | (nb << 16));
                m = max(m, max(wa & 0xffffu, a1));
            }
        } else {
            for (int x = x0 + lane; x < x0 + nx; x += 32) {
                const int x1 = x + 1 < rx ? x + 1 : rx - 1;
                const uint32_t v00 = a[x], v10 = a[x1], v01 = b[x], v11 = b[x1];
                if (quad) quad[erd::quad_index(x, y, z, rx, ry, qb_nbx, qb_slab)] = make_uint2(v00 | (v10 << 16), v01 | (v11 << 16));
                m = max(m, v00);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0 && m) atomicMax(vmax, m);
}

cudaError_t er_launch_box_quads_max(const uint16_t* vox, const int res[3], const int lo[3], const int n[3], uint2* quad, int qb_nbx,
                                    unsigned long long qb_slab, unsigned int* vmax, cudaStream_t s)
{
    const long long rows = (long long)n[1] * n[2];
    if (rows == 0 || n[0] == 0) return cudaSuccess;
    const long long want = (rows + 7) / 8;
    const unsigned blocks = (unsigned)(want < 152 * 16 ? want : 152 * 16);
    /* pairs: the rows' first voxels and quads aligned, the box's pairs whole */
    const bool pairs = quad && qb_nbx == 0 && (res[0] & 1) == 0 && (lo[0] & 1) == 0 && (n[0] & 1) == 0 && ((uintptr_t)vox & 3u) == 0 &&
                       ((uintptr_t)quad & 15u) == 0;
    if (pairs)
        k_box_quads_max<2><<<blocks, 256, 0, s>>>(vox, res[0], res[1], lo[0], lo[1], lo[2], n[0], n[1], n[2], quad, qb_nbx, qb_slab, vmax);
    else
        k_box_quads_max<1><<<blocks, 256, 0, s>>>(vox, res[0], res[1], lo[0], lo[1], lo[2], n[0], n[1], n[2], quad, qb_nbx, qb_slab, vmax);
    return cudaGetLastError();
}

/* ====================================================================== */
/* Allocation-free majorant build                                           */
/* ====================================================================== */
/*
 * Some callers cannot call cudaMalloc or cudaFree at the point where they
 * need a majorant grid: an application that rebuilds the grid inside its
 * frame loop (every edit of the opacity transfer function changes it), where
 * cudaMalloc/cudaFree would synchronise the whole device and stall the
 * frame; and hosts whose device memory is owned by their own pool allocator
 * and forbid allocations behind its back.  er_build_majorant_device_noalloc
 * serves them: the caller passes the inputs (voxels, sigma table) and the
 * output grid, and the two scratch buffers of the build (per-brick voxel
 * min/max, range-maximum table over the sigma table) live in the file-scope
 * device arrays below instead of library allocations.
 *
 * Limits: at most ER_NOALLOC_MAX_BRICKS bricks (2^20: a 1024x1024x512 volume
 * with 8^3 bricks) and ER_NOALLOC_MAX_SIGMA sigma entries (the full uint16
 * range).  Together the arrays take 8.25 MiB of device memory on every GPU
 * that loads the library, held until the process exits.
 *
 * Sharing: every call uses the same arrays, which keep the previous call's
 * contents.  Nothing in them has to start at zero: each call writes every
 * min/max entry and every range-table entry it reads before reading it.
 * Calls that overlap on the GPU (for example on two streams at once) race on
 * the arrays and must be serialised by the caller.
 *
 * Set-up: the first call on a device, with that device current, resolves the
 * arrays' device addresses with cudaGetSymbolAddress (the host-side names of
 * __device__ arrays are not device addresses).  Make that first call before
 * any stream capture.  The addresses belong to the device's current context;
 * when that context is replaced (cudaDeviceReset, then new work), the next
 * call sees a new context ID and resolves them again.
 */
#include <cuda.h>
#include <mutex>

#define ER_NOALLOC_MAX_BRICKS (1u << 20)
#define ER_NOALLOC_MAX_SIGMA 65536
#define ER_NOALLOC_MAX_LEVELS 17

static __device__ __align__(256) uint32_t g_noalloc_minmax[ER_NOALLOC_MAX_BRICKS];
static __device__ __align__(256) float g_noalloc_rmq[ER_NOALLOC_MAX_LEVELS * ER_NOALLOC_MAX_SIGMA];

namespace {

struct NoallocScratch {
    uint32_t* minmax;
    float* rmq;
    unsigned long long ctx_id;     /* context the addresses belong to (0: unknown) */
    bool ready;
};

#define ER_NOALLOC_MAX_DEVICES 64
std::mutex g_noalloc_mutex;
NoallocScratch g_noalloc[ER_NOALLOC_MAX_DEVICES];

/* The driver's cuCtxGetCurrent and cuCtxGetId, looked up through the runtime
   (the library does not link libcuda).  A context's ID is unique for the
   life of the process, so a device whose context was destroyed and made
   again (cudaDeviceReset) shows a new ID, and the arrays' addresses, which
   belong to the module loaded into the old context, are resolved again. */
typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long*);
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;
bool g_ctx_fns_looked_up = false;

/* ID of the current context, 0 when it cannot be read */
unsigned long long current_context_id()
{
    if (!g_ctx_fns_looked_up) {
        g_ctx_fns_looked_up = true;
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_ctx_get_current = (CtxGetCurrentFn)f;
        f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_ctx_get_id = (CtxGetIdFn)f;
        cudaGetLastError();
    }
    if (!g_ctx_get_current || !g_ctx_get_id) return 0;
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (g_ctx_get_current(&c) != CUDA_SUCCESS || !c) return 0;
    if (g_ctx_get_id(c, &id) != CUDA_SUCCESS) return 0;
    return id;
}

/* device addresses of the scratch arrays in the current device's context:
   resolved once per context (the first call on a device, and again after
   its context was replaced); every call when the context ID cannot be read */
cudaError_t noalloc_scratch(int device, NoallocScratch* out)
{
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    NoallocScratch& s = g_noalloc[device];
    const unsigned long long id = current_context_id();
    if (!s.ready || id == 0 || id != s.ctx_id) {
        void* a = nullptr;
        void* b = nullptr;
        s.ready = false;
        cudaError_t e = cudaGetSymbolAddress(&a, g_noalloc_minmax);
        if (e != cudaSuccess) return e;
        e = cudaGetSymbolAddress(&b, g_noalloc_rmq);
        if (e != cudaSuccess) return e;
        s.minmax = (uint32_t*)a;
        s.rmq = (float*)b;
        /* the first runtime call above makes the primary context current
           when nothing had: read the ID again */
        s.ctx_id = id ? id : current_context_id();
        s.ready = true;
    }
    *out = s;
    return cudaSuccess;
}

er_status noalloc_fail(er_status st, const char* msg)
{
    er_internal_set_error(msg);
    return st;
}

}  // namespace

extern "C" ER_API er_status er_build_majorant_device_noalloc(const uint16_t* d_voxels, const int32_t resolution[3], int32_t brick,
                                                             const float* d_sigma, int32_t sigma_count, float density_scale,
                                                             float* d_majorant, void* stream)
{
    char msg[256];
    if (!d_voxels || !resolution || !d_sigma || !d_majorant) return noalloc_fail(ER_ERR_INVALID_ARGUMENT, "NULL argument");
    if (brick < 1 || brick > 64) {
        snprintf(msg, sizeof(msg), "brick %d out of range [1, 64]", brick);
        return noalloc_fail(ER_ERR_INVALID_ARGUMENT, msg);
    }
    if (sigma_count < 1 || sigma_count > ER_NOALLOC_MAX_SIGMA) {
        snprintf(msg, sizeof(msg), "sigma_count %d out of range [1, %d]", sigma_count, ER_NOALLOC_MAX_SIGMA);
        return noalloc_fail(ER_ERR_INVALID_ARGUMENT, msg);
    }
    int res[3], nb[3];
    for (int i = 0; i < 3; i++) {
        if (resolution[i] <= 0) return noalloc_fail(ER_ERR_INVALID_ARGUMENT, "resolution must be positive");
        res[i] = resolution[i];
        nb[i] = (res[i] + brick - 1) / brick;
    }
    const unsigned long long total = (unsigned long long)nb[0] * nb[1] * nb[2];
    if (total > ER_NOALLOC_MAX_BRICKS) {
        snprintf(msg, sizeof(msg),
                 "%llu bricks exceed the allocation-free limit of %u (use a larger brick or er_build_majorant_device)", total,
                 ER_NOALLOC_MAX_BRICKS);
        return noalloc_fail(ER_ERR_INVALID_ARGUMENT, msg);
    }
    int levels = 1;
    while ((1 << levels) <= sigma_count) levels++;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess && (device < 0 || device >= ER_NOALLOC_MAX_DEVICES)) return noalloc_fail(ER_ERR_INVALID_ARGUMENT, "device index out of range");
    NoallocScratch s;
    if (e == cudaSuccess) e = noalloc_scratch(device, &s);
    if (e == cudaSuccess)
        e = er_launch_majorant(d_voxels, res, brick, nb, d_sigma, sigma_count, s.rmq, levels, s.minmax, density_scale, d_majorant,
                               (cudaStream_t)stream);
    if (e != cudaSuccess) {
        snprintf(msg, sizeof(msg), "er_build_majorant_device_noalloc: %s", cudaGetErrorString(e));
        return noalloc_fail(ER_ERR_CUDA, msg);
    }
    return ER_OK;
}
