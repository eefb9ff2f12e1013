/*
 * er_post.cu - post-processing kernels (compiled with --fmad=false).
 *
 *   k_post_frame  : the three reference kernels that follow the transport
 *                   kernel in RenderEstimate (Source/core.cu:130-135) fused
 *                   into one pass: 3x3 Gaussian of the frame
 *                   (Source/filterframeestimate.cuh:33-64), running estimate
 *                   R += (F - R) / max(N, 1) (Source/estimate.cuh:27-32) and
 *                   tone map to RGBA8 (Source/tonemap.cuh:30-59).  One read of
 *                   the 3x3 neighbourhood (cached), one read and one write of
 *                   the running estimate, one 4-byte write.
 *   k_post_mean   : the same for the spp-batched path: sample mean of a sum
 *                   buffer, Gaussian of the mean, tone map.
 *   k_tonemap     : tone map of a scaled XYZA buffer.
 *   k_bilateral_h/v : separable bilateral filter on RGBA8, the design of
 *                   Source/filterrunningestimate.cuh:35-200 (window end
 *                   exclusive, alpha 255, luminance-difference range weight).
 *   k_gradient_magnitude : per-voxel |grad I| at voxel centres
 *                   (Source/gradientmagnitude.cuh:28-44 design,
 *                   Source/volumes.h:93-114 arithmetic) with a max reduction.
 */
#include <string.h>

#include "er_kernels.h"
#include "er_path.cuh"

using namespace erd;

ER_D uchar4 tonemap_px(float4 R, float exposure)
{
    float rgb[3];
    rgb[0] = 3.240479f * R.x - 1.537150f * R.y - 0.498535f * R.z;
    rgb[1] = -0.969256f * R.x + 1.875991f * R.y + 0.041556f * R.z;
    rgb[2] = 0.055648f * R.x - 0.204043f * R.y + 1.057311f * R.z;
    unsigned char o[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        float c = 1.0f - er_expf(-(rgb[i] / exposure));
        c = smax(0.0f, smin(c, 1.0f));
        o[i] = (unsigned char)(255.0f * c);
    }
    return make_uchar4(o[0], o[1], o[2], (unsigned char)(R.w * 255.0f));
}

/* Gauss2D(1, dx, dy) - Source/filterframeestimate.cuh:28-31 - of a 3x3
   window takes three values, by dx^2 + dy^2; made once on the host (er_expf
   has the same bits there) instead of nine exponentials a pixel */
struct GaussW {
    float w[3];
};

static GaussW gauss_weights()
{
    GaussW g;
    for (int d = 0; d < 3; d++) g.w[d] = er_expf(-((float)d / (2 * 1.0f * 1.0f)));
    return g;
}

template <bool FROM_SUM>
ER_D float4 filtered_pixel(const float4* __restrict__ src, float inv_n_div, int x, int y, int W, int H, int filter, const GaussW& G)
{
    const size_t c = (size_t)y * W + x;
    if (!filter) {
        float4 v = src[c];
        if (FROM_SUM) v = make_float4(v.x / inv_n_div, v.y / inv_n_div, v.z / inv_n_div, v.w / inv_n_div);
        return v;
    }
    const int x0 = (x - 1) > 0 ? (x - 1) : 0;
    const int x1 = (x + 1) < (W - 1) ? (x + 1) : (W - 1);
    const int y0 = (y - 1) > 0 ? (y - 1) : 0;
    const int y1 = (y + 1) < (H - 1) ? (y + 1) : (H - 1);
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f, tot = 0.0f;
#pragma unroll
    for (int dy = -1; dy <= 1; dy++) {
#pragma unroll
        for (int dx = -1; dx <= 1; dx++) {
            const int xx = x + dx, yy = y + dy;
            if (xx < x0 || xx > x1 || yy < y0 || yy > y1) continue;
            const float w = G.w[dx * dx + dy * dy];
            float4 f = src[(size_t)yy * W + xx];
            if (FROM_SUM) f = make_float4(f.x / inv_n_div, f.y / inv_n_div, f.z / inv_n_div, f.w / inv_n_div);
            s0 += f.x * w; s1 += f.y * w; s2 += f.z * w; s3 += f.w * w;
            tot += w;
        }
    }
    float4 ctr = src[c];
    if (FROM_SUM) ctr.w = ctr.w / inv_n_div;
    s3 = ctr.w;
    if (tot > 0.0f) return make_float4(s0 / tot, s1 / tot, s2 / tot, s3 / tot);
    return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

__global__ void k_post_frame(const float4* __restrict__ frame, float4* __restrict__ running, uchar4* __restrict__ rgba, int W,
                             int H, int no_iterations, float exposure, int filter, const GaussW G)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const size_t c = (size_t)y * W + x;
    const float4 F = filtered_pixel<false>(frame, 1.0f, x, y, W, H, filter, G);
    const float div = smax((float)no_iterations, 1.0f);
    const float4 A = running[c];
    const float4 R = make_float4(A.x + (F.x - A.x) / div, A.y + (F.y - A.y) / div, A.z + (F.z - A.z) / div, A.w + (F.w - A.w) / div);
    running[c] = R;
    rgba[c] = tonemap_px(R, exposure);
}

__global__ void k_post_mean(const float4* __restrict__ sum, float n, float4* __restrict__ running, uchar4* __restrict__ rgba, int W,
                            int H, float exposure, int filter, const GaussW G)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const size_t c = (size_t)y * W + x;
    const float4 R = filtered_pixel<true>(sum, n, x, y, W, H, filter, G);
    running[c] = R;
    rgba[c] = tonemap_px(R, exposure);
}

/* k_post_mean for every view of a batch (blockIdx.z = view); an accumulating
   view's sum holds samples [0, first + spp) of its stream */
__global__ void k_post_batch(const WfView* __restrict__ views, const GaussW G)
{
    const WfView& V = views[blockIdx.z];
    if (!V.display) return;
    const int W = V.P.film[0], H = V.P.film[1];
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const float n = V.accumulate ? (float)(V.first + (uint32_t)V.spp) : (float)V.spp;
    const size_t c = (size_t)y * W + x;
    const float4 R = filtered_pixel<true>(V.sum, n, x, y, W, H, V.filter, G);
    V.running[c] = R;
    V.rgba[c] = tonemap_px(R, V.exposure);
}

__global__ void k_tonemap(const float4* __restrict__ xyza, float scale, uchar4* __restrict__ rgba, int n, float exposure)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 v = xyza[i];
    if (scale != 1.0f) v = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
    rgba[i] = tonemap_px(v, exposure);
}

/* luminance with the weights of the LUMINANCE macro (Source/color.h:37-51) */
ER_D float lum255(uchar4 c)
{
    float L = 0.0f;
    L += 0.212671f * (float)c.x;
    L += 0.715160f * (float)c.y;
    L += 0.072169f * (float)c.z;
    return L;
}

/* The window's pixels and their luminances are made once per block in shared
   memory (a 4K film at radius 2: 161 us a pass before, when every tap read
   its range weight from the constant bank at a lane's own index and computed
   its luminance again).  The tile is BIL_N pixels along the pass's axis by
   BIL_M across; the range weights sit in shared memory too.  Films of under
   600 tiles of 64 take 16 (a pixel to a thread), as four pixels one after the
   other on a part of the chip are the longer way.  Both passes at radius 2 and
   12, us, a tap's own reads and luminance / 64 / 16: 200 x 150 5.6, 16.2 / 9.6,
   22.5 / 5.3, 8.7; 641 x 479 16.6, 94.7 / 13.7, 31.1 / 12.3, 22.4; 1024^2 46.6,
   298 / 24.7, 60 / 28.1, 55.8; 3840 x 2160 341, 2312 / 134, 365 / -. */
#define BIL_M 16

template <bool HORIZONTAL, int BIL_N>
__global__ void __launch_bounds__(256) k_bilateral(const uchar4* __restrict__ in, uchar4* __restrict__ out, int W, int H, BilateralTables T)
{
    extern __shared__ uint32_t tile[];          /* (BIL_N + 2 r) * BIL_M pixels, then as many luminances */
    __shared__ float range[256];
    const int r = T.radius;
    const int span = BIL_N + 2 * r;
    float* lum = (float*)(tile + span * BIL_M);
    /* the grid's x is the film's, of any width; its y the film's rows */
    const int n0 = (HORIZONTAL ? blockIdx.x : blockIdx.y) * BIL_N, m0 = (HORIZONTAL ? blockIdx.y : blockIdx.x) * BIL_M;
    const int N = HORIZONTAL ? W : H, M = HORIZONTAL ? H : W;
    range[threadIdx.x] = T.range[threadIdx.x];
    /* neighbouring threads read neighbouring pixels of the film's rows */
    for (int i = threadIdx.x; i < span * BIL_M; i += 256) {
        const int n = HORIZONTAL ? i % span : i / BIL_M, m = HORIZONTAL ? i / span : i % BIL_M;
        int a = n0 - r + n, b = m0 + m;
        a = a < 0 ? 0 : (a > N - 1 ? N - 1 : a);
        b = b > M - 1 ? M - 1 : b;
        const uchar4 c = HORIZONTAL ? in[(size_t)b * W + a] : in[(size_t)a * W + b];
        tile[i] = (uint32_t)c.x | ((uint32_t)c.y << 8) | ((uint32_t)c.z << 16);
        lum[i] = lum255(c);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < BIL_N * BIL_M; i += 256) {
        const int n = HORIZONTAL ? i % BIL_N : i / BIL_M, m = HORIZONTAL ? i / BIL_N : i % BIL_M;
        const int p = n0 + n, q = m0 + m;
        if (p >= N || q >= M) continue;
        const int k0 = (p - r) > 0 ? (p - r) : 0;
        const int k1 = (p + r) < (N - 1) ? (p + r) : (N - 1);
        const int step = HORIZONTAL ? 1 : BIL_M;
        const int row = HORIZONTAL ? m * span : m;
        const float lc = lum[row + (n + r) * step];
        float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, tot = 0.0f;
        for (int k = k0; k < k1; k++) {     /* window end exclusive (Source/filterrunningestimate.cuh:88,157) */
            const int t = row + (k - n0 + r) * step;
            const uint32_t c = tile[t];
            int d = (int)fabsf(lum[t] - lc);
            d = d > 255 ? 255 : d;
            const float w = T.spatial[r + k - p] * range[d];
            tot += w;
            s0 += (float)(c & 0xffu) * w; s1 += (float)((c >> 8) & 0xffu) * w; s2 += (float)(c >> 16) * w;
        }
        uchar4 o;
        if (tot > 0.0f) {
            o.x = (unsigned char)eclamp(s0 / tot, 0.0f, 255.0f);
            o.y = (unsigned char)eclamp(s1 / tot, 0.0f, 255.0f);
            o.z = (unsigned char)eclamp(s2 / tot, 0.0f, 255.0f);
        } else {
            o.x = 0; o.y = 0; o.z = 0;
        }
        o.w = 255;
        out[HORIZONTAL ? (size_t)q * W + p : (size_t)p * W + q] = o;
    }
}

ER_D float voxel_gradient_magnitude(const Params& P, int X, int Y, int Z)
{
    const float sx = 2.0f * P.half_size[0], sy = 2.0f * P.half_size[1], sz = 2.0f * P.half_size[2];
    const v3 p = V3(P.minp[0] + sx * (((float)X + 0.5f) * (1.0f / (float)P.res[0])),
                    P.minp[1] + sy * (((float)Y + 0.5f) * (1.0f / (float)P.res[1])),
                    P.minp[2] + sz * (((float)Z + 0.5f) * (1.0f / (float)P.res[2])));
    return gradient_magnitude(P, p);
}

/* out of line: the pass that looks few voxels up keeps its registers for the walk */
static __device__ __noinline__ float voxel_gradient_magnitude_c(const Params& P, int X, int Y, int Z) { return voxel_gradient_magnitude(P, X, Y, Z); }

/* per-voxel gradient magnitude at voxel centres + max; the magnitude volume
   (optional) saturates at 65535 */
__global__ void k_gradient_magnitude(const Params P, uint16_t* __restrict__ gm, unsigned int* __restrict__ max_bits)
{
    const int X = blockIdx.x * blockDim.x + threadIdx.x;
    const int Y = blockIdx.y * blockDim.y + threadIdx.y;
    const int Z = blockIdx.z * blockDim.z + threadIdx.z;
    float g = 0.0f;
    if (X < P.res[0] && Y < P.res[1] && Z < P.res[2]) {
        g = voxel_gradient_magnitude(P, X, Y, Z);
        if (gm) {
            const size_t idx = (size_t)Z * P.res[0] * P.res[1] + (size_t)Y * P.res[0] + X;
            gm[idx] = (uint16_t)(g < 65535.0f ? g : 65535.0f);
        }
    }
    /* block max through warp shuffles, one atomic per warp; non-negative
       floats order like their bit patterns */
    unsigned int b = __float_as_uint(g);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned int v = __shfl_xor_sync(0xffffffffu, b, o);
        b = v > b ? v : b;
    }
    if ((threadIdx.x + threadIdx.y * blockDim.x + threadIdx.z * blockDim.x * blockDim.y) % 32 == 0) atomicMax(max_bits, b);
}

/* The largest gradient magnitude alone, for the shader switch, of a volume
   with one spacing on all axes.  A voxel's six lookups lie (but for rounding)
   at its neighbours' centres, where the blend is the mean of a cell's eight
   voxels: integer sums give each magnitude to within a known error, and only
   the voxels that may hold the maximum make their six lookups: a pass for the
   largest lower bound, then the exact magnitudes of the voxels whose upper
   bound reaches it.  tol: how far a lookup may be from its cell's mean (three
   truncations, the weights' rounding).

   That pays where few voxels reach the bound.  Where the largest lower bound
   is not well above the error (flat and smooth volumes: gm_bounds_tell) most
   would, and where many do all the same (a volume of one slope) the exact pass
   stops at a 64th of them: the volume is left to k_gradient_magnitude.  In
   large grids an eighth of the blocks, spread over the volume, bounds first,
   and the rest only if that tells; a volume whose values are all within the
   error (a few labels) is not asked.  With and without the two passes, ms at
   512^3: shells 1.5 and 4.3, one slope 5.2 and 4.3 (6.2 before it stopped),
   smooth 4.43 and 4.32 (4.89 with all blocks first), eight labels 4.3 and 4.3
   (4.9); at 300^3 shells 0.30 and 0.93, smooth 1.07 and 0.92.

   A block walks GM_Z planes of a GM_X x GM_Y tile of cells (a ring of halo
   around the voxels): a thread sums its cell's four voxels of a plane, adds
   the plane before, and shares three planes of cell sums.  Every voxel's six
   lookups take 1213 us at 384x384x256. */
#define GM_X 32
#define GM_Y 16
#define GM_Z 32

/* whether the bounds rule voxels out: the largest lower bound is over three
   times what tol alone adds to an upper one (at eight times, the 384x384x256
   blobs went the long way) */
__host__ __device__ inline bool gm_bounds_tell(float low, float tol, float h) { return low > 3.0f * 2.0f * 1.7320508f * tol * h; }

/* Four blocks an SM (32 registers) for the bounds, and for the exact pass in a
   grid of many waves (GM_EXACT_WIDE), its lookups out of line: all passes at
   512^3 1.46 ms, the exact one at two blocks 1.84.  In a smaller grid, where a
   block's own time counts, inline at two (128^3: 75 us, out of line 87). */
enum { GM_FIRST = 0, GM_REST = 1, GM_EXACT = 2, GM_EXACT_WIDE = 3 };

/* bits: the largest magnitude, voxels looked up, the largest lower bound of the
   first pass and of the rest (two words: a pass decides on words that it does
   not write, so that a block's threads all decide the same) */
template <int PASS>
__global__ void __launch_bounds__(GM_X * GM_Y, PASS == GM_EXACT ? 2 : 4) k_gm_cells(const Params P, float tol, unsigned int share, unsigned int most,
                                                              unsigned int* bits)
{
    constexpr bool EXACT = PASS >= GM_EXACT;
    __shared__ int cells[3][GM_Y][GM_X];
    __shared__ int stop;
    if (!EXACT && ((blockIdx.x + blockIdx.y + blockIdx.z) % share == 0) != (PASS == GM_FIRST)) return;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int X = (int)blockIdx.x * (GM_X - 2) - 1 + tx, Y = (int)blockIdx.y * (GM_Y - 2) - 1 + ty;
    const int z0 = (int)blockIdx.z * GM_Z, z1 = min(z0 + GM_Z, P.res[2]);
    const size_t rx = (size_t)P.res[0], slice = rx * (size_t)P.res[1];
    const size_t xa = (size_t)iclamp(X, 0, P.res[0] - 1), xb = (size_t)iclamp(X + 1, 0, P.res[0] - 1);
    const size_t ya = (size_t)iclamp(Y, 0, P.res[1] - 1) * rx, yb = (size_t)iclamp(Y + 1, 0, P.res[1] - 1) * rx;
    auto plane = [&](int z) -> int {
        const uint16_t* v = P.vox + (size_t)iclamp(z, 0, P.res[2] - 1) * slice;
        return (int)__ldg(v + ya + xa) + (int)__ldg(v + ya + xb) + (int)__ldg(v + yb + xa) + (int)__ldg(v + yb + xb);
    };
    const bool inner = tx > 0 && tx < GM_X - 1 && ty > 0 && ty < GM_Y - 1 && X < P.res[0] && Y < P.res[1];
    const float h = 0.5f / P.spacing[0];
    const float low = PASS == GM_FIRST ? 0.0f : __uint_as_float(EXACT ? max(bits[2], bits[3]) : bits[2]);
    if (PASS != GM_FIRST && !gm_bounds_tell(low, tol, h)) return;
    unsigned int best = 0;
    /* voxels looked up so far: asked about before a block's first and added
       every eighth plane (in every plane it cost a tenth of the pass) */
    const bool asks = EXACT && tx == 0 && ty == 0;
    unsigned int seen = 0, looks = 0;
    if (asks) {
        stop = 0;
        seen = *(volatile unsigned int*)(bits + 1);
    }
    int prev = plane(z0 - 1);
    /* cell z is in cells[(z + 3) % 3]; voxel z needs cells z - 1, z and z + 1 */
    for (int z = z0 - 1; z <= z1; z++) {
        const int next = plane(z + 1);
        cells[(z + 3) % 3][ty][tx] = prev + next;
        prev = next;
        if (asks && (z & 7) == 0 && seen > most) stop = 1;
        __syncthreads();
        if (EXACT && (z & 7) == 0 && stop) return;
        const int Z = z - 1;
        bool look = false;
        if (Z >= z0 && inner) {
            const int c = (Z + 3) % 3;
            const float dx = fabsf((float)(cells[c][ty][tx - 1] - cells[c][ty][tx + 1])) * 0.125f;
            const float dy = fabsf((float)(cells[c][ty - 1][tx] - cells[c][ty + 1][tx])) * 0.125f;
            const float dz = fabsf((float)(cells[(Z + 2) % 3][ty][tx] - cells[(Z + 4) % 3][ty][tx])) * 0.125f;
            if (EXACT) {
                const float a = (dx + 2.0f * tol) * h, b = (dy + 2.0f * tol) * h, e = (dz + 2.0f * tol) * h;
                look = sqrtf(a * a + b * b + e * e) * 1.00001f >= low;
            } else {
                const float a = fmaxf(dx - 2.0f * tol, 0.0f) * h, b = fmaxf(dy - 2.0f * tol, 0.0f) * h, e = fmaxf(dz - 2.0f * tol, 0.0f) * h;
                best = max(best, __float_as_uint(sqrtf(a * a + b * b + e * e) * 0.99999f));
            }
        }
        if (look) {
            best = max(best, __float_as_uint(PASS == GM_EXACT ? voxel_gradient_magnitude(P, X, Y, Z) : voxel_gradient_magnitude_c(P, X, Y, Z)));
            looks++;
        }
        if (EXACT && ((z & 7) == 4 || z == z1)) {
            const unsigned int n = __reduce_add_sync(0xffffffffu, looks);
            if (tx == 0 && n) atomicAdd(bits + 1, n);
            if (asks) seen = *(volatile unsigned int*)(bits + 1);
            looks = 0;
        }
        /* the next plane overwrites cell z - 2, which voxel z - 1 has read */
        __syncthreads();
    }
    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (tx == 0 && best) atomicMax(bits + (EXACT ? 0 : 2 + PASS), best);
}

__global__ void k_math_eval(int fn, int n, const float* __restrict__ x, const float* __restrict__ y, float* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float a = x[i];
    const float b = y ? y[i] : 0.0f;
    float r = 0.0f;
    switch (fn) {
    case 0: r = er_logf(a); break;
    case 1: r = er_expf(a); break;
    case 2: r = er_sinf(a); break;
    case 3: r = er_cosf(a); break;
    case 4: r = er_tanf(a); break;
    case 5: r = er_powf(a, b); break;
    case 6: r = er_acosf(a); break;
    case 7: r = er_atan2f(a, b); break;
    default: break;
    }
    out[i] = r;
}

/* ---- launchers ---- */

cudaError_t er_launch_math_eval(int fn, int n, const float* x, const float* y, float* out, cudaStream_t s)
{
    k_math_eval<<<(n + 255) / 256, 256, 0, s>>>(fn, n, x, y, out);
    return cudaGetLastError();
}

cudaError_t er_launch_post_frame(const float4* frame, float4* running, uchar4* rgba, int W, int H, int n_iter, float exposure,
                                 int filter, cudaStream_t s)
{
    const dim3 b(16, 8), g((W + 15) / 16, (H + 7) / 8);
    k_post_frame<<<g, b, 0, s>>>(frame, running, rgba, W, H, n_iter, exposure, filter, gauss_weights());
    return cudaGetLastError();
}

cudaError_t er_launch_post_mean(const float4* sum, float n, float4* running, uchar4* rgba, int W, int H, float exposure, int filter,
                                cudaStream_t s)
{
    const dim3 b(16, 8), g((W + 15) / 16, (H + 7) / 8);
    k_post_mean<<<g, b, 0, s>>>(sum, n, running, rgba, W, H, exposure, filter, gauss_weights());
    return cudaGetLastError();
}

cudaError_t er_launch_post_batch(const WfView* d_views, int n_views, int max_w, int max_h, cudaStream_t s)
{
    const dim3 b(16, 8), g((max_w + 15) / 16, (max_h + 7) / 8, n_views);
    k_post_batch<<<g, b, 0, s>>>(d_views, gauss_weights());
    return cudaGetLastError();
}

cudaError_t er_launch_tonemap(const float4* xyza, float scale, uchar4* rgba, int n, float exposure, cudaStream_t s)
{
    k_tonemap<<<(n + 255) / 256, 256, 0, s>>>(xyza, scale, rgba, n, exposure);
    return cudaGetLastError();
}

cudaError_t er_launch_bilateral(const uchar4* in, uchar4* tmp, uchar4* out, int W, int H, const BilateralTables& T,
                                cudaStream_t s)
{
    /* radius <= 127: at most 318 * 16 * 8 B = 40.7 KB */
    const size_t rows = (size_t)((H + BIL_M - 1) / BIL_M), columns = (size_t)((W + BIL_M - 1) / BIL_M);
    const bool few = (size_t)((W + 63) / 64) * rows < 600;
    const int n = few ? 16 : 64;
    const size_t bytes = (size_t)(n + 2 * T.radius) * BIL_M * 8;
    const dim3 gh((W + n - 1) / n, (unsigned)rows), gv((unsigned)columns, (H + n - 1) / n);
    if (few) {
        k_bilateral<true, 16><<<gh, 256, bytes, s>>>(in, tmp, W, H, T);
        k_bilateral<false, 16><<<gv, 256, bytes, s>>>(tmp, out, W, H, T);
    } else {
        k_bilateral<true, 64><<<gh, 256, bytes, s>>>(in, tmp, W, H, T);
        k_bilateral<false, 64><<<gv, 256, bytes, s>>>(tmp, out, W, H, T);
    }
    return cudaGetLastError();
}

cudaError_t er_launch_gradient_magnitude(const Params& P, uint16_t* gm, unsigned int* max_bits, cudaStream_t s)
{
    const dim3 b(8, 8, 8);
    const dim3 g((P.res[0] + 7) / 8, (P.res[1] + 7) / 8, (P.res[2] + 7) / 8);
    k_gradient_magnitude<<<g, b, 0, s>>>(P, gm, max_bits);
    return cudaGetLastError();
}

static float gradient_max_tol(const Params& P, int vmax)
{
    int most = P.res[0];
    for (int i = 1; i < 3; i++) most = P.res[i] > most ? P.res[i] : most;
    /* a lookup's local coordinate is off by a few ulps of the volume's extent, 1e-6 of it at most */
    return 3.5f + 3e-6f * (float)most * (float)vmax;
}

static unsigned int gradient_max_most(const Params& P)
{
    const unsigned long long n = (unsigned long long)P.res[0] * P.res[1] * P.res[2] / 64;
    return n < 0x7fffffffull ? (unsigned int)n + 1024u : 0x7fffffffu;
}

bool er_gradient_max_applies(const Params& P, int vmax)
{
    /* the mean's argument: one spacing, weights within a tenth of a half, and grids within the launch limits */
    const int most = P.res[0] > P.res[1] ? (P.res[0] > P.res[2] ? P.res[0] : P.res[2]) : (P.res[1] > P.res[2] ? P.res[1] : P.res[2]);
    /* no lower bound is above sqrt(3) (vmax - 2 tol) h: up to 8 tol none tells */
    return P.spacing[0] == P.spacing[1] && P.spacing[1] == P.spacing[2] && P.spacing[0] > 0.0f && most <= 50000 &&
           (float)vmax > 8.0f * gradient_max_tol(P, vmax);
}

bool er_gradient_max_found(const Params& P, int vmax, const unsigned int bits[4])
{
    const unsigned int low_bits = bits[2] > bits[3] ? bits[2] : bits[3];
    float low;
    memcpy(&low, &low_bits, sizeof(low));
    return gm_bounds_tell(low, gradient_max_tol(P, vmax), 0.5f / P.spacing[0]) && bits[1] <= gradient_max_most(P);
}

cudaError_t er_launch_gradient_max(const Params& P, int vmax, unsigned int* bits, cudaStream_t s)
{
    const float tol = gradient_max_tol(P, vmax);
    const unsigned int most = gradient_max_most(P);
    const dim3 b(GM_X, GM_Y), g((P.res[0] + GM_X - 3) / (GM_X - 2), (P.res[1] + GM_Y - 3) / (GM_Y - 2), (P.res[2] + GM_Z - 1) / GM_Z);
    /* a grid of few waves takes about as long for an eighth of its blocks */
    const size_t blocks = (size_t)g.x * g.y * g.z;
    const unsigned int share = blocks < 8192 ? 1 : 8;
    k_gm_cells<GM_FIRST><<<g, b, 0, s>>>(P, tol, share, most, bits);
    if (share > 1) k_gm_cells<GM_REST><<<g, b, 0, s>>>(P, tol, share, most, bits);
    if (blocks < 2500) k_gm_cells<GM_EXACT><<<g, b, 0, s>>>(P, tol, share, most, bits);
    else k_gm_cells<GM_EXACT_WIDE><<<g, b, 0, s>>>(P, tol, share, most, bits);
    return cudaGetLastError();
}
