/*
 * One fine pixel of the joint bilateral upsampling, shared by the context
 * path's k_jbu (hpm_jbu.cu) and the allocation-free k_jbu_noalloc
 * (hpm_noalloc.cu), so that the two cannot drift apart.
 *
 * Behaviour of the reference's JBU_cu (HPM-MVS/HPM.cu:1971-2052): for a fine
 * pixel p the window is (s*s+1) x (s*s+1) taps of the coarse grid around
 * o = p * (coarse_w / fine_w) (coordinates truncated, then clamped), the
 * spatial weight is exp(-d^2 / (2 * 0.5^2)) in coarse units and the range
 * weight exp(-dI^2 / (2 * 25.5^2)) compares the guide at p with the guide at
 * p + (i, j) in FINE pixels (the mixed-space window of the reference is kept).
 * Depth is the weighted mean; the normal is the normalised weighted sum.
 *
 * The coarse depth and normal come packed as one float4 (nx, ny, nz, depth)
 * per coarse pixel, so that every tap is a single 16-byte read-only load.
 * The reference computes both gaussians in double precision (pow/exp of a
 * double); here they are FP32 expf of the same arguments.
 *
 * What bounds it is the arithmetic of the (s*s+1)^2 taps (two expf each).  A
 * tap whose coarse sample is more than sqrt(45) coarse pixels away has a
 * spatial weight exp(-90) or less, which the build's flush of subnormals makes
 * zero, and adding zero changes no sum: at scale 4 these are 152 of the 289
 * taps.  They are left out where every value in reach of the block is finite
 * (a weight of zero times an infinity is not zero); elsewhere all taps are
 * taken, and at scales below 4, whose windows hold few such taps or none, so
 * that looking for them costs more than it saves (jbu_cuts).  Away from
 * the borders, with a power of two as the scale, coordinates are exact and a
 * row's taps are a plain run of the coarse grid, without conversions and
 * clamps.  1600x1200 from 400x300: 760 us with all taps, 423 us now, the
 * same bits.
 */
#pragma once

#include <cuda_runtime.h>

namespace hpm {

constexpr int kJbuBlockX = 32, kJbuBlockY = 8;

/* A grid's y ends at 65,535, so the block rows beyond continue along z (524,280
 * rows and more of a narrow image). */
inline dim3 jbu_grid(int cols, int rows)
{
    const unsigned n = ((unsigned)rows + kJbuBlockY - 1) / kJbuBlockY;
    return dim3(((unsigned)cols + kJbuBlockX - 1) / kJbuBlockX, n < 65535u ? n : 65535u, (n + 65534u) / 65535u);
}
__device__ __forceinline__ int jbu_block_row() { return (blockIdx.z * gridDim.y + blockIdx.y) * kJbuBlockY; }

/* Squared distance in coarse pixels beyond which a spatial weight is zero:
 * exp(-90) is where subnormals are flushed (the Makefile's --use_fast_math), and
 * exp(-104) rounds to zero in any FP32.  Asked of expf itself, so that the
 * header is right under either build. */
__device__ __forceinline__ float jbu_reach2() { return expf(-90.0f) == 0.0f ? 45.0f : 52.0f; }

enum JbuTaps { kJbuAll, kJbuNear, kJbuInner };

__device__ __forceinline__ int jbu_coarse(float v, int n)
{
    const int r = __float2int_rz(v);
    return r > 0 ? (r < n ? r : n - 1) : 0;
}

/* The scales whose kernel looks for the taps out of reach (CUT).  1600x1200
 * with all taps and with those in reach, by scale: 2 85 and 91 us (no tap is
 * out of reach), 3 316 and 386, 4 760 and 423 (775 and 615 for 1601x1201, whose
 * coordinates are not exact), 5 1829 and 779.  A kernel of its own for the rest:
 * as a branch of one kernel, all taps at scale 3 took 351 us. */
inline bool jbu_cuts(int image_scale) { return image_scale >= 4; }

/* How the block's pixels take their taps (the same answer in all threads; all
 * must call). */
template <bool CUT>
__device__ __forceinline__ JbuTaps jbu_block_taps(const float *__restrict__ guide, int cols, int rows,
                                                  const float4 *__restrict__ coarse, int s_cols, int s_rows,
                                                  int image_scale)
{
    if constexpr (!CUT) return kJbuAll;
    const float scale = (float)(1.0 * s_cols / cols);
    const int nn = (image_scale * image_scale + 1) / 2;
    const int x0 = blockIdx.x * kJbuBlockX, y0 = jbu_block_row();
    const int x1 = min(x0 + kJbuBlockX, cols) - 1, y1 = min(y0 + kJbuBlockY, rows) - 1;
    const int tid = threadIdx.y * kJbuBlockX + threadIdx.x;
    bool finite = true;
    const int cx0 = jbu_coarse(x0 * scale - nn, s_cols), cx1 = jbu_coarse(x1 * scale + nn, s_cols);
    const int cy0 = jbu_coarse(y0 * scale - nn, s_rows), cy1 = jbu_coarse(y1 * scale + nn, s_rows);
    const int cw = cx1 - cx0 + 1, cn = cw * (cy1 - cy0 + 1);
    for (int i = tid; i < cn; i += kJbuBlockX * kJbuBlockY) {
        const float4 c = __ldg(coarse + (size_t)(cy0 + i / cw) * s_cols + cx0 + i % cw);
        finite = finite && isfinite(c.x) && isfinite(c.y) && isfinite(c.z) && isfinite(c.w);
    }
    const int gx0 = max(x0 - nn, 0), gy0 = max(y0 - nn, 0);
    const int gw = min(x1 + nn, cols - 1) - gx0 + 1, gn = gw * (min(y1 + nn, rows - 1) - gy0 + 1);
    for (int i = tid; i < gn; i += kJbuBlockX * kJbuBlockY)
        finite = finite && isfinite(__ldg(guide + (size_t)(gy0 + i / gw) * cols + gx0 + i % gw));
    if (__syncthreads_or(!finite)) return kJbuAll;
    const bool exact = (__float_as_uint(scale) & 0x7fffffu) == 0u && cols < (1 << 16) && rows < (1 << 16);
    const bool inside = x0 * scale >= nn && y0 * scale >= nn && x1 * scale + nn < s_cols && y1 * scale + nn < s_rows &&
                        x0 >= nn && y0 >= nn && x1 + nn < cols && y1 + nn < rows;
    return exact && inside ? kJbuInner : kJbuNear;
}

struct JbuSums {
    float nf, ctot, nx, ny, nz;
    __device__ __forceinline__ void add(float4 c, float dis, float ref_pix, float nb)
    {
        const float inv_2sd2 = 1.0f / (2.0f * 0.5f * 0.5f);
        const float inv_2sr2 = 1.0f / (2.0f * 25.5f * 25.5f);
        const float sg = expf(-dis * inv_2sd2);
        const float xp = fabsf(ref_pix - nb);
        const float rg = expf(-(xp * xp) * inv_2sr2);
        const float tg = sg * rg;
        nf += tg;
        ctot += c.w * tg;
        nx += c.x * tg;
        ny += c.y * tg;
        nz += c.z * tg;
    }
};

/* The window's taps with clamped coordinates: all, or those in reach. */
template <bool NEAR>
__device__ __forceinline__ void jbu_window(const float *__restrict__ guide, int cols, int rows,
                                           const float4 *__restrict__ coarse, int s_cols, int s_rows, int nn, int px,
                                           int py, float ox, float oy, float ref_pix, JbuSums &s)
{
    const float reach2 = jbu_reach2();
    for (int j = -nn; j <= nn; ++j) {
        const int ry = jbu_coarse(oy + (float)j, s_rows);
        const int rys = min(max(py + j, 0), rows - 1);
        const float dy = oy - (float)ry;
        if (NEAR && dy * dy > reach2) continue;
        const float *grow = guide + (size_t)rys * cols;
        for (int i = -nn; i <= nn; ++i) {
            const int rx = jbu_coarse(ox + (float)i, s_cols);
            const float dx = ox - (float)rx;
            const float dis = dx * dx + dy * dy;
            if (NEAR && dis > reach2) continue;
            const int rxs = min(max(px + i, 0), cols - 1);
            s.add(__ldg(coarse + (size_t)ry * s_cols + rx), dis, ref_pix, __ldg(grow + rxs));
        }
    }
}

/* Returns (nx, ny, nz, depth) of fine pixel (px, py). */
__device__ __forceinline__ float4 jbu_pixel(const float *__restrict__ guide, int cols, int rows,
                                            const float4 *__restrict__ coarse, int s_cols, int s_rows,
                                            int image_scale, int px, int py, JbuTaps taps)
{
    const float scale = (float)(1.0 * s_cols / cols);
    const int nn = (image_scale * image_scale + 1) / 2;
    const float oy = py * scale, ox = px * scale;
    const float ref_pix = __ldg(guide + (size_t)py * cols + px);
    JbuSums s = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (taps == kJbuInner) {
        const float reach2 = jbu_reach2();
        const int bx = __float2int_rz(ox), by = __float2int_rz(oy);
        const float fx = ox - (float)bx, fy = oy - (float)by;
        const int nj = min(nn, reach2 < 49.0f ? 7 : 8);
        for (int j = -nj; j <= nj; ++j) {
            const float dy = fy - (float)j;
            /* the row's taps within reach, and at most one more at each end */
            const int ni = min(nn, (int)sqrtf(fmaxf(reach2 - dy * dy, 0.0f)) + 1);
            const float4 *crow = coarse + (size_t)(by + j) * s_cols + bx;
            const float *grow = guide + (size_t)(py + j) * cols + px;
#pragma unroll 4
            for (int i = -ni; i <= ni; ++i) {
                const float dx = fx - (float)i;
                s.add(__ldg(crow + i), dx * dx + dy * dy, ref_pix, __ldg(grow + i));
            }
        }
    } else if (taps == kJbuNear) {
        jbu_window<true>(guide, cols, rows, coarse, s_cols, s_rows, nn, px, py, ox, oy, ref_pix, s);
    } else {
        jbu_window<false>(guide, cols, rows, coarse, s_cols, s_rows, nn, px, py, ox, oy, ref_pix, s);
    }
    float4 n = make_float4(s.nx / s.nf, s.ny / s.nf, s.nz / s.nf, 0.0f);
    const float inv = rsqrtf(n.x * n.x + n.y * n.y + n.z * n.z);
    n.x *= inv;
    n.y *= inv;
    n.z *= inv;
    n.w = s.ctot / s.nf;
    return n;
}

}  // namespace hpm
