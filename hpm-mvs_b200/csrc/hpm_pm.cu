/*
 * PatchMatch kernels of the B200-native HPM-MVS path (sm_100a).
 *
 * Behaviour follows the reference's HPM-MVS/HPM.cu kernel for kernel; the
 * per-function comments cite the lines.  What is different is how the work
 * maps to the machine:
 *
 *  - Reference-window hoisting.  The reference recomputes the 36 bilateral
 *    weights of a pixel's 11x11/stride-2 window (one exp, one sqrt, two
 *    divides each) and all reference-side sums inside every NCC call
 *    (HPM.cu:345-368), i.e. ~23 x S times per pixel per half-step.  Here they
 *    are computed once per pixel per launch and kept in shared memory, beside
 *    a tile of the reference image: each NCC tap then costs shared loads
 *    instead of an exp, a sqrt and two texture fetches.
 *  - Source views are sampled by the texture unit (float cudaArray, linear
 *    filter, clamped edges: the reference's own texture set-up), so the
 *    bilinear samples are the reference's bit for bit.  The filter rounds
 *    coordinates to 1/256 (half up) and only the far corner's weight
 *    A*B/256; a textbook bilinear gather differs by up to ~0.5 gray levels
 *    per tap.
 *  - A warp scores its pixels' windows together (ncc_quad), packed 32 at a
 *    time whatever pixel they belong to.
 *  - The per-pixel cost matrix (cost_array[8][32], 1.5 KB of local memory per
 *    thread in the reference) is handed from the site/direction kernel to the
 *    selection and the refinement through L2.
 *  - Counter-based Philox random numbers: no 48-byte curand state per pixel
 *    in HBM and no curand_init skip-ahead; draws come in the reference's
 *    order.
 *  - Half-step kernels are launched back to back on one stream with no
 *    host synchronisation (the reference synchronises after every launch).
 */
#include <cfloat>
#include <cstdlib>

#include "hpm_internal.h"

namespace hpm {

namespace {

constexpr double kPiD = 3.14159265358979323846; /* M_PI, HPM-MVS/main.h:41 */
constexpr int kBlockX = 32;
constexpr int kBlockY = 2;
constexpr int kBlock = kBlockX * kBlockY;

/* Pixels of one half-step (one checkerboard colour) per warp: ww per row
 * over 32 / ww rows, so that the 32 lanes sample a compact 2D patch of each
 * source image (the texture cache is tiled in 2D).  A block is two such
 * warps stacked vertically.  ww is 8 unless the batched form's tile tuning
 * picks 4 or 16 for a view size; wide blocks have further warps, which own no
 * pixels (launch_prop_n). */
static_assert(kBlock == 64, "two warps own a block's pixels");

/* (px, py) of this thread in a half-step of `color`, for the block's tile
 * (bx, by) */
__device__ __forceinline__ void half_step_pixel_at(int bx, int by, int ww, int color, int &px, int &py)
{
    const int lane = threadIdx.x, wv = threadIdx.y, wh = 32 / ww;
    py = by * (2 * wh) + wv * wh + lane / ww;
    px = bx * (2 * ww) + 2 * (lane % ww) + ((py + color) & 1);
}

/* Blocks per SM that the window kernels are compiled for: 14 to 16 warps, so
 * that no more than a few words of a thread spill and the blocks' shared memory
 * leaves 92 KB or more to the texture cache (1600x1200, 5 sources, at 7, 8, 9 and
 * 10 blocks: k_prop_dirs 1.70, 1.68, 1.71, 1.73 ms, k_prop_refine 0.95, 0.96,
 * 2.14, 2.13; 641x481 with 4 sources behaves alike; k_init with 10 sources at 6, 8
 * and 10 blocks: 1.05, 1.02, 1.67 ms). */
#ifndef HPM_P0_MIN_BLOCKS
#define HPM_P0_MIN_BLOCKS 8
#endif
#ifndef HPM_P1_MIN_BLOCKS
#define HPM_P1_MIN_BLOCKS 8
#endif
#ifndef HPM_P2_MIN_BLOCKS
#define HPM_P2_MIN_BLOCKS 7
#endif
/* warps per SM of their wide forms for small images (kBlocks8) */
constexpr int kWideWarps = 16;
/* k_prop_select waits for loads (cost rows, source depths): 32 warps, although
 * some registers spill (1600x1200, 10 sources, plain and geometric pass, by
 * blocks per SM: 6 0.76 and 0.83 ms, 12 0.50 and 0.83, 16 0.47 and 0.71; with
 * rows loaded a view ahead, which came later, 0.28 in a plain pass at 16). */
#ifndef HPM_P3_MIN_BLOCKS
#define HPM_P3_MIN_BLOCKS 16
#endif

/* ------------------------------------------------------------------ */
/* Philox4x32-10 (Salmon et al., SC'11), counter = (pixel, step, n/4, salt) */
/* ------------------------------------------------------------------ */
struct Rng {
    uint32_t k0, k1, pixel, step, salt, n;
    uint32_t b0, b1, b2, b3;

    __device__ void init(uint32_t klo, uint32_t khi, uint32_t px, uint32_t st, uint32_t sa)
    {
        k0 = klo;
        k1 = khi;
        pixel = px;
        step = st;
        salt = sa;
        n = 0;
    }

    __device__ void block()
    {
        uint32_t c0 = pixel, c1 = step, c2 = n >> 2, c3 = salt;
        uint32_t a0 = k0, a1 = k1;
#pragma unroll
        for (int r = 0; r < 10; ++r) {
            const uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
            const uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
            const uint32_t n0 = hi1 ^ c1 ^ a0;
            const uint32_t n2 = hi0 ^ c3 ^ a1;
            c0 = n0;
            c1 = lo1;
            c2 = n2;
            c3 = lo0;
            a0 += 0x9E3779B9u;
            a1 += 0xBB67AE85u;
        }
        b0 = c0;
        b1 = c1;
        b2 = c2;
        b3 = c3;
    }

    /* the stream after `drawn` draws */
    __device__ void resume(uint32_t klo, uint32_t khi, uint32_t px, uint32_t st, uint32_t sa, uint32_t drawn)
    {
        init(klo, khi, px, st, sa);
        n = drawn;
        if (n & 3u) block();
    }

    /* uniform in (0,1]: ((x >> 8) + 1) * 2^-24 */
    __device__ float uniform()
    {
        if ((n & 3u) == 0) block();
        const uint32_t j = n & 3u;
        const uint32_t x = j == 0 ? b0 : (j == 1 ? b1 : (j == 2 ? b2 : b3));
        ++n;
        return (float)((x >> 8) + 1u) * (1.0f / 16777216.0f);
    }
};

/* ------------------------------------------------------------------ */
/* Sampling                                                            */
/* ------------------------------------------------------------------ */

/* texel at integer position (tex2D at x+0.5, y+0.5), edges repeated */
__device__ __forceinline__ float texel(const float *__restrict__ img, int w, int h, int x, int y)
{
    x = min(max(x, 0), w - 1);
    y = min(max(y, 0), h - 1);
    return __ldg(img + (size_t)y * w + x);
}

/* Two FP32 operations per instruction (fma/mul/add.f32x2): half the issue
 * slots, each half rounded as the scalar operation. */
__device__ __forceinline__ unsigned long long pack2(float2 a)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long r)
{
    float2 a;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
    return a;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    unsigned long long r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)), "l"(pack2(c)));
    return unpack2(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    unsigned long long r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
    return unpack2(r);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    unsigned long long r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
    return unpack2(r);
}
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
/* The bilateral weight of a tap (HPM.cu:339-341) is exp(spatial + range):
 * the spatial terms of the window's 6 x 6 taps depend on |i| and |j| only and
 * are kept per block, those of rows 2 pair and 2 pair + 1 side by side. */
struct Spatial {
    float2 term[3][3]; /* [row pair][|j| = 5, 3, 1] */
};

__device__ __forceinline__ float rcp_approx(float a)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

__device__ __forceinline__ void spatial_terms(float sigma, Spatial *out)
{
    const int t = threadIdx.y * kBlockX + threadIdx.x;
    if (t < 18) {
        const int i = 2 * (t / 3) - 5, j = 5 - 2 * (t % 3);
        const float x = (float)i, y = (float)j;
        const float term = -sqrtf(x * x + y * y) * rcp_approx(2.0f * sigma * sigma);
        reinterpret_cast<float *>(&out->term[t / 6][t % 3])[(t / 3) & 1] = term;
    }
    __syncthreads();
}

__device__ __forceinline__ float tap_weight(float spatial, float ref, float center, float range_scale)
{
    return expf(__fmaf_rn(-fabsf(ref - center), range_scale, spatial));
}

/* The reference window of a pixel: its weights in shared memory, written once
 * by ref_window ([row pair][column][thread]: the weights of two rows side by
 * side for the packed sums of ncc_quad), and its pixels, read at each use from
 * a tile of the block's surroundings in shared memory (WinRow for blocks of
 * whole rows, WinTile for half-steps).  Computing the weights again at each
 * use would halve the block's shared memory but costs more than the texture
 * cache gains (refinement at 1600x1200, 10 sources: 1.80 against 1.57 ms). */
struct WinRow {
    static constexpr int kRows = kBlockY + 10, kPitch = kBlockX + 10;
    const Spatial *sp;
    float range_scale, mid; /* the pixel's own value */
    float2 *w;              /* its column of weights */
    const float *tile;      /* its first tap */
    __device__ __forceinline__ float ref(int ti, int tj) const { return tile[2 * tj * kPitch + 2 * ti]; }
};

/* Shared memory of a 32 x 2 block's reference windows.  The tile is read once
 * where 36 clamped loads a window came from global memory before, each with
 * its own clamping (k_init at 1600x1200, 10 sources: 1.11 -> 1.02 ms, in
 * geometric passes 0.96 -> 0.83; 641x481 with 4: 0.085 -> 0.074). */
struct RowMem {
    float2 w[kTaps / 2 * kBlock];
    float tile[WinRow::kRows * WinRow::kPitch];
    Spatial sp;

    /* fills the tile (all threads; edges repeated) and the spatial terms;
     * returns the window of the thread's pixel */
    __device__ __forceinline__ WinRow load(const ViewDev &rv, float sigma_spatial, float sigma_color)
    {
        const int x0 = (int)blockIdx.x * kBlockX - 5, y0 = (int)blockIdx.y * kBlockY - 5;
        const int tid = threadIdx.y * kBlockX + threadIdx.x;
        for (int i = tid; i < WinRow::kRows * WinRow::kPitch; i += kBlock)
            tile[i] = texel(rv.img, rv.w, rv.h, x0 + i % WinRow::kPitch, y0 + i / WinRow::kPitch);
        spatial_terms(sigma_spatial, &sp);
        const float *first = tile + threadIdx.y * WinRow::kPitch + threadIdx.x;
        return {&sp, rcp_approx(2.0f * sigma_color * sigma_color), first[5 * WinRow::kPitch + 5], w + tid, first};
    }
};

/* Half-step blocks: every tap of a pixel has the pixel's own checkerboard
 * colour (both offsets are odd), so the tile holds that colour only: row R is
 * image row y = y0 - 5 + R, entry c of it the column
 * x0 + par(y + 1) - 5 + 2 c, where par(y) = (y + colour) & 1 is the
 * parity of the updated columns of row y.  A tap of the pixel at (lx, ly) of
 * the block's patch is then row ly + 2 tj, entry lx + ti.  The pitch keeps a
 * warp's rows (of WW pixels each) on different banks. */
template <int WW>
struct WinTile {
    static constexpr int WH = 32 / WW, kRows = 2 * WH + 10, kCols = WW + 5;
    static constexpr int kPitch = WW == 4 ? 12 : (WW == 8 ? 24 : 48);
    const Spatial *sp;
    float range_scale, mid; /* the pixel's own value */
    float2 *w;              /* its column of weights */
    const float *tile;      /* its first tap */
    __device__ __forceinline__ float ref(int ti, int tj) const { return tile[2 * tj * kPitch + ti]; }
};

/* weights of rows 2 pair and 2 pair + 1 in column tj, given their pixels */
template <typename Win>
__device__ __forceinline__ float2 tap_weights(const Win &win, int pair, int tj, float2 ref)
{
    const float2 s = win.sp->term[pair][tj < 3 ? tj : 5 - tj];
    return make_float2(tap_weight(s.x, ref.x, win.mid, win.range_scale), tap_weight(s.y, ref.y, win.mid, win.range_scale));
}

/* Shared memory of a half-step block and its place in the image.  Pixel q of
 * the block (0 .. 63, a warp's 32 in lane order) lies at (x(q), y(q)). */
template <int WW>
struct Patch {
    using Tile = WinTile<WW>;
    const Spatial *sp;
    float2 *w;
    float *tile;
    float range_scale;
    int x0, y0, color;

    __device__ __forceinline__ int y(int q) const { return y0 + q / WW; }
    __device__ __forceinline__ int x(int q) const { return x0 + 2 * (q % WW) + ((y(q) + color) & 1); }
    __device__ __forceinline__ Tile win(int q) const
    {
        const float *first = tile + q / WW * Tile::kPitch + q % WW;
        return {sp, range_scale, first[5 * Tile::kPitch + 2 + ((y(q) + color) & 1)], w + q, first};
    }
};

/* Shared memory of a half-step block's reference windows. */
template <int WW>
struct PatchMem {
    using Tile = WinTile<WW>;
    float2 w[kTaps / 2 * kBlock];
    float tile[Tile::kRows * Tile::kPitch];
    Spatial sp;

    /* fills the tile (all threads; edges repeated) and the spatial terms */
    template <int NW>
    __device__ __forceinline__ Patch<WW> load(const PMArgs &a, int color)
    {
        const ViewDev &rv = a.view[0];
        const int x0 = (int)blockIdx.x * 2 * WW, y0 = (int)blockIdx.y * 2 * (32 / WW);
        for (int i = threadIdx.y * kBlockX + threadIdx.x; i < Tile::kRows * Tile::kCols; i += kBlockX * NW) {
            const int r = i / Tile::kCols, c = i - r * Tile::kCols, ty = y0 - 5 + r;
            tile[r * Tile::kPitch + c] = texel(rv.img, rv.w, rv.h, x0 + ((ty + 1 + color) & 1) - 5 + 2 * c, ty);
        }
        spatial_terms(a.sigma_spatial, &sp);
        return {&sp, w, tile, rcp_approx(2.0f * a.sigma_color * a.sigma_color), x0, y0, color};
    }
};

/* ------------------------------------------------------------------ */
/* Geometry (HPM.cu:65-133, 227-316, 445-481)                           */
/* ------------------------------------------------------------------ */

__device__ __forceinline__ void normalize3(float4 &v) /* HPM.cu:77-84 */
{
    const float n2 = v.x * v.x + v.y * v.y + v.z * v.z;
    const float inv = rsqrtf(n2);
    v.x *= inv;
    v.y *= inv;
    v.z *= inv;
}

__device__ __forceinline__ float4 view_direction(const HpmCamera &c, int px, int py, float depth)
{
    float X0 = depth * (px - c.K[2]) / c.K[0];
    float X1 = depth * (py - c.K[5]) / c.K[4];
    float X2 = depth;
    const float norm = sqrtf(X0 * X0 + X1 * X1 + X2 * X2);
    return make_float4(X0 / norm, X1 / norm, X2 / norm, 0.0f);
}

__device__ __forceinline__ float distance_to_origin(const HpmCamera &c, int px, int py, float depth, float4 n)
{
    const float X0 = depth * (px - c.K[2]) / c.K[0];
    const float X1 = depth * (py - c.K[5]) / c.K[4];
    const float X2 = depth;
    return -(n.x * X0 + n.y * X1 + n.z * X2);
}

__device__ __forceinline__ float depth_from_plane(const HpmCamera &c, float4 h, int px, int py)
{
    return -h.w * c.K[0] / ((px - c.K[2]) * h.x + (c.K[0] / c.K[4]) * (py - c.K[5]) * h.y + c.K[0] * h.z);
}

__device__ __forceinline__ float4 transform_normal(const HpmCamera &c, float4 h)
{
    float4 r;
    r.x = c.R[0] * h.x + c.R[3] * h.y + c.R[6] * h.z;
    r.y = c.R[1] * h.x + c.R[4] * h.y + c.R[7] * h.z;
    r.z = c.R[2] * h.x + c.R[5] * h.y + c.R[8] * h.z;
    r.w = h.w;
    return r;
}

__device__ __forceinline__ float4 transform_normal_to_ref(const HpmCamera &c, float4 h)
{
    float4 r;
    r.x = c.R[0] * h.x + c.R[1] * h.y + c.R[2] * h.z;
    r.y = c.R[3] * h.x + c.R[4] * h.y + c.R[5] * h.z;
    r.z = c.R[6] * h.x + c.R[7] * h.y + c.R[8] * h.z;
    r.w = h.w;
    return r;
}

__device__ __forceinline__ float dot3(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

__device__ float4 random_normal(const HpmCamera &c, int px, int py, Rng &rng, float depth) /* HPM.cu:135-161 */
{
    float q1 = 1.0f, q2 = 1.0f, s = 2.0f;
    while (s >= 1.0f) {
        q1 = 2.0f * rng.uniform() - 1.0f;
        q2 = 2.0f * rng.uniform() - 1.0f;
        s = q1 * q1 + q2 * q2;
    }
    const float sq = sqrtf(1.0f - s);
    float4 n = make_float4(2.0f * q1 * sq, 2.0f * q2 * sq, 1.0f - 2.0f * s, 0.0f);
    const float4 v = view_direction(c, px, py, depth);
    if (n.x * v.x + n.y * v.y + n.z * v.z > 0.0f) {
        n.x = -n.x;
        n.y = -n.y;
        n.z = -n.z;
    }
    normalize3(n);
    return n;
}

__device__ float4 perturbed_normal(const HpmCamera &c, int px, int py, float4 normal, Rng &rng,
                                   float pert) /* HPM.cu:163-198 */
{
    const float4 v = view_direction(c, px, py, 1.0f);
    const float a1 = (rng.uniform() - 0.5f) * pert;
    const float a2 = (rng.uniform() - 0.5f) * pert;
    const float a3 = (rng.uniform() - 0.5f) * pert;
    const float s1 = sinf(a1), s2 = sinf(a2), s3 = sinf(a3);
    const float c1 = cosf(a1), c2 = cosf(a2), c3 = cosf(a3);
    float R[9];
    R[0] = c2 * c3;
    R[1] = c3 * s1 * s2 - c1 * s3;
    R[2] = s1 * s3 + c1 * c3 * s2;
    R[3] = c2 * s3;
    R[4] = c1 * c3 + s1 * s2 * s3;
    R[5] = c1 * s2 * s3 - c3 * s1;
    R[6] = -s2;
    R[7] = c2 * s1;
    R[8] = c1 * c2;
    float4 p;
    p.x = R[0] * normal.x + R[1] * normal.y + R[2] * normal.z;
    p.y = R[3] * normal.x + R[4] * normal.y + R[5] * normal.z;
    p.z = R[6] * normal.x + R[7] * normal.y + R[8] * normal.z;
    p.w = normal.w;
    if (dot3(p, v) >= 0.0f) p = normal;
    normalize3(p);
    return p;
}

/* ComputeHomography (HPM.cu:227-287) with the hypothesis-independent part
 * (relative pose) precomputed per view pair. */
__device__ __forceinline__ void homography(const HpmCamera &rc, const HpmCamera &sc, const PairGeom &g, float4 h,
                                           float *H)
{
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        H[3 * i + 0] = g.Rrel[3 * i + 0] - g.trel[i] * h.x / h.w;
        H[3 * i + 1] = g.Rrel[3 * i + 1] - g.trel[i] * h.y / h.w;
        H[3 * i + 2] = g.Rrel[3 * i + 2] - g.trel[i] * h.z / h.w;
    }
    float tmp[9];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        tmp[3 * i + 0] = H[3 * i + 0] / rc.K[0];
        tmp[3 * i + 1] = H[3 * i + 1] / rc.K[4];
        tmp[3 * i + 2] = -H[3 * i + 0] * rc.K[2] / rc.K[0] - H[3 * i + 1] * rc.K[5] / rc.K[4] + H[3 * i + 2];
    }
    H[0] = sc.K[0] * tmp[0] + sc.K[2] * tmp[6];
    H[1] = sc.K[0] * tmp[1] + sc.K[2] * tmp[7];
    H[2] = sc.K[0] * tmp[2] + sc.K[2] * tmp[8];
    H[3] = sc.K[4] * tmp[3] + sc.K[5] * tmp[6];
    H[4] = sc.K[4] * tmp[4] + sc.K[5] * tmp[7];
    H[5] = sc.K[4] * tmp[5] + sc.K[5] * tmp[8];
    H[6] = sc.K[8] * tmp[6];
    H[7] = sc.K[8] * tmp[7];
    H[8] = sc.K[8] * tmp[8];
}

/* ComputeCorrespondingPoint (HPM.cu:289-296).  Integer pixel coordinates
 * are passed as floats: (float)(px + i) == (float)px + i exactly. */
__device__ __forceinline__ float2 warp(const float *H, float px, float py)
{
    const float x = H[0] * px + H[1] * py + H[2];
    const float y = H[3] * px + H[4] * py + H[5];
    const float z = H[6] * px + H[7] * py + H[8];
    return make_float2(x / z, y / z);
}

/* ------------------------------------------------------------------ */
/* Hoisted reference window                                            */
/* ------------------------------------------------------------------ */

struct RefStats {
    float inv;  /* 1 / sum of weights */
    float mean; /* weighted mean of the reference window */
    float var;  /* weighted variance of the reference window */
};

/* The reference-side half of ComputeBilateralNCC (HPM.cu:318-386) of a
 * thread's pixel: per-tap weights into shared memory, sums in the reference's
 * row-then-total order. */
template <typename Win>
__device__ RefStats ref_window(const Win &win)
{
    float sum_ref = 0.0f, sum_ref_ref = 0.0f, wsum = 0.0f;
    for (int pair = 0; pair < 3; ++pair) {
        float2 r_ref = make_float2(0.0f, 0.0f), r_rr = r_ref, r_w = r_ref;
#pragma unroll
        for (int tj = 0; tj < 6; ++tj) {
            const float2 rp = make_float2(win.ref(2 * pair, tj), win.ref(2 * pair + 1, tj));
            const float2 wgt = tap_weights(win, pair, tj, rp);
            win.w[(pair * 6 + tj) * kBlock] = wgt;
            const float2 m = mul2(wgt, rp);
            r_ref = add2(r_ref, m);
            r_rr = fma2(m, rp, r_rr);
            r_w = add2(r_w, wgt);
        }
        sum_ref = __fadd_rn(__fadd_rn(sum_ref, r_ref.x), r_ref.y);
        sum_ref_ref = __fadd_rn(__fadd_rn(sum_ref_ref, r_rr.x), r_rr.y);
        wsum = __fadd_rn(__fadd_rn(wsum, r_w.x), r_w.y);
    }
    RefStats s;
    s.inv = 1.0f / wsum;
    s.mean = sum_ref * s.inv;
    s.var = __fmaf_rn(sum_ref_ref, s.inv, -__fmul_rn(s.mean, s.mean));
    return s;
}

/* Nine source samples of a window, one of each 2 x 2 block of its taps: at
 * (x0 + 4 bi, y0 + 4 bj), the warped position (ComputeCorrespondingPoint,
 * HPM.cu:289-296) through the texture unit at +0.5 (HPM.cu:358-359).  One
 * definition for the NCC and the tap-sample export, so that both evaluate the
 * same expression. */
__device__ __forceinline__ void fetch_block(cudaTextureObject_t tex, const float *H, float x0, float y0, float *s)
{
    const float2 Hx = make_float2(H[0], H[3]), Hy = make_float2(H[1], H[4]), Hc = make_float2(H[2], H[5]);
    float2 my[3];
    float mz[3];
#pragma unroll
    for (int bj = 0; bj < 3; ++bj) {
        const float y = y0 + (float)(4 * bj);
        my[bj] = mul2(Hy, both(y));
        mz[bj] = __fmul_rn(H[7], y);
    }
#pragma unroll
    for (int bi = 0; bi < 3; ++bi) {
        const float x = x0 + (float)(4 * bi);
        const float2 z01 = add2(fma2(both(H[6]), both(x), make_float2(mz[0], mz[1])), both(H[8]));
        const float z2 = __fadd_rn(__fmaf_rn(H[6], x, mz[2]), H[8]);
#pragma unroll
        for (int bj = 0; bj < 3; ++bj) {
            const float2 xy = add2(fma2(Hx, both(x), my[bj]), Hc);
            const float2 q = add2(mul2(xy, both(rcp_approx(bj == 0 ? z01.x : (bj == 1 ? z01.y : z2)))), both(0.5f));
            s[bi * 3 + bj] = tex2D<float>(tex, q.x, q.y);
        }
    }
}

constexpr unsigned kAll = 0xffffffffu; /* a whole warp */

/* a or b, by a byte selector (0x3210 or 0x7654) */
__device__ __forceinline__ float pick(float a, float b, unsigned sel)
{
    return __uint_as_float(__byte_perm(__float_as_uint(a), __float_as_uint(b), sel));
}

/* The source-side half of ComputeBilateralNCC (HPM.cu:325-397), one window
 * per lane, for the whole warp at once: every lane passes the pixel (px, py),
 * plane, reference window and statistics of the window it wants, and whether
 * it wants one (need); all 32 lanes must call, with the same view.
 *
 * The four lanes of a quad fetch one window at a time, a 2 x 2 block of its
 * taps per texture instruction, then hand the samples to the window's own
 * lane, which sums them in the reference's order.  The texture unit serves a
 * quad whose taps lie together at 2.9 to 3.1 taps per clock and SM whatever
 * the planes of neighbouring pixels; with one window per lane, as many taps of
 * unrelated windows in a quad run at 1.2, and at 0.5 with little texture
 * cache.  Products and sums are paired into two-wide instructions, since the
 * issue slots are the next bound, with the roundings spelled out.
 *
 * The view goes through a warp reduction, whose result the hardware keeps once
 * per warp, so that the compiler takes it as the same in all lanes: otherwise
 * each texture instruction becomes a loop over the distinct texture handles of
 * its lanes (k_prop_refine at 1600x1200, 10 sources: 3.70 against 1.80 ms; a
 * shuffle does it too, but k_prop_dirs then takes 1.76 against 1.68 ms with 5). */
template <typename Win>
__device__ __forceinline__ float ncc_quad(const PMArgs &a, int v, int px, int py, bool need, float4 h, const Win &win,
                                          const RefStats &rs)
{
    v = (int)__reduce_max_sync(kAll, (unsigned)v);
    const HpmCamera &sc = a.cam[v];
    float H[9];
    homography(a.cam[0], sc, a.pairs[v], h, H);
    const float fpx = (float)px, fpy = (float)py;
    const float2 pt = warp(H, fpx, fpy);
    /* the reference reaches 2 for a flat window after the taps */
    const bool go = need && !(pt.x >= sc.width || pt.x < 0.0f || pt.y >= sc.height || pt.y < 0.0f) &&
                    !(rs.var < 1e-5f);
    const unsigned ball = __ballot_sync(kAll, go);
    if (ball == 0) return 2.0f;
    const cudaTextureObject_t tex = a.view[v].tex;
    const int lane = threadIdx.x, l = lane & 3;
    const unsigned quad = (ball >> (lane & 28)) & 15u;
    float s[4][9];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        float G[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) G[e] = __shfl_sync(kAll, H[e], w, 4);
        const float gx = __shfl_sync(kAll, fpx, w, 4), gy = __shfl_sync(kAll, fpy, w, 4);
        /* without a window to fetch the samples stay unset: only the lane
         * that has none sums them */
        if ((quad >> w) & 1u) {
            /* lane l takes tap l ^ w of each block (bit 0: along x, bit 1:
             * along y), so that the hand-over below needs no select on the
             * receiving side */
            const int tp = l ^ w;
            fetch_block(tex, G, gx + (float)(2 * (tp & 1) - 5), gy + (float)(2 * (tp >> 1) - 5), s[w]);
        }
    }
    /* byte selectors, not predicates: too many are live for those */
    const unsigned pick1 = (l & 1) ? 0x7654u : 0x3210u, pick2 = (l & 2) ? 0x7654u : 0x3210u;
    float sum_src = 0.0f, sum_src_src = 0.0f, sum_ref_src = 0.0f;
#pragma unroll
    for (int bi = 0; bi < 3; ++bi) {
        /* rows 2 bi and 2 bi + 1 side by side */
        float2 r_src = make_float2(0.0f, 0.0f), r_ss = r_src, r_rs = r_src;
#pragma unroll
        for (int bj = 0; bj < 3; ++bj) {
            const int b = bi * 3 + bj;
            /* p[d] = s[l ^ d][b]: what lane l ^ d is waiting for */
            float q[4], p[4], tap[4];
#pragma unroll
            for (int d = 0; d < 4; ++d) q[d] = pick(s[d][b], s[d ^ 1][b], pick1);
#pragma unroll
            for (int d = 0; d < 4; ++d) p[d] = pick(q[d], q[d ^ 2], pick2);
            tap[0] = p[0];
#pragma unroll
            for (int d = 1; d < 4; ++d) tap[d] = __shfl_xor_sync(kAll, p[d], d);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float2 sp = make_float2(tap[2 * e], tap[2 * e + 1]);
                const float2 rp = make_float2(win.ref(2 * bi, 2 * bj + e), win.ref(2 * bi + 1, 2 * bj + e));
                const float2 wt = win.w[(bi * 6 + 2 * bj + e) * kBlock], wr = mul2(wt, rp);
                const float2 m = mul2(wt, sp);
                r_src = add2(r_src, m);
                r_ss = fma2(m, sp, r_ss);
                r_rs = fma2(wr, sp, r_rs);
            }
        }
        sum_src = __fadd_rn(__fadd_rn(sum_src, r_src.x), r_src.y);
        sum_src_src = __fadd_rn(__fadd_rn(sum_src_src, r_ss.x), r_ss.y);
        sum_ref_src = __fadd_rn(__fadd_rn(sum_ref_src, r_rs.x), r_rs.y);
    }
    const float mean_src = __fmul_rn(sum_src, rs.inv);
    const float var_src = __fmaf_rn(sum_src_src, rs.inv, -__fmul_rn(mean_src, mean_src));
    if (!go || var_src < 1e-5f) return 2.0f;
    const float covar = __fmaf_rn(sum_ref_src, rs.inv, -__fmul_rn(rs.mean, mean_src));
    const float vv = sqrtf(rs.var * var_src);
    return fmaxf(0.0f, fminf(2.0f, 1.0f - covar / vv));
}

/* another lane's statistics */
__device__ __forceinline__ RefStats stats_of(const RefStats &rs, int lane)
{
    return {__shfl_sync(kAll, rs.inv, lane), __shfl_sync(kAll, rs.mean, lane), __shfl_sync(kAll, rs.var, lane)};
}

__device__ __forceinline__ unsigned lanes_below() { return (1u << threadIdx.x) - 1u; }

/* ComputeMultiViewCostVector (HPM.cu:438-443) of the warp's pixels into
 * out[v * stride] of the lanes that want it; all 32 lanes must call. */
template <typename Win>
__device__ __forceinline__ void cost_vector(const PMArgs &a, int px, int py, bool need, float4 h, const Win &win,
                                            const RefStats &rs, float *out, int stride)
{
#pragma unroll 1
    for (int v = 1; v < a.n; ++v) {
        const float c = ncc_quad(a, v, px, py, need, h, win, rs);
        if (need) out[(size_t)(v - 1) * stride] = c;
    }
    if (a.counters && need) atomicAdd(&a.counters[0], (unsigned long long)(a.n - 1));
}

__device__ __forceinline__ void sort_small(float *d, int n) /* HPM.cu:3-12 */
{
    int j;
    for (int i = 1; i < n; i++) {
        const float tmp = d[i];
        for (j = i; j >= 1 && tmp < d[j - 1]; j--) d[j] = d[j - 1];
        d[j] = tmp;
    }
}

/* ComputeMultiViewInitialCostandSelectedViews (HPM.cu:399-436) from a cost
 * vector cv[v * stride]. */
__device__ float initial_cost_from(const PMArgs &a, const float *cv, int stride, uint32_t *views)
{
    float srt[kMaxSrc];
    const int S = a.n - 1;
    int valid = 0;
    for (int v = 0; v < S; ++v) {
        srt[v] = cv[(size_t)v * stride];
        if (srt[v] < 2.0f) valid++;
    }
    sort_small(srt, S);
    uint32_t sel = 0;
    const int top_k = min(valid, a.top_k);
    float result = 2.0f;
    if (top_k > 0) {
        float cost = 0.0f;
        for (int i = 0; i < top_k; ++i) cost += srt[i];
        const float thr = srt[top_k - 1];
        for (int i = 0; i < S; ++i)
            if (cv[(size_t)i * stride] <= thr) sel |= 1u << i;
        result = cost / top_k;
    }
    *views = sel;
    return result;
}

__device__ __forceinline__ void world_point(const HpmCamera &c, float x, float y, float depth, float *P)
{
    float X0 = depth * (x - c.K[2]) / c.K[0];
    float X1 = depth * (y - c.K[5]) / c.K[4];
    float X2 = depth;
    const float T0 = c.R[0] * X0 + c.R[3] * X1 + c.R[6] * X2;
    const float T1 = c.R[1] * X0 + c.R[4] * X1 + c.R[7] * X2;
    const float T2 = c.R[2] * X0 + c.R[5] * X1 + c.R[8] * X2;
    const float Cx = -(c.R[0] * c.t[0] + c.R[3] * c.t[1] + c.R[6] * c.t[2]);
    const float Cy = -(c.R[1] * c.t[0] + c.R[4] * c.t[1] + c.R[7] * c.t[2]);
    const float Cz = -(c.R[2] * c.t[0] + c.R[5] * c.t[1] + c.R[8] * c.t[2]);
    P[0] = T0 + Cx;
    P[1] = T1 + Cy;
    P[2] = T2 + Cz;
}

__device__ __forceinline__ void project(const float *P, const HpmCamera &c, float *pt, float &depth)
{
    const float t0 = c.R[0] * P[0] + c.R[1] * P[1] + c.R[2] * P[2] + c.t[0];
    const float t1 = c.R[3] * P[0] + c.R[4] * P[1] + c.R[5] * P[2] + c.t[1];
    const float t2 = c.R[6] * P[0] + c.R[7] * P[1] + c.R[8] * P[2] + c.t[2];
    depth = c.K[6] * t0 + c.K[7] * t1 + c.K[8] * t2;
    pt[0] = (c.K[0] * t0 + c.K[1] * t1 + c.K[2] * t2) / depth;
    pt[1] = (c.K[3] * t0 + c.K[4] * t1 + c.K[5] * t2) / depth;
}

/* ComputeGeomConsistencyCost (HPM.cu:483-508; capped at a.geom_max, 5 there
 * and 3 in ACMM.cu:494-519), in two halves, so that callers can have several
 * source depths on their way before they use one: the world point of pixel
 * (px, py) on plane h, its place in view v with the depth there, and the
 * distance of that depth's reprojection. */
__device__ __forceinline__ void geom_point(const PMArgs &a, float4 h, int px, int py, float *P)
{
    const float depth = depth_from_plane(a.cam[0], h, px, py);
    world_point(a.cam[0], (float)px, (float)py, depth, P);
}

__device__ __forceinline__ float geom_source(const PMArgs &a, int v, const float *P, float *spt)
{
    float sd;
    project(P, a.cam[v], spt, sd);
    const ViewDev &sv = a.view[v];
    return texel(sv.depth, sv.w, sv.h, __float2int_rz(spt[0]), __float2int_rz(spt[1]));
}

__device__ __forceinline__ float geom_distance(const PMArgs &a, int v, int px, int py, const float *spt, float src_depth)
{
    if (src_depth == 0.0f) return a.geom_max;
    float Q[3], bpt[2], rd;
    world_point(a.cam[v], spt[0], spt[1], src_depth, Q);
    project(Q, a.cam[0], bpt, rd);
    const float dx = px - bpt[0], dy = py - bpt[1];
    return fminf(a.geom_max, sqrtf(dx * dx + dy * dy));
}

__device__ __forceinline__ void count_geom(const PMArgs &a, unsigned n)
{
    if (a.counters) atomicAdd(&a.counters[1], (unsigned long long)n);
}

/* ------------------------------------------------------------------ */
/* Kernels                                                             */
/* ------------------------------------------------------------------ */

/* R_relative and t_relative of HPM.cu:229-255, with the same expressions. */
__global__ void k_pair_geom(const __grid_constant__ PMArgs a, PairGeom *out)
{
    const int v = threadIdx.x;
    if (v < 1 || v >= a.n) return;
    const HpmCamera &ref_camera = a.cam[0], &src_camera = a.cam[v];
    float ref_C[3], src_C[3];
    ref_C[0] = -(ref_camera.R[0] * ref_camera.t[0] + ref_camera.R[3] * ref_camera.t[1] + ref_camera.R[6] * ref_camera.t[2]);
    ref_C[1] = -(ref_camera.R[1] * ref_camera.t[0] + ref_camera.R[4] * ref_camera.t[1] + ref_camera.R[7] * ref_camera.t[2]);
    ref_C[2] = -(ref_camera.R[2] * ref_camera.t[0] + ref_camera.R[5] * ref_camera.t[1] + ref_camera.R[8] * ref_camera.t[2]);
    src_C[0] = -(src_camera.R[0] * src_camera.t[0] + src_camera.R[3] * src_camera.t[1] + src_camera.R[6] * src_camera.t[2]);
    src_C[1] = -(src_camera.R[1] * src_camera.t[0] + src_camera.R[4] * src_camera.t[1] + src_camera.R[7] * src_camera.t[2]);
    src_C[2] = -(src_camera.R[2] * src_camera.t[0] + src_camera.R[5] * src_camera.t[1] + src_camera.R[8] * src_camera.t[2]);
    PairGeom g;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            g.Rrel[3 * i + j] = src_camera.R[3 * i + 0] * ref_camera.R[3 * j + 0] +
                                src_camera.R[3 * i + 1] * ref_camera.R[3 * j + 1] +
                                src_camera.R[3 * i + 2] * ref_camera.R[3 * j + 2];
    float C_relative[3];
    C_relative[0] = (ref_C[0] - src_C[0]);
    C_relative[1] = (ref_C[1] - src_C[1]);
    C_relative[2] = (ref_C[2] - src_C[2]);
    for (int i = 0; i < 3; ++i)
        g.trel[i] = src_camera.R[3 * i + 0] * C_relative[0] + src_camera.R[3 * i + 1] * C_relative[1] +
                    src_camera.R[3 * i + 2] * C_relative[2];
    out[v] = g;
}

/* Where a pixel's per-pixel buffers live.  Linear pixel indices 2k and
 * 2k + 1 always have different checkerboard colours (neighbours in a row, or
 * across a row end when W is odd), so center >> 1 numbers the pixels of one
 * colour densely: a half-step's hand-off rows (cand_*, one colour at a time)
 * are indexed by it, and the cost-vector cache keeps one such plane per
 * colour.  A half-step then writes whole 32-byte sectors instead of every
 * other word of them. */
struct Slot {
    size_t nh; /* pixels of one colour, rounded up: ceil(W * H / 2) */
    int hc;    /* hand-off slot: center >> 1 */
    size_t cs; /* cache slot: colour plane + hc */
};

__device__ __forceinline__ Slot slot_of(const PMArgs &a, int px, int py)
{
    Slot sl;
    sl.nh = ((size_t)a.W * a.H + 1) >> 1;
    sl.hc = (py * a.W + px) >> 1;
    sl.cs = (size_t)((px + py) & 1) * sl.nh + (size_t)sl.hc;
    return sl;
}

/* Cost-vector cache: for every pixel the cost vector of its current
 * hypothesis, [view][colour][slot].  Written by the initialisation and by
 * every update, read instead of re-scoring the current hypothesis
 * (HPM.cu:1637-1638): NCC is a pure function of (pixel, plane, view), so the
 * cached values are the ones the re-score would produce. */
__device__ __forceinline__ float *cache_at(const PMArgs &a, int v, const Slot &sl)
{
    return a.cost_cache + (size_t)v * 2 * sl.nh + sl.cs;
}

/* RandomInitialization, HPM.cu:510-558.  One thread per pixel. */
__device__ __forceinline__ void init_body(const PMArgs &a, int px, int py, const WinRow &win, float *sCV, int tid)
{
    const bool act = px < a.W && py < a.H;
    /* lanes outside the image stay for the warp's windows, on a pixel inside */
    const int cx = min(px, a.W - 1), cy = min(py, a.H - 1);
    const int center = cy * a.W + cx;
    const HpmCamera &cam = a.cam[0];
    const RefStats rs = ref_window(win);
    Rng rng;
    rng.init(a.seed_lo, a.seed_hi, (uint32_t)center, 0u, a.salt);
    float4 h;
    if (a.geom || a.hier) {
        if (a.hier == 1) {
            /* ACMM+NESP hierarchy pass (ACMM.cu:538-604): the acceptance
             * threshold is the initial cost of the plane the reference holds
             * before the normal is filled in, a zero normal with the depth as
             * its distance (ACMM.cpp:707-713 sets only .w of a fresh,
             * zero-filled array); at the maps' own size (hier 2) the
             * reference leaves it unset, taken as 0 */
            const float4 hz = make_float4(0.0f, 0.0f, 0.0f, a.planes[center].w);
            float *cvz = sCV + tid;
            cost_vector(a, px, py, act, hz, win, rs, cvz, kBlock);
            uint32_t unused;
            if (act) a.pre_costs[center] = initial_cost_from(a, cvz, kBlock, &unused);
        } else if (a.hier == 2) {
            if (act) a.pre_costs[center] = 0.0f;
        }
        h = transform_normal_to_ref(cam, a.planes[center]);
        const float depth = h.w;
        h.w = distance_to_origin(cam, cx, cy, depth, h);
    } else if (a.prior) {
        if (a.masks[center] > 0 && a.costs[center] >= 0.1f) {
            const float pert = 0.02f;
            const float4 hp = a.prior_planes[center];
            float dp = hp.w;
            const float lo = (1 - 3 * pert) * dp;
            const float hi = (1 + 3 * pert) * dp;
            dp = rng.uniform() * (hi - lo) + lo;
            h = perturbed_normal(cam, cx, cy, hp, rng, (float)(3 * pert * kPiD));
            h.w = dp;
        } else {
            /* the previous pass's world-frame normal, reused as it is
             * (HPM.cu:547-551); with fix_quirks rotated back to the
             * reference frame first, as the geometric branch does */
            h = a.fix_quirks ? transform_normal_to_ref(cam, a.planes[center]) : a.planes[center];
            const float depth = h.w;
            h.w = distance_to_origin(cam, cx, cy, depth, h);
        }
    } else {
        const float depth = rng.uniform() * (a.dmax - a.dmin) + a.dmin;
        h = random_normal(cam, cx, cy, rng, depth);
        h.w = distance_to_origin(cam, cx, cy, depth, h);
    }
    float *cv = sCV + tid;
    cost_vector(a, px, py, act, h, win, rs, cv, kBlock);
    if (!act) return;
    uint32_t sel;
    const float c = initial_cost_from(a, cv, kBlock, &sel);
    a.planes[center] = h;
    a.costs[center] = c;
    a.views[center] = sel;
    if (a.cost_cache) {
        const Slot sl = slot_of(a, cx, cy);
        for (int v = 0; v < a.n - 1; ++v) *cache_at(a, v, sl) = cv[v * kBlock];
    }
}

__global__ void __launch_bounds__(kBlock, HPM_P0_MIN_BLOCKS) k_init(const __grid_constant__ PMArgs a)
{
    __shared__ RowMem sRow;
    __shared__ float sCV[kMaxSrc * kBlock];
    const int tid = threadIdx.y * kBlockX + threadIdx.x;
    init_body(a, blockIdx.x * kBlockX + threadIdx.x, blockIdx.y * kBlockY + threadIdx.y,
              sRow.load(a.view[0], a.sigma_spatial, a.sigma_color), sCV, tid);
}

/* Validity of the first site of direction k at extension round r (HPM.cu:1252-1445 and the
 * Extended* functions 560-1034).  Directions: 0 left_up, 1 up_far, 2 right_up, 3 down_far,
 * 4 right_down, 5 left_far, 6 left_down, 7 right_far (HPM.cu:1245). */
__device__ __forceinline__ bool first_site_valid(int k, int r, int px, int py, int W, int H)
{
    const int s = 10 * r, d = 8 * r;
    switch (k) {
    case 1: return py > 4 + s;
    case 3: return py < H - 5 - s;
    case 5: return px > 4 + s;
    case 7: return px < W - 5 - s;
    case 0: return px > 4 + d && py > 5 + d;
    case 2: return px < W - 6 - d && py > 4 + d;
    case 4: return px < W - 5 - d && py < H - 6 - d;
    default: return px > 5 + d && py < H - 5 - d;
    }
}

/* NESP site choice of one direction at round r.  Strips: 5 sites 2 apart
 * from +/-(5+10r), the right strip keeps the maximum (HPM.cu:1330, 744;
 * the minimum with fix_quirks).
 * Polylines: start (+/-5|6) shifted 8r outward, then 7 zig-zag steps of 2
 * (HPM.cu:1346-1471). */
__device__ __forceinline__ int select_site(const PMArgs &a, int k, int r, int px, int py)
{
    const int W = a.W, H = a.H;
    const float *costs = a.costs;
    /* all sites' costs are loaded before the first is compared */
    int q[8];
    float c[8];
    bool in[8];
    const int n = (k & 1) ? 5 : 8;
    if (k & 1) {
        const int dx = (k == 5) ? -1 : (k == 7 ? 1 : 0);
        const int dy = (k == 1) ? -1 : (k == 3 ? 1 : 0);
        const int off = 5 + 10 * r;
        bool ok = true;
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            if (i > 0) {
                switch (k) {
                case 1: ok = ok && py > 4 + 2 * i + 10 * r; break;
                case 3: ok = ok && py < H - 5 - 2 * i - 10 * r; break;
                case 5: ok = ok && px > 4 + 2 * i + 10 * r; break;
                default: ok = ok && px < W - 5 - 2 * i - 10 * r; break;
                }
            }
            q[i] = (py + dy * (off + 2 * i)) * W + (px + dx * (off + 2 * i));
            in[i] = ok;
            c[i] = ok ? costs[q[i]] : 0.0f;
        }
    } else {
        int sx, sy, ex, ey, ox, oy; /* start, even step, odd step */
        switch (k) {
        case 0: sx = -5 - 8 * r; sy = -6 - 8 * r; ex = -2; ey = 0; ox = 0; oy = -2; break;
        case 2: sx = 6 + 8 * r; sy = -5 - 8 * r; ex = 0; ey = -2; ox = 2; oy = 0; break;
        case 4: sx = 5 + 8 * r; sy = 6 + 8 * r; ex = 2; ey = 0; ox = 0; oy = 2; break;
        default: sx = -6 - 8 * r; sy = 5 + 8 * r; ex = 0; ey = 2; ox = -2; oy = 0; break;
        }
        int x = px + sx, y = py + sy;
        bool ok = true;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (i > 0) {
                x += (i & 1) ? ex : ox;
                y += (i & 1) ? ey : oy;
                ok = ok && x >= 0 && x < W && y < H && y >= 0;
            }
            q[i] = y * W + x;
            in[i] = ok;
            c[i] = ok ? costs[q[i]] : 0.0f;
        }
    }
    int best = q[0];
    float cmin = c[0];
#pragma unroll
    for (int i = 1; i < 8; ++i)
        if (i < n && in[i] && ((k == 7 && !a.fix_quirks) ? (cmin < c[i]) : (c[i] < cmin))) {
            cmin = c[i];
            best = q[i];
        }
    return best;
}

__device__ __forceinline__ float restricted_prior(float depth_diff, float angle_cos, float two_dss, float two_ass)
{
    const float gamma = 0.5f;
    const float angle_diff = acosf(angle_cos);
    return gamma + expf(-depth_diff * depth_diff / two_dss) * expf(-angle_diff * angle_diff / two_ass);
}

__device__ __forceinline__ bool same_plane(float4 p, float4 q)
{
    return __float_as_uint(p.x) == __float_as_uint(q.x) && __float_as_uint(p.y) == __float_as_uint(q.y) &&
           __float_as_uint(p.z) == __float_as_uint(q.z) && __float_as_uint(p.w) == __float_as_uint(q.w);
}

/* One red/black half-step runs as three kernels that hand the per-pixel cost
 * matrix over through L2 instead of holding it in shared memory for the
 * whole pixel update (8 x S floats per pixel is what limits occupancy):
 *
 *   k_prop_dirs    NESP site choice, direction cost vectors, extension
 *                  (HPM.cu:1222-1543)
 *   k_prop_select  joint view selection and candidate choice
 *                  (HPM.cu:1548-1725)
 *   k_prop_refine  PlaneHypothesisRefinement (HPM.cu:1143-1220)
 *
 * The selection is one thread per pixel with an array per view in registers;
 * between the window loops of the other two its code alone pushed them out of
 * the instruction cache.  The other colour is read-only during all three, so
 * splitting the pixel update changes nothing in what is computed. */

#define CAG(k, v) a.cand_costs[(size_t)((k) * S + (v)) * sl.nh + sl.hc]
/* Hand-off stores use the streaming cache policy (st.global.cs, evict
 * first): the rows are read once by the next kernel, and at ~0.5 GB a
 * half-step they would otherwise push the source images out of L2. */
#define CAG_PUT(k, v, x) __stcs(&CAG(k, v), (x))

/* Where the cost row of direction k lives, 4 bits per direction in the
 * pixel's hand-off code (cand_flags): the row itself, the cost-vector cache
 * (the candidate equals the current hypothesis), the row of an earlier
 * direction with the same plane, or nowhere (an invalid direction, whose row
 * holds 2 at [0][0] and 0 elsewhere because float cost_array[8][32] =
 * { 2.0f } sets only [0][0], HPM.cu:1244).  Copies and invalid rows are
 * resolved on reading instead of being written out. */
constexpr uint32_t kRowCache = 8, kRowOwn = 9, kRowNone = 10;
constexpr uint32_t kCodeAllNone = 0xAAAAAAAAu;

__device__ __forceinline__ bool dir_valid(uint32_t code, int k) { return ((code >> (4 * k)) & 15u) != kRowNone; }

__device__ __forceinline__ float dir_cost(const PMArgs &a, uint32_t code, int k, int v, int S, const Slot &sl)
{
    const uint32_t src = (code >> (4 * k)) & 15u;
    if (src == kRowOwn) return CAG(k, v);
    if (src == kRowCache) return *cache_at(a, v, sl);
    if (src < 8) return CAG(src, v);
    return (a.fix_quirks || (k == 0 && v == 0)) ? 2.0f : 0.0f; /* fix_quirks: the intended {2, 2, ...} */
}

/* Shared memory of the direction kernel's block: the sites of each pixel's
 * candidates, the statistics of its window, and the windows still to score,
 * packed: lanes take them 32 at a time whatever pixel they belong to, so that
 * a pixel with few distinct candidates leaves no idle lanes.  item: candidate
 * << 6 | pixel of the block; judge: of direction 0's row, the costs below the
 * three rounds' thresholds and those above 1.2, 8 bits each. */
struct DirItems {
    int pos[8][kBlock];
    RefStats stats[kBlock];
    uint32_t judge[kBlock];
    uint16_t item[kBlockY][8 * 32];
    int count[kBlockY];
};

__device__ __forceinline__ uint32_t judge_cost(float c, const float *good)
{
    return (c < good[0] ? 1u : 0u) | (c < good[1] ? 1u << 8 : 0u) | (c < good[2] ? 1u << 16 : 0u) |
           (c > 1.2f ? 1u << 24 : 0u);
}

template <int WW, int NW>
__device__ __forceinline__ void prop_dirs_body(const PMArgs &a, int iter, const Patch<WW> &patch, DirItems &items)
{
    const int W = a.W, H = a.H, S = a.n - 1;
    /* the first two warps own the block's pixels, others only score */
    const int lane = threadIdx.x, wv = threadIdx.y, q0 = (wv & 1) * kBlockX;
    const bool owner = NW == kBlockY || wv < kBlockY;
    const int px = patch.x(q0 + lane), py = patch.y(q0 + lane);
    const bool act = owner && px < W && py < a.rows_cov;
    /* lanes outside the image stay for the warp's windows, on a pixel inside */
    const int cx = min(px, W - 1), cy = min(py, H - 1);
    const int center = cy * W + cx;
    const Slot sl = slot_of(a, cx, cy);
    const float4 cur = a.planes[center];
    if (owner) {
        items.stats[q0 + lane] = ref_window(patch.win(q0 + lane));
        items.judge[q0 + lane] = 0;
    }
    /* JudgeExtend's threshold of each round, by one lane each */
    float good[3];
    {
        const int r = min(lane, 2);
        const float g = (float)(0.8 * exp(-iter * iter * (3 - r) / 90.0));
#pragma unroll
        for (int i = 0; i < 3; ++i) good[i] = __shfl_sync(kAll, g, i);
    }

    int pos[8];
    uint32_t flags = 0;
    pos[0] = center - 5 - 6 * W;
    pos[1] = center - W * 5;
    pos[2] = center + 6 - 5 * W;
    pos[3] = center + W * 5;
    pos[4] = center + 5 + 6 * W;
    pos[5] = center - 5;
    pos[6] = center - 6 + 5 * W;
    pos[7] = center + 5;
    /* 1) NESP sites of the 8 directions.  Identical planes give identical
     * cost vectors: a candidate whose plane equals the current hypothesis
     * (cost vector cached) or an earlier candidate reuses those values
     * (dir_cost resolves the row on reading). */
    uint32_t code = kCodeAllNone; /* 4 bits per direction */
    uint32_t eval_mask = 0;
    float4 plane[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        plane[k] = cur;
        if (!act || !first_site_valid(k, 0, px, py, W, H)) continue;
        flags |= 1u << k;
        pos[k] = select_site(a, k, 0, px, py);
        items.pos[k][q0 + lane] = pos[k];
        plane[k] = a.planes[pos[k]];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (!((flags >> k) & 1u)) continue;
        uint32_t src = same_plane(plane[k], cur) ? kRowCache : kRowNone;
#pragma unroll
        for (int j = 0; j < k; ++j)
            if (src == kRowNone && ((flags >> j) & 1u) && same_plane(plane[k], plane[j])) src = (uint32_t)j;
        if (src == kRowNone) {
            src = kRowOwn;
            eval_mask |= 1u << k;
        }
        code = (code & ~(15u << (4 * k))) | (src << (4 * k));
    }
    /* direction 0's row, where it is not scored here: judged on the spot */
    auto judge_row = [&](uint32_t src) {
        const float *row = src == kRowCache ? cache_at(a, 0, sl) : &CAG(src, 0);
        const size_t stride = src == kRowCache ? 2 * sl.nh : sl.nh;
        uint32_t sum = 0;
#pragma unroll 5
        for (int v = 0; v < S; ++v) sum += judge_cost(row[(size_t)v * stride], good);
        items.judge[q0 + lane] = sum;
    };
    if ((code & 15u) == kRowCache) judge_row(kRowCache);
    /* 2) the distinct candidates, view by view, so that the threads of a
     * block sample one source image at a time (texture-cache locality).
     * Round 0 scores the sites; rounds 1 to 3 are the extension.
     * Extension: only the left-up polyline can extend, because
     * bool symbol_eight_orientations[10] = { true } sets index 0 only
     * (HPM.cu:1475).  JudgeExtend: HPM.cu:1036-1059, from counts kept while
     * the row is scored.  The extension has few windows a view, so both warps'
     * are packed together and the views dealt out to the warps. */
    bool extend = (flags & 1u) != 0;
    bool detached = false; /* rows that copy direction 0's first row hold their own copy */
#pragma unroll 1
    for (int round = 0; round < 4; ++round) {
        int total = 0;
        if (round == 0) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const bool mine = (eval_mask >> k) & 1u;
                const unsigned m = __ballot_sync(kAll, mine);
                if (mine) items.item[wv & 1][total + __popc(m & lanes_below())] = (uint16_t)(k << 6 | (q0 + lane));
                total += __popc(m);
            }
            if constexpr (NW == kBlockY) {
                __syncwarp();
            } else { /* an owner's windows go to every second warp, view by view */
                if (owner && lane == 0) items.count[wv] = total;
                __syncthreads();
                total = items.count[wv & 1];
            }
        } else {
            const int r = round - 1;
            bool mine = false;
            if (!__syncthreads_or(extend)) break; /* also: the rows and counts of the last round are there */
            if (extend) {
                const uint32_t counts = items.judge[q0 + lane];
                if (((counts >> (8 * r)) & 255u) >= 1u && (counts >> 24) <= 2u) extend = false;
            }
            /* an invalid first site keeps site and costs: flag[0] is set */
            if (extend && first_site_valid(0, r, px, py, W, H)) {
                const int best = select_site(a, 0, r, px, py);
                /* a better previous site is kept */
                if (!(a.costs[best] > a.costs[pos[0]])) {
                    const float4 prev = a.planes[pos[0]];
                    const float4 p = a.planes[best];
                    pos[0] = best;
                    items.pos[0][q0 + lane] = best;
                    if (!same_plane(p, prev)) {
                        /* direction 0's row changes: the rows that refer to
                         * it keep the values it had when they were chosen */
                        if (!detached) {
                            detached = true;
#pragma unroll
                            for (int k = 1; k < 8; ++k)
                                if (((code >> (4 * k)) & 15u) == 0u) {
                                    for (int v = 0; v < S; ++v) CAG_PUT(k, v, dir_cost(a, code, 0, v, S, sl));
                                    code = (code & ~(15u << (4 * k))) | (kRowOwn << (4 * k));
                                }
                        }
                        float first[8]; /* loaded together; equal planes have equal first components */
#pragma unroll
                        for (int j = 1; j < 8; ++j) first[j] = ((flags >> j) & 1u) ? a.planes[pos[j]].x : 0.0f;
                        int src = -1;
#pragma unroll
                        for (int j = 1; j < 8; ++j)
                            if (src < 0 && ((flags >> j) & 1u) && __float_as_uint(first[j]) == __float_as_uint(p.x) &&
                                same_plane(p, a.planes[pos[j]]))
                                src = j;
                        if (same_plane(p, cur)) {
                            code = (code & ~15u) | kRowCache;
                            judge_row(kRowCache);
                        } else if (src >= 0) {
                            const uint32_t sj = (code >> (4 * src)) & 15u, at = sj == kRowOwn ? (uint32_t)src : sj;
                            code = (code & ~15u) | at;
                            judge_row(at);
                        } else {
                            mine = true;
                            code = (code & ~15u) | kRowOwn;
                            items.judge[q0 + lane] = 0;
                        }
                    }
                }
            }
            eval_mask = mine ? 1u : 0u;
            const unsigned m = __ballot_sync(kAll, mine);
            if (owner && lane == 0) items.count[wv] = __popc(m);
            __syncthreads();
            if (mine) items.item[0][(wv ? items.count[0] : 0) + __popc(m & lanes_below())] = (uint16_t)(q0 + lane);
            total = items.count[0] + items.count[1];
            __syncthreads();
        }
        const uint16_t *list = items.item[round == 0 ? wv & 1 : 0];
        const int step = round == 0 ? NW / kBlockY : NW;
#pragma unroll 1
        for (int v = round == 0 ? wv / kBlockY : wv; v < S; v += step)
#pragma unroll 1
            for (int base = 0; base < total; base += 32) {
                const bool need = base + lane < total;
                const int it = list[need ? base + lane : 0], k = it >> 6, q = it & 63;
                const RefStats st = items.stats[q];
                const int qx = patch.x(q), qy = patch.y(q);
                const float c = ncc_quad(a, v + 1, qx, qy, need, a.planes[need ? items.pos[k][q] : center], patch.win(q), st);
                if (need) {
                    __stcs(&a.cand_costs[(size_t)(k * S + v) * sl.nh + ((qy * W + qx) >> 1)], c);
                    if (k == 0) atomicAdd(&items.judge[q], judge_cost(c, good));
                }
            }
        if (a.counters && eval_mask) atomicAdd(&a.counters[0], (unsigned long long)(__popc(eval_mask) * S));
    }
    __syncthreads();
    if (!act) return;
    /* 3) every valid direction's row in its own slot: a row that refers to
     * the cost-vector cache or to an earlier direction (always one that owns
     * its row) is copied there, so that the refinement reads each row with
     * one load and no decoding; the code then holds only own and none */
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t src = (code >> (4 * k)) & 15u;
        if (src == kRowOwn || src == kRowNone) continue;
        for (int v = 0; v < S; ++v) CAG_PUT(k, v, src == kRowCache ? *cache_at(a, v, sl) : CAG(src, v));
        code = (code & ~(15u << (4 * k))) | (kRowOwn << (4 * k));
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) __stcs(&a.cand_pos[(size_t)k * sl.nh + sl.hc], pos[k]);
    __stcs(&a.cand_flags[sl.hc], code);
}

/* WW: pixels of one colour per warp row (the half-step tile, tuned per view
 * size by the batched form; 8 elsewhere) */
template <int WW, int NW>
__global__ void __launch_bounds__(kBlockX *NW, NW == kBlockY ? HPM_P1_MIN_BLOCKS : kWideWarps / NW)
    k_prop_dirs(const __grid_constant__ PMArgs a, int iter, int color)
{
    __shared__ PatchMem<WW> sPatch;
    __shared__ DirItems sItems;
    prop_dirs_body<WW, NW>(a, iter, sPatch.template load<NW>(a, color), sItems);
}

/* What the selection hands to the refinement, per pixel (rf_* in PMArgs):
 * plane and (cost, its depth, its restricted cost, the current hypothesis's
 * cost) after the neighbours, the view weights (at most 15 draws, 4 bits per
 * view) and the row of the cost vector that belongs to the plane.
 * ACMM: the ACMM+NESP variant (ACMM.cu:1548-1629): geometric weight 0.2 on
 * the current hypothesis, no NaN fallback.  A separate instantiation. */
constexpr int kRowCurrent = 15;
constexpr int kViewDraws = 15; /* HPM.cu:1590 */

/* weight of view v: 4 bits each, 16 views per word */
__device__ __forceinline__ float view_weight(unsigned long long lo, unsigned long long hi, int v)
{
    return (float)((v < 16 ? lo >> (4 * v) : hi >> (4 * (v - 16))) & 15ull);
}

template <int SMAX, bool ACMM>
__device__ __forceinline__ void prop_select_body(const PMArgs &a, int iter, int px, int py)
{
    constexpr float kGeomW = ACMM ? 0.2f : 0.1f; /* HPM.cu:1642; ACMM.cu:1596 */
    if (px >= a.W || py >= a.rows_cov) return;
    const int W = a.W, S = a.n - 1;
    const int center = py * W + px;
    const Slot sl = slot_of(a, px, py);
    const HpmCamera &cam = a.cam[0];
    const uint32_t code = a.cand_flags[sl.hc];
    uint32_t flags = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (dir_valid(code, k)) flags |= 1u << k;
    int pos[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) pos[k] = a.cand_pos[(size_t)k * sl.nh + sl.hc];
#define FLAG(k) (((flags >> (k)) & 1u) != 0)
/* cost of direction k for view v: every valid direction owns its row (step
 * 3 of prop_dirs_body); an invalid one holds the reference's {2, 0, ...}
 * (HPM.cu:1244), or 2 everywhere with fix_quirks */
#define ROWC(k, v) (FLAG(k) ? CAG(k, v) : ((a.fix_quirks || ((k) == 0 && (v) == 0)) ? 2.0f : 0.0f))
    Rng rng;
    rng.init(a.seed_lo, a.seed_hi, (uint32_t)center, (uint32_t)(1 + iter), a.salt);

    /* Multi-hypothesis joint view selection, HPM.cu:1548-1613. */
    float vw[SMAX];
    float sp[SMAX];
    const uint32_t nbm[4] = {FLAG(1) ? a.views[center - W * 5] : 0u, FLAG(3) ? a.views[center + W * 5] : 0u,
                             FLAG(5) ? a.views[center - 5] : 0u, FLAG(7) ? a.views[center + 5] : 0u};
    const float thr = (float)(0.8 * expf((float)(iter * iter) / (-90.0f)));
    /* the kernel waits for the rows, so a view's are loaded while the view
     * before it is judged (0.47 -> 0.43 ms at 1600x1200, 10 sources) */
    float next[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) next[k] = ROWC(k, 0);
#pragma unroll
    for (int v = 0; v < SMAX; ++v) {
        float row[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            row[k] = next[k];
            if (v + 1 < S) next[k] = ROWC(k, v + 1);
        }
        vw[v] = 0.0f;
        sp[v] = 0.0f;
        if (v >= S) continue;
        float prior = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (FLAG(2 * i + 1)) prior += ((nbm[i] >> v) & 1u) ? 0.9f : 0.1f;
        float count = 0;
        int count_false = 0;
        float tmpw = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float c = row[k];
            if (c < thr) {
                tmpw += expf(c * c / (-0.18f));
                count++;
            }
            if (c > 1.2f) count_false++;
        }
        float p = 0.0f;
        if (count > 2 && count_false < 3)
            p = tmpw / count;
        else if (count_false < 3)
            p = expf(thr * thr / (-0.32f));
        sp[v] = p * prior;
    }
    {
        float s = 0.0f;
#pragma unroll
        for (int v = 0; v < SMAX; ++v)
            if (v < S) s += sp[v];
        const float inv = 1.0f / s;
        float cum = 0.0f;
#pragma unroll
        for (int v = 0; v < SMAX; ++v)
            if (v < S) {
                cum += sp[v] * inv;
                sp[v] = cum;
            }
    }
    for (int smp = 0; smp < kViewDraws; ++smp) {
        const float rp = rng.uniform() - FLT_EPSILON;
        bool done = false;
#pragma unroll
        for (int v = 0; v < SMAX; ++v) {
            if (!done && v < S && sp[v] > rp) {
                vw[v] += 1.0f;
                done = true;
            }
        }
    }
    float wn = 0.0f;
    /* the integer view weights, 4 bits per view (at most 15 draws), for
     * loops over the selected views with a run-time index */
    unsigned long long vw_lo = 0, vw_hi = 0;
#pragma unroll
    for (int v = 0; v < SMAX; ++v)
        if (v < S && vw[v] > 0) {
            wn += vw[v];
            if (v < 16)
                vw_lo |= (unsigned long long)vw[v] << (4 * v);
            else
                vw_hi |= (unsigned long long)vw[v] << (4 * (v - 16));
        }

    /* candidates' costs, and the current hypothesis's (HPM.cu:1637-1650) from
     * the cost-vector cache */
    const float4 cur = a.planes[center];
    float fc[8], cost_now = 0.0f;
    if (a.geom) {
        /* view by view, three planes' source depths on their way at a time;
         * one plane after the other over all views the kernel waited for each
         * (1600x1200, 10 sources: 2.05 against 0.69 ms) */
        float P[9][3], f[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            geom_point(a, k < 8 && FLAG(k) ? a.planes[pos[k]] : cur, px, py, P[k]);
            f[k] = 0.0f;
        }
#pragma unroll 1
        for (int v = 0; v < S; ++v) {
            const float w = view_weight(vw_lo, vw_hi, v);
            if (!(w > 0.0f)) continue;
#pragma unroll
            for (int b = 0; b < 9; b += 3) {
                float spt[3][2], d[3], row[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    d[i] = geom_source(a, v + 1, P[b + i], spt[i]);
                    row[i] = b + i < 8 ? ROWC(b + i, v) : *cache_at(a, v, sl);
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int k = b + i;
                    const float g = geom_distance(a, v + 1, px, py, spt[i], d[i]);
                    const float c = k == 8 ? __fmaf_rn(kGeomW, g, row[i])
                                           : (FLAG(k) ? __fmaf_rn(0.1f, g, row[i]) : row[i] + 0.1f * 5.0f);
                    f[k] = __fmaf_rn(w, c, f[k]);
                }
            }
            count_geom(a, __popc(flags) + 1);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) fc[k] = f[k] / wn;
        cost_now = f[8];
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) fc[k] = 0.0f;
        /* view by view, its nine costs on their way together and the views of
         * zero weight left out whole; candidate by candidate each view's load
         * stood behind a branch of its own (0.43 -> 0.28 ms) */
#pragma unroll 1
        for (int v = 0; v < S; ++v) {
            const float w = view_weight(vw_lo, vw_hi, v);
            if (!(w > 0.0f)) continue;
            float row[9];
#pragma unroll
            for (int k = 0; k < 8; ++k) row[k] = ROWC(k, v);
            row[8] = *cache_at(a, v, sl);
#pragma unroll
            for (int k = 0; k < 8; ++k) fc[k] = __fmaf_rn(w, row[k], fc[k]);
            cost_now = __fmaf_rn(w, row[8], cost_now);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) fc[k] /= wn;
    }
    cost_now /= wn;
    int min_idx = 0;
    {
        float m = fc[0];
#pragma unroll
        for (int k = 1; k < 8; ++k)
            if (fc[k] <= m) {
                m = fc[k];
                min_idx = k;
            }
    }

    float4 plane = cur;
    int best_row = -1; /* -1: the cached current hypothesis */
    float cost = cost_now;
    bool sel_new = false; /* the selected views change to the weighted ones */
    float depth_now = depth_from_plane(cam, plane, px, py);

    float restricted_cost = 0.0f;
    if (a.prior) {
        const float depth_sigma = (a.dmax - a.dmin) / 64.0f;
        const float two_dss = 2 * depth_sigma * depth_sigma;
        const float angle_sigma = (float)(kPiD * (5.0f / 180.0f));
        const float two_ass = 2 * angle_sigma * angle_sigma;
        const float4 pp = a.prior_planes[center];
        const float depth_prior = depth_from_plane(cam, pp, px, py);
        const float beta = 0.18f;
        if (a.masks[center] > 0) {
            float rfc[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                rfc[k] = 0.0f;
                if (FLAG(k)) {
                    const float4 hq = a.planes[pos[k]];
                    const float dn = depth_from_plane(cam, hq, px, py);
                    const float pr = restricted_prior(dn - depth_prior, dot3(pp, hq), two_dss, two_ass);
                    rfc[k] = expf(-fc[k] * fc[k] / beta) * pr;
                }
            }
            int max_idx = 0;
            {
                float m = rfc[0];
#pragma unroll
                for (int k = 1; k < 8; ++k)
                    if (rfc[k] >= m) {
                        m = rfc[k];
                        max_idx = k;
                    }
            }
            const float dn = depth_from_plane(cam, plane, px, py);
            const float pr = restricted_prior(dn - depth_prior, dot3(pp, plane), two_dss, two_ass);
            const float rcn = expf(-cost_now * cost_now / beta) * pr;
            if (FLAG(max_idx)) {
                const float4 hb = a.planes[pos[max_idx]];
                const float db = depth_from_plane(cam, hb, px, py);
                if (db >= a.dmin && db <= a.dmax && rfc[max_idx] > rcn) {
                    depth_now = db;
                    plane = hb;
                    best_row = max_idx;
                    cost = fc[max_idx];
                    restricted_cost = rfc[max_idx];
                    sel_new = true;
                }
            }
        } else if (FLAG(min_idx)) {
            const float4 hb = a.planes[pos[min_idx]];
            const float db = depth_from_plane(cam, hb, px, py);
            if (db >= a.dmin && db <= a.dmax && fc[min_idx] < cost_now) {
                depth_now = db;
                plane = hb;
                best_row = min_idx;
                cost = fc[min_idx];
            }
        }
    }
    if (!a.prior && FLAG(min_idx)) {
        const float4 hb = a.planes[pos[min_idx]];
        const float db = depth_from_plane(cam, hb, px, py);
        if (db >= a.dmin && db <= a.dmax && fc[min_idx] < cost_now) {
            depth_now = db;
            plane = hb;
            best_row = min_idx;
            cost = fc[min_idx];
            sel_new = true;
        }
        if (!ACMM && cost != cost) { /* the ACMM+NESP variant has no such fallback */
            depth_now = db;
            plane = hb;
            best_row = min_idx;
            sel_new = true;
        }
    }

    a.rf_plane[sl.hc] = plane;
    a.rf_state[sl.hc] = make_float4(cost, depth_now, restricted_cost, cost_now);
    uint32_t *weights = a.rf_views + (size_t)sl.hc * (SMAX > 16 ? 4 : 2);
    weights[0] = (uint32_t)vw_lo;
    weights[1] = (uint32_t)(vw_lo >> 32);
    if constexpr (SMAX > 16) {
        weights[2] = (uint32_t)vw_hi;
        weights[3] = (uint32_t)(vw_hi >> 32);
    }
    /* the direction's flags are read for the last time above */
    a.cand_flags[sl.hc] = (uint32_t)(best_row < 0 ? kRowCurrent : best_row) | (sel_new ? 16u : 0u);
#undef ROWC
#undef FLAG
}

template <int SMAX, int WW, bool ACMM>
__global__ void __launch_bounds__(kBlock, HPM_P3_MIN_BLOCKS) k_prop_select(const __grid_constant__ PMArgs a, int iter, int color)
{
    int px, py;
    half_step_pixel_at(blockIdx.x, blockIdx.y, WW, color, px, py);
    prop_select_body<SMAX, ACMM>(a, iter, px, py);
}

/* Shared memory of the refinement, per owner warp: its pixels' candidate
 * planes and the weighted sums of their costs; per block, the pixels whose
 * winner's cost vector is not complete yet. */
template <int NC, int NW>
struct RefineItems {
    float4 cand[kBlockY][NC][32];
    float cost[kBlockY][NC][32];
    uint8_t rank[NW][kBlock];
    uint32_t missing[kBlock];
};

/* With more warps than owners also the windows' statistics, the pixels that
 * weigh each view, and (dynamic) each candidate's cost in each
 * view, which the owners sum in the views' order. */
struct RefineShare {
    RefStats stats[kBlock];
    uint8_t rank[kBlockY][kMaxSrc][32];
    uint8_t count[kBlockY][kMaxSrc];
};

/* PROP: the prior-net form, whose network proposal a.proposals[center] is a
 * sixth refinement candidate, scored by the same NCC (and prior terms) as the
 * other five and accepted by the same rule.  It takes no random draws, so
 * the random stream of the other candidates is unchanged.
 * ACMM: the ACMM+NESP variant (ACMM.cu:623-667): geometric weight 0.2 on the
 * refined hypotheses, and in a hierarchy pass the threshold rule on the
 * result.  A separate instantiation. */
template <bool PROP, bool ACMM, int WW, int NW>
__device__ __forceinline__ void prop_refine_body(const PMArgs &a, int iter, const Patch<WW> &patch,
                                                 RefineItems<PROP ? 6 : 5, NW> &items, RefineShare *share,
                                                 float *costs)
{
    constexpr float kGeomW = ACMM ? 0.2f : 0.1f; /* HPM.cu:1189; ACMM.cu:651 */
    constexpr int NC = PROP ? 6 : 5;
    const int W = a.W, S = a.n - 1;
    /* the first two warps own the block's pixels, others only score */
    const int lane = threadIdx.x, wv = threadIdx.y & 1, q0 = wv * kBlockX;
    const bool owner = NW == kBlockY || threadIdx.y < kBlockY;
    int px = patch.x(q0 + lane), py = patch.y(q0 + lane);
    const bool act = owner && px < W && py < a.rows_cov;
    /* lanes outside the image (and warps that own none) stay for the block's
     * windows, on a pixel inside, with no view weight and no write */
    px = min(px, W - 1);
    py = min(py, a.H - 1);
    const int center = py * W + px;
    const Slot sl = slot_of(a, px, py);
    const HpmCamera &cam = a.cam[0];
    /* PlaneHypothesisRefinement, HPM.cu:1143-1220 */
    RefStats rs = {0.0f, 0.0f, 0.0f};
    if (owner) rs = ref_window(patch.win(q0 + lane));
    float4 plane = a.rf_plane[sl.hc];
    const float4 state = a.rf_state[sl.hc];
    float cost = state.x, depth_now = state.y, restricted_cost = state.z;
    const uint32_t row_code = a.cand_flags[sl.hc];
    int best_row = (int)(row_code & 15u); /* kRowCurrent: the cached current hypothesis */
    unsigned long long vw_lo = 0, vw_hi = 0;
    if (act) {
        const uint32_t *weights = a.rf_views + (size_t)sl.hc * (S > 16 ? 4 : 2);
        vw_lo = weights[0] | (unsigned long long)weights[1] << 32;
        if (S > 16) vw_hi = weights[2] | (unsigned long long)weights[3] << 32;
    }
    /* the selected views and the sum of their (integer) weights */
    uint32_t tsv = 0;
    float wn = 0.0f;
    for (int v = 0; v < S; ++v) {
        const float w = view_weight(vw_lo, vw_hi, v);
        if (w > 0) tsv |= 1u << v;
        wn += w;
    }
    Rng rng;
    rng.resume(a.seed_lo, a.seed_hi, (uint32_t)center, (uint32_t)(1 + iter), a.salt, kViewDraws);
    {
        const float pert = 0.02f;
        const float depth_sigma = (a.dmax - a.dmin) / 64.0f;
        const float two_dss = 2 * depth_sigma * depth_sigma;
        const float angle_sigma = (float)(kPiD * (5.0f / 180.0f));
        const float two_ass = 2 * angle_sigma * angle_sigma;
        const float beta = 0.18f;
        float depth_prior = 0.0f;
        const bool use_prior = a.prior && a.masks[center] > 0;
        float4 pp = make_float4(0, 0, 0, 0);
        float depth_rand;
        float4 n_rand;
        if (use_prior) {
            pp = a.prior_planes[center];
            depth_prior = depth_from_plane(cam, pp, px, py);
            depth_rand = rng.uniform() * 6 * depth_sigma + (depth_prior - 3 * depth_sigma);
            n_rand = perturbed_normal(cam, px, py, pp, rng, angle_sigma);
        } else {
            depth_rand = rng.uniform() * (a.dmax - a.dmin) + a.dmin;
            n_rand = random_normal(cam, px, py, rng, depth_now);
        }
        const float lo = (1 - pert) * depth_now, hi = (1 + pert) * depth_now;
        float depth_pert = rng.uniform() * (hi - lo) + lo;
        /* do { ... } while (d < min && d > max) never repeats (HPM.cu:1170-1172);
         * with fix_quirks the draw repeats while out of range, at most 8 times */
        for (int t = 1; a.fix_quirks && t < 8 && (depth_pert < a.dmin || depth_pert > a.dmax); ++t)
            depth_pert = rng.uniform() * (hi - lo) + lo;
        const float4 n_pert = perturbed_normal(cam, px, py, plane, rng, (float)(pert * kPiD));
        const float depths[5] = {depth_rand, depth_now, depth_rand, depth_now, depth_pert};
        const float4 normals[5] = {plane, n_rand, n_rand, n_pert, plane};
        /* The five candidates are built before any is scored (HPM.cu:1180-
         * 1183), so they are scored view by view with the view index uniform
         * across the warp (one source texture per texture instruction, one
         * source image at a time per block); each NCC value goes to the
         * candidate's hand-off row for the cache. */
        float cand_depth[NC];
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            float4 c = normals[i];
            c.w = distance_to_origin(cam, px, py, depths[i], c);
            if (owner) items.cand[wv][i][lane] = c;
            cand_depth[i] = depths[i];
        }
        if constexpr (PROP) {
            const float4 c = a.proposals[center];
            if (owner) items.cand[wv][5][lane] = c;
            cand_depth[5] = depth_from_plane(cam, c, px, py);
        }
        /* one window: its cost into the hand-off row; with the geometric term */
        auto score = [&](int v, int i, int q, bool need, const RefStats &st) -> float {
            const float4 h = items.cand[q >> 5][i][q & 31];
            const int qx = patch.x(q), qy = patch.y(q);
            /* the geometric term's source depth comes in under the window */
            float spt[2], depth = 0.0f;
            if (a.geom && need) {
                float P[3];
                geom_point(a, h, qx, qy, P);
                depth = geom_source(a, v + 1, P, spt);
            }
            float c = ncc_quad(a, v + 1, qx, qy, need, h, patch.win(q), st);
            if (need) {
                __stcs(&a.cand_costs[(size_t)((kRefineRow + i) * S + v) * sl.nh + ((qy * W + qx) >> 1)], c);
                if (a.geom) {
                    c = __fmaf_rn(kGeomW, geom_distance(a, v + 1, qx, qy, spt, depth), c);
                    count_geom(a, 1);
                }
            }
            return c;
        };
        /* the candidates of the pixels that weigh a view, packed: a pixel's
         * together, candidates 0 and 2 (which share the random depth, hence
         * the window centre) and 1, 3, 4 (at or near the current depth) next
         * to each other, so that windows with the same centre meet in the
         * texture cache */
        if constexpr (NW == kBlockY) {
#pragma unroll
            for (int i = 0; i < NC; ++i) items.cost[wv][i][lane] = 0.0f;
#pragma unroll 1
            for (int v = 0; v < S; ++v) {
                const float weight = view_weight(vw_lo, vw_hi, v);
                const bool selected = weight > 0.0f;
                const unsigned m = __ballot_sync(kAll, selected);
                if (m == 0) continue;
                const int total = __popc(m) * NC;
                if (selected) items.rank[wv][__popc(m & lanes_below())] = (uint8_t)lane;
                __syncwarp();
#pragma unroll 1
                for (int base = 0; base < total; base += 32) {
                    const bool need = base + lane < total;
                    const int j = need ? base + lane : 0, n = j / NC, p = items.rank[wv][n];
                    const int i = (0x543120 >> (4 * (j - n * NC))) & 15;
                    const RefStats st = stats_of(rs, p);
                    const float w = __shfl_sync(kAll, weight, p);
                    const float c = score(v, i, q0 + p, need, st);
                    if (need) items.cost[wv][i][p] = __fmaf_rn(w, c, items.cost[wv][i][p]);
                }
                __syncwarp();
            }
        } else {
            if (owner) {
                share->stats[q0 + lane] = rs;
                for (int v = 0; v < S; ++v) {
                    const bool selected = (tsv >> v) & 1u;
                    const unsigned m = __ballot_sync(kAll, selected);
                    if (selected) share->rank[wv][v][__popc(m & lanes_below())] = (uint8_t)lane;
                    if (lane == 0) share->count[wv][v] = (uint8_t)__popc(m);
                }
            }
            __syncthreads();
#pragma unroll 1
            for (int v = threadIdx.y / kBlockY; v < S; v += NW / kBlockY) {
                const int total = share->count[wv][v] * NC;
#pragma unroll 1
                for (int base = 0; base < total; base += 32) {
                    const bool need = base + lane < total;
                    const int j = need ? base + lane : 0, n = j / NC, q = q0 + share->rank[wv][v][n];
                    const int i = (0x543120 >> (4 * (j - n * NC))) & 15;
                    const float c = score(v, i, q, need, share->stats[q]);
                    if (need) costs[(v * NC + i) * kBlock + q] = c;
                }
            }
            __syncthreads();
            if (owner) {
#pragma unroll
                for (int i = 0; i < NC; ++i) {
                    float sum = 0.0f;
                    for (int v = 0; v < S; ++v)
                        if ((tsv >> v) & 1u)
                            sum = __fmaf_rn(view_weight(vw_lo, vw_hi, v), costs[(v * NC + i) * kBlock + q0 + lane], sum);
                    items.cost[wv][i][lane] = sum;
                }
            }
        }
        if (a.counters && tsv) atomicAdd(&a.counters[0], (unsigned long long)(NC * __popc(tsv)));
        /* by the owners alone: they write their sums without another barrier */
#pragma unroll
        for (int i = 0; owner && i < NC; ++i) {
            const float tci = items.cost[wv][i][lane] / wn;
            const float4 ci = items.cand[wv][i][lane];
            const float depth_before = depth_from_plane(cam, ci, px, py);
            bool take;
            if (use_prior) {
                const float dd = cand_depth[i] - depth_prior;
                const float pr = restricted_prior(dd, dot3(pp, ci), two_dss, two_ass);
                const float rtc = expf(-tci * tci / beta) * pr;
                take = depth_before >= a.dmin && depth_before <= a.dmax && rtc > restricted_cost;
                if (take) restricted_cost = rtc;
            } else {
                take = depth_before >= a.dmin && depth_before <= a.dmax && tci < cost;
            }
            if (take) {
                depth_now = depth_before;
                plane = ci;
                cost = tci;
                best_row = kRefineRow + i;
            }
        }
    }
    /* ACMM+NESP hierarchy pass (ACMM.cu:1617-1624): the update is kept only
     * where it beats the threshold by 0.1; otherwise the pixel keeps its
     * plane with the current hypothesis's cost under this half-step's view
     * weights (its selected views may still have changed) */
    if constexpr (ACMM) {
        if (a.pre_costs && !(cost < a.pre_costs[center] - 0.1f)) {
            plane = a.planes[center];
            cost = state.w;
            best_row = kRowCurrent;
        }
    }
    /* the winner's cost vector for the cache: the views without a weight have
     * not been scored for the refinement candidates.  They are few, so both
     * warps' are packed together, and the views dealt out to the warps. */
    const bool took = act && best_row >= kRefineRow && best_row != kRowCurrent;
    const uint32_t all = S == 32 ? kAll : (1u << S) - 1u;
    __syncthreads();
    if (owner) {
        items.cand[wv][0][lane] = plane;
        items.cost[wv][0][lane] = rs.inv;
        items.cost[wv][1][lane] = rs.mean;
        items.cost[wv][2][lane] = rs.var;
        items.missing[q0 + lane] = took ? all & ~tsv : 0u;
    }
    __syncthreads();
#pragma unroll 1
    for (int v = threadIdx.y; v < S; v += NW) {
        int total = 0;
#pragma unroll
        for (int half = 0; half < kBlockY; ++half) {
            const bool mine = (items.missing[half * kBlockX + lane] >> v) & 1u;
            const unsigned m = __ballot_sync(kAll, mine);
            if (mine) items.rank[threadIdx.y][total + __popc(m & lanes_below())] = (uint8_t)(half * kBlockX + lane);
            total += __popc(m);
        }
        __syncwarp();
#pragma unroll 1
        for (int base = 0; base < total; base += 32) {
            const bool need = base + lane < total;
            const int q = need ? items.rank[threadIdx.y][base + lane] : 0, qw = q >> 5, p = q & 31;
            const RefStats st = {items.cost[qw][0][p], items.cost[qw][1][p], items.cost[qw][2][p]};
            const int qx = patch.x(q), qy = patch.y(q);
            const float c = ncc_quad(a, v + 1, qx, qy, need, items.cand[qw][0][p], patch.win(q), st);
            if (need) *cache_at(a, v, slot_of(a, qx, qy)) = c;
        }
        __syncwarp();
    }
    if (a.counters && took) atomicAdd(&a.counters[0], (unsigned long long)(S - __popc(tsv)));
    if (!act) return;
    a.planes[center] = plane;
    a.costs[center] = cost;
    if (row_code & 16u) a.views[center] = tsv;
    if (best_row == kRowCurrent) return;
    for (int v = 0; v < S; ++v)
        if (!took || ((tsv >> v) & 1u)) *cache_at(a, v, sl) = CAG(best_row, v);
}

template <bool PROP, int WW, bool ACMM, int NW>
__global__ void __launch_bounds__(kBlockX *NW, NW == kBlockY ? HPM_P2_MIN_BLOCKS : kWideWarps / NW)
    k_prop_refine(const __grid_constant__ PMArgs a, int iter, int color)
{
    __shared__ PatchMem<WW> sPatch;
    __shared__ RefineItems<PROP ? 6 : 5, NW> sItems;
    const Patch<WW> patch = sPatch.template load<NW>(a, color);
    if constexpr (NW == kBlockY) {
        prop_refine_body<PROP, ACMM, WW, NW>(a, iter, patch, sItems, nullptr, nullptr);
    } else {
        __shared__ RefineShare sShare;
        extern __shared__ float sCosts[]; /* [S][candidates][kBlock] */
        prop_refine_body<PROP, ACMM, WW, NW>(a, iter, patch, sItems, &sShare, sCosts);
    }
}
#undef CAG_PUT
#undef CAG

/* GetDepthandNormal, HPM.cu:1751-1764 */
__global__ void k_depth_normal(const __grid_constant__ PMArgs a, float4 *planes)
{
    const int px = blockIdx.x * blockDim.x + threadIdx.x;
    const int py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= a.W || py >= a.H) return;
    const int c = py * a.W + px;
    float4 h = planes[c];
    h.w = depth_from_plane(a.cam[0], h, px, py);
    planes[c] = transform_normal(a.cam[0], h);
}

/* Moves the least of x[0 .. K-1] to x[0] and the greatest to x[K-1]. */
template <int K>
__device__ __forceinline__ void ends(float *x)
{
    auto order = [](float &lo, float &hi) {
        const float l = fminf(lo, hi);
        hi = fmaxf(lo, hi);
        lo = l;
    };
#pragma unroll
    for (int i = 0; i < K / 2; ++i) order(x[i], x[K - 1 - i]);
#pragma unroll
    for (int i = 1; i < (K + 1) / 2; ++i) order(x[0], x[i]);
#pragma unroll
    for (int i = K / 2; i < K - 1; ++i) order(x[i], x[K - 1]);
}

/* The median of 21 values by forgetful selection: of any 12 of them neither the least
 * nor the greatest can be the median, so both are dropped and the next value
 * comes in, until three are left.  x is used up. */
template <int K = 12>
__device__ __forceinline__ float median21(float *x, const float *rest)
{
    ends<K>(x);
    if constexpr (K == 3) {
        return x[1];
    } else {
        x[0] = *rest; /* x[K - 1] is left out from here on */
        return median21<K - 1>(x, rest + 1);
    }
}

/* CheckerboardFilter, HPM.cu:1766-1904.  Away from the borders all 21 depths
 * are there and the median is taken in registers; sorting them in a local
 * array was all of the kernel's time (1600x1200, one colour: 173 us, now 43).
 * At the borders, and where a depth is not a number (the sort's order then
 * matters), the reference's sort runs. */
__global__ void k_filter(const __grid_constant__ PMArgs a, float4 *pl, const float *costs, int color)
{
    const int py = blockIdx.y * blockDim.y + threadIdx.y;
    const int px = blockIdx.x * (2 * blockDim.x) + 2 * threadIdx.x + ((py + color) & 1);
    const int W = a.W, H = a.H;
    if (px >= W || py >= a.rows_cov) return;
    const int center = py * W + px;
    if (costs[center] < 0.001f) return;
    if (px > 4 && px < W - 5 && py > 4 && py < H - 5) {
        const float *d = &pl[center].w;
        const int offset[21] = {0,         -W,        -3 * W,     -5 * W,     W,          3 * W,      5 * W,
                                -1,        -3,        -5,         1,          3,          5,          -W + 2,
                                W + 2,     -W - 2,    W - 2,      -1 - 2 * W, 1 - 2 * W,  -1 + 2 * W, 1 + 2 * W};
        float x[21];
        bool numbers = true;
#pragma unroll
        for (int i = 0; i < 21; ++i) x[i] = d[4 * offset[i]];
#pragma unroll
        for (int i = 0; i < 21; ++i) numbers = numbers && x[i] == x[i];
        if (numbers) {
            pl[center].w = median21(x, x + 12);
            return;
        }
    }
    float f[21];
    int n = 0;
    f[n++] = pl[center].w;
    const int left = center - 1, leftleft = center - 3, up = center - W, upup = center - 3 * W;
    const int down = center + W, downdown = center + 3 * W, right = center + 1, rightright = center + 3;
    if (py > 0) f[n++] = pl[up].w;
    if (py > 2) f[n++] = pl[upup].w;
    if (py > 4) f[n++] = pl[upup - W * 2].w;
    if (py < H - 1) f[n++] = pl[down].w;
    if (py < H - 3) f[n++] = pl[downdown].w;
    if (py < H - 5) f[n++] = pl[downdown + W * 2].w;
    if (px > 0) f[n++] = pl[left].w;
    if (px > 2) f[n++] = pl[leftleft].w;
    if (px > 4) f[n++] = pl[leftleft - 2].w;
    if (px < W - 1) f[n++] = pl[right].w;
    if (px < W - 3) f[n++] = pl[rightright].w;
    if (px < W - 5) f[n++] = pl[rightright + 2].w;
    if (py > 0 && px < W - 2) f[n++] = pl[up + 2].w;
    if (py < H - 1 && px < W - 2) f[n++] = pl[down + 2].w;
    if (py > 0 && px > 1) f[n++] = pl[up - 2].w;
    if (py < H - 1 && px > 1) f[n++] = pl[down - 2].w;
    if (px > 0 && py > 2) f[n++] = pl[left - W * 2].w;
    if (px < W - 1 && py > 2) f[n++] = pl[right - W * 2].w;
    if (px > 0 && py < H - 2) f[n++] = pl[left + W * 2].w;
    if (px < W - 1 && py < H - 2) f[n++] = pl[right + W * 2].w;
    sort_small(f, n);
    const int m = n / 2;
    pl[center].w = (n % 2 == 0) ? (f[m - 1] + f[m]) / 2 : f[m];
}

__global__ void __launch_bounds__(kBlock) k_cost_vectors(const __grid_constant__ PMArgs a, const float4 *planes,
                                                          float *out)
{
    __shared__ RowMem sRow;
    const WinRow win = sRow.load(a.view[0], a.sigma_spatial, a.sigma_color);
    const int px = blockIdx.x * kBlockX + threadIdx.x;
    const int py = blockIdx.y * kBlockY + threadIdx.y;
    const bool act = px < a.W && py < a.H;
    const int cx = min(px, a.W - 1), cy = min(py, a.H - 1);
    const RefStats rs = ref_window(win);
    const int c = cy * a.W + cx;
    const int S = a.n - 1;
    cost_vector(a, px, py, act, planes[c], win, rs, out + (size_t)c * S, 1);
}

__global__ void __launch_bounds__(kBlock) k_initial_costs(const __grid_constant__ PMArgs a, const float4 *planes,
                                                          float *cost, uint32_t *views)
{
    __shared__ RowMem sRow;
    const WinRow win = sRow.load(a.view[0], a.sigma_spatial, a.sigma_color);
    __shared__ float sCV[kMaxSrc * kBlock];
    const int tid = threadIdx.y * kBlockX + threadIdx.x;
    const int px = blockIdx.x * kBlockX + threadIdx.x;
    const int py = blockIdx.y * kBlockY + threadIdx.y;
    const bool act = px < a.W && py < a.H;
    const int cx = min(px, a.W - 1), cy = min(py, a.H - 1);
    const RefStats rs = ref_window(win);
    const int c = cy * a.W + cx;
    cost_vector(a, px, py, act, planes[c], win, rs, sCV + tid, kBlock);
    if (act) cost[c] = initial_cost_from(a, sCV + tid, kBlock, &views[c]);
}

__global__ void k_geom_costs(const __grid_constant__ PMArgs a, const float4 *planes, float *out)
{
    const int px = blockIdx.x * blockDim.x + threadIdx.x;
    const int py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= a.W || py >= a.H) return;
    const int c = py * a.W + px;
    const int S = a.n - 1;
    float P[3];
    geom_point(a, planes[c], px, py, P);
    for (int v = 1; v < a.n; ++v) {
        float spt[2];
        const float d = geom_source(a, v, P, spt);
        out[(size_t)c * S + v - 1] = geom_distance(a, v, px, py, spt, d);
        count_geom(a, 1);
    }
}

/* The 36 source samples of the NCC window of listed pixels, per source view
 * (the values ncc_quad weighs), and whether the warped centre is inside. */
__global__ void k_tap_samples(const __grid_constant__ PMArgs a, const float4 *planes, const int *pixels, int n,
                              float *out, int *inside)
{
    const int S = a.n - 1;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n * S) return;
    const int pi = k / S, v = k % S + 1;
    const int px = pixels[pi] % a.W, py = pixels[pi] / a.W;
    const HpmCamera &sc = a.cam[v];
    float H[9];
    homography(a.cam[0], sc, a.pair[v], planes[pixels[pi]], H);
    const float fpx = (float)px, fpy = (float)py;
    const float2 pt = warp(H, fpx, fpy);
    inside[k] = !(pt.x >= sc.width || pt.x < 0.0f || pt.y >= sc.height || pt.y < 0.0f);
#pragma unroll
    for (int tp = 0; tp < 4; ++tp) {
        float s[9];
        fetch_block(a.view[v].tex, H, fpx + (float)(2 * (tp & 1) - 5), fpy + (float)(2 * (tp >> 1) - 5), s);
#pragma unroll
        for (int b = 0; b < 9; ++b)
            out[(size_t)k * kTaps + (2 * (b / 3) + (tp & 1)) * 6 + 2 * (b % 3) + (tp >> 1)] = s[b];
    }
}

template <bool PROP, int WW, bool ACMM, int NW>
cudaError_t launch_refine(const PMArgs &a, int iter, int color, dim3 grid, cudaStream_t s)
{
    size_t bytes = 0;
    if constexpr (NW > kBlockY) {
        constexpr size_t per_source = sizeof(float) * (PROP ? 6 : 5) * kBlock;
        bytes = per_source * (a.n - 1);
        /* the limit belongs to the kernel, not to the launch: the same value
         * for every size, since another thread may launch with more sources */
        const cudaError_t e = cudaFuncSetAttribute(k_prop_refine<PROP, WW, ACMM, NW>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)(per_source * kMaxSrc));
        if (e != cudaSuccess) return e;
    }
    k_prop_refine<PROP, WW, ACMM, NW><<<grid, dim3(kBlockX, NW), bytes, s>>>(a, iter, color);
    return cudaGetLastError();
}

template <int SMAX, int WW, int NW>
cudaError_t launch_prop_t(const PMArgs &a, int iter, int color, dim3 grid, cudaStream_t s)
{
    k_prop_dirs<WW, NW><<<grid, dim3(kBlockX, NW), 0, s>>>(a, iter, color);
    const dim3 b(kBlockX, kBlockY);
    if constexpr (WW == 8) { /* the ACMM+NESP variant runs the default tile */
        if (a.acmm) {
            k_prop_select<SMAX, WW, true><<<grid, b, 0, s>>>(a, iter, color);
            return launch_refine<false, WW, true, NW>(a, iter, color, grid, s);
        }
    }
    k_prop_select<SMAX, WW, false><<<grid, b, 0, s>>>(a, iter, color);
    return a.proposals ? launch_refine<true, WW, false, NW>(a, iter, color, grid, s)
                       : launch_refine<false, WW, false, NW>(a, iter, color, grid, s);
}

/* Warps per block of 64 pixels.  Two where the blocks fill the GPU; on small
 * images, where a block's chain of windows is all there is to wait for, more
 * warps share them: eight while two such blocks per SM hold them (148 SMs),
 * four while four do.  A pass in ms with 2, 4 and 8 warps, by blocks: 54 0.80,
 * 0.58, 0.51; 247 1.85, 1.43, 1.28; 294 1.86, 1.45, 1.30; 345 3.81, 2.96, 3.01;
 * 486 1.29, 1.14, 1.35; 600 2.32, 2.28, 2.39; 950 2.94, 3.62, 4.58.  The blocks
 * of all passes that run at the same time count (a.beside): a batched scene of
 * 12 views of 160x120 (150 blocks each) takes 32.3 ms with eight warps, as one
 * view alone would have them, and 24.4 with two. */
constexpr long long kBlocks8 = 2 * 148, kBlocks4 = 4 * 148;
template <int SMAX, int WW>
cudaError_t launch_prop_n(const PMArgs &a, int iter, int color, cudaStream_t s)
{
    constexpr int WH = 32 / WW;
    const dim3 grid((a.W + 2 * WW - 1) / (2 * WW), (a.rows_cov + 2 * WH - 1) / (2 * WH));
    if constexpr (WW == 8) {
        const long long blocks = (long long)grid.x * grid.y + a.beside / (2 * kBlock);
        if (blocks <= kBlocks8) return launch_prop_t<SMAX, WW, 8>(a, iter, color, grid, s);
        if (blocks <= kBlocks4) return launch_prop_t<SMAX, WW, 4>(a, iter, color, grid, s);
    }
    return launch_prop_t<SMAX, WW, kBlockY>(a, iter, color, grid, s);
}

template <int WW>
cudaError_t launch_prop_w(const PMArgs &a, int iter, int color, cudaStream_t s)
{
    const int S = a.n - 1;
    if (S <= 4) return launch_prop_n<4, WW>(a, iter, color, s);
    if (S <= 8) return launch_prop_n<8, WW>(a, iter, color, s);
    if (S <= 12) return launch_prop_n<12, WW>(a, iter, color, s);
    if (S <= 16) return launch_prop_n<16, WW>(a, iter, color, s);
    return launch_prop_n<kMaxSrc, WW>(a, iter, color, s);
}

}  // namespace

int rows_covered(int H)
{
    const int cov = 2 * (((H / 2) + 15) / 16) * 16;
    return cov < H ? cov : H;
}

cudaError_t launch_pair_geom(const PMArgs &a, PairGeom *out, cudaStream_t s)
{
    k_pair_geom<<<1, 64, 0, s>>>(a, out);
    return cudaGetLastError();
}

static dim3 pixel_grid(int W, int H) { return dim3((W + kBlockX - 1) / kBlockX, (H + kBlockY - 1) / kBlockY); }

cudaError_t launch_init(const PMArgs &a, cudaStream_t s)
{
    k_init<<<pixel_grid(a.W, a.H), dim3(kBlockX, kBlockY), 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_propagate(const PMArgs &a, int iter, int color, cudaStream_t s, int ww)
{
    if (a.rows_cov <= 0) return cudaSuccess;
    if (a.acmm) ww = 8; /* its refinement kernel exists for this tile only */
    switch (ww) {
    case 4: return launch_prop_w<4>(a, iter, color, s);
    case 8: return launch_prop_w<8>(a, iter, color, s);
    case 16: return launch_prop_w<16>(a, iter, color, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_depth_normal_filter(const PMArgs &a, float4 *planes, const float *costs, cudaStream_t s)
{
    dim3 b(16, 16), g((a.W + 15) / 16, (a.H + 15) / 16);
    k_depth_normal<<<g, b, 0, s>>>(a, planes);
    if (a.rows_cov > 0) {
        dim3 fb(32, 8), fg((a.W + 63) / 64, (a.rows_cov + 7) / 8);
        k_filter<<<fg, fb, 0, s>>>(a, planes, costs, 0);
        k_filter<<<fg, fb, 0, s>>>(a, planes, costs, 1);
    }
    return cudaGetLastError();
}

cudaError_t launch_cost_vectors(const PMArgs &a, const float4 *planes, float *out, cudaStream_t s)
{
    k_cost_vectors<<<pixel_grid(a.W, a.H), dim3(kBlockX, kBlockY), 0, s>>>(a, planes, out);
    return cudaGetLastError();
}

cudaError_t launch_initial_costs(const PMArgs &a, const float4 *planes, float *cost, uint32_t *views,
                                 cudaStream_t s)
{
    k_initial_costs<<<pixel_grid(a.W, a.H), dim3(kBlockX, kBlockY), 0, s>>>(a, planes, cost, views);
    return cudaGetLastError();
}

cudaError_t launch_tap_samples(const PMArgs &a, const float4 *planes, const int *pixels, int n, float *out,
                               int *inside, cudaStream_t s)
{
    const int total = n * (a.n - 1);
    if (total > 0) k_tap_samples<<<(total + 127) / 128, 128, 0, s>>>(a, planes, pixels, n, out, inside);
    return cudaGetLastError();
}

cudaError_t launch_geom_costs(const PMArgs &a, const float4 *planes, float *out, cudaStream_t s)
{
    dim3 b(16, 16), g((a.W + 15) / 16, (a.H + 15) / 16);
    k_geom_costs<<<g, b, 0, s>>>(a, planes, out);
    return cudaGetLastError();
}

}  // namespace hpm
