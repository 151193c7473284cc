// imgproc.cu — per-level image preprocessing for the dense tracker.
//
// Reference semantics (paths relative to the reference project root):
//   RGB -> gray            FullSystem/src/System.cpp:47-49 (cv::cvtColor RGB2GRAY): BT.601
//                          luma in 14-bit fixed point, gray = (4899 R + 9617 G + 1868 B
//                          + 8192) >> 14 (0.299/0.587/0.114 scaled by 2^14 and rounded).
//   u16 -> metres          System.cpp:52 (convertTo with the depth scale).
//   intensity pyramid      RGBDTracking.cu:66-116 (cv::cuda::pyrDown: separable
//                          [1 4 6 4 1]/16 Gaussian, reflect-101 border, keep even samples).
//   gradients              ImageProc.cu:7-40: 0.5 * central difference, 0 on the border.
//   inverse depth          ImageProc.cu:141-164: 1/z for 0.2 < z < 8, else 0.
//   nearest pyr-down       ImageProc.cu:166-187: dst(x,y) = src(2x,2y); the reference
//                          leaves the last row and column unwritten, here they are
//                          written as invalid (0 / w = -1).
//   vertex map             ImageProc.cu:189-220: z = 1/invz, valid when invz > 0 and z < 3.
//   normal map             ImageProc.cu:222-260: normalize((v(x,y+1)-v)x(v(x+1,y)-v)),
//                          invalid on the last row/column or when a vertex is invalid.
//   model pyramid          RGBDTracking.cu:140-150 (SetReferenceModel); the reference runs
//                          the float pyr-down on the float4 model (its coarse model levels
//                          are unusable); here the intended float4 nearest pyr-down is used.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "yas_internal.h"
#include "yas_track.h"

namespace yas {

__device__ __forceinline__ int reflect101(int i, int n) {
    if (i < 0) i = -i;
    if (i >= n) i = 2 * (n - 1) - i;
    return i;
}

// Up to three levels of the intensity pyramid, with their gradients, from one
// launch.  A CTA owns 32 x 32 pixels of the first level (16 x 16 of the second,
// 8 x 8 of the third) and computes what their Gaussians and gradients reach in
// shared memory: 49 x 49, 23 x 23 and 10 x 10 pixels.  The levels are too small
// to fill the GPU, and what they cost is their launches, each waiting for the
// one before; next to that the halo's arithmetic is cheap (2.3 and 2.1 times
// the pixels, but a column sum is made once instead of once per tap).
// The vertical 5-tap sums come first, then the horizontal ones; one rounding per
// operation, fixed order: the stored pyramid is bit-identical to the CPU
// restatement's.
// kSource: bytes per pixel of the source (1 gray, 3 RGB, converted; the source
// is level 0, stored with its gradients), or 0 for a level stored before.
// kQuads: four pixels a load and a store, for images whose width, source pitch
// and source address are multiples of 4 (a quad is then inside or outside).
// Calls one after another, three levels, a launch per level and gradient before
// and this: 320x240 20.5 / 6.2 us (the call's own cost), 640x480 20.5 / 6.2
// (pixel by pixel 8.2), 1280x720 24.9 / 10.3 (12.3); five levels 36.9 / 12.3.
struct ImagePyramid {
    const void *src;
    int pitch;  // bytes
    int n;      // levels, the first one included
    int w[3], h[3];
    float *inten[3], *gx[3], *gy[3];  // no gradients where gx is null
};

constexpr int kPyrTile = 32;
// rows and columns in front of the tile, rows and row lengths (even: column
// sums are made in pairs; the first level's columns by quads)
__host__ __device__ constexpr int pyr_halo_y(int l) { return l == 0 ? 10 : (l == 1 ? 4 : 1); }
__host__ __device__ constexpr int pyr_halo_x(int l) { return l == 0 ? 12 : (l == 1 ? 4 : 1); }
__host__ __device__ constexpr int pyr_rows(int l) { return l == 0 ? 49 : (l == 1 ? 23 : 10); }
__host__ __device__ constexpr int pyr_cols(int l) { return l == 0 ? 52 : (l == 1 ? 24 : 10); }
template <int l>
using PyrRegion = float[pyr_rows(l)][pyr_cols(l)];

__device__ __forceinline__ float luma(unsigned r, unsigned g, unsigned b) {
    return (float)((int)(r * 4899u + g * 9617u + b * 1868u + 8192u) >> 14);
}

template <int kSource>
__device__ __forceinline__ float source_value(const ImagePyramid &p, int x, int y) {
    if (kSource == 0) return __ldg(reinterpret_cast<const float *>(static_cast<const char *>(p.src) + (size_t)y * p.pitch) + x);
    const uint8_t *q = static_cast<const uint8_t *>(p.src) + (size_t)y * p.pitch + x * kSource;
    return kSource == 1 ? (float)__ldg(q) : luma(__ldg(q), __ldg(q + 1), __ldg(q + 2));
}

template <int kSource>
__device__ __forceinline__ float4 source_quad(const ImagePyramid &p, int x, int y) {
    const uint8_t *q = static_cast<const uint8_t *>(p.src) + (size_t)y * p.pitch + x * kSource;
    const unsigned *u = reinterpret_cast<const unsigned *>(q);
    const unsigned a = __ldg(u);
    if (kSource == 1)
        return make_float4((float)(a & 255u), (float)((a >> 8) & 255u), (float)((a >> 16) & 255u), (float)(a >> 24));
    const unsigned b = __ldg(u + 1), c = __ldg(u + 2);
    return make_float4(luma(a & 255u, (a >> 8) & 255u, (a >> 16) & 255u),
                       luma(a >> 24, b & 255u, (b >> 8) & 255u),
                       luma((b >> 16) & 255u, b >> 24, c & 255u),
                       luma((c >> 8) & 255u, (c >> 16) & 255u, c >> 24));
}

__device__ __forceinline__ float half_step(float a, float b, bool inner) { return inner ? (b - a) * 0.5f : 0.0f; }

// Level l of the CTA's tile from shared memory to the images.
template <int l>
__device__ __forceinline__ void store_level(const ImagePyramid &p, const PyrRegion<l> &g) {
    constexpr int T = kPyrTile >> l;
    const int w = p.w[l], h = p.h[l];
    for (int i = threadIdx.x; i < T * T; i += blockDim.x) {
        const int lx = i % T, ly = i / T, x = blockIdx.x * T + lx, y = blockIdx.y * T + ly;
        if (x >= w || y >= h) continue;
        const int r = ly + pyr_halo_y(l), c = lx + pyr_halo_x(l), k = y * w + x;
        p.inten[l][k] = g[r][c];
        if (!p.gx[l]) continue;
        const bool inner = x >= 1 && y >= 1 && x <= w - 2 && y <= h - 2;
        p.gx[l][k] = half_step(g[r][c - 1], g[r][c + 1], inner);
        p.gy[l][k] = half_step(g[r - 1][c], g[r + 1][c], inner);
    }
}

// The first level's, a quad per thread.
__device__ __forceinline__ void store_quads(const ImagePyramid &p, const PyrRegion<0> &g) {
    const int w = p.w[0], h = p.h[0], lx = 4 * (threadIdx.x & 7), ly = threadIdx.x >> 3;
    const int x = blockIdx.x * kPyrTile + lx, y = blockIdx.y * kPyrTile + ly;
    if (x >= w || y >= h) return;
    const int r = ly + pyr_halo_y(0), c = lx + pyr_halo_x(0), k = y * w + x;
    const float4 v = *reinterpret_cast<const float4 *>(&g[r][c]);
    *reinterpret_cast<float4 *>(p.inten[0] + k) = v;
    if (!p.gx[0]) return;
    const bool row = y >= 1 && y <= h - 2, first = row && x >= 1, last = row && x + 3 <= w - 2;
    const float4 u = *reinterpret_cast<const float4 *>(&g[r - 1][c]), d = *reinterpret_cast<const float4 *>(&g[r + 1][c]);
    *reinterpret_cast<float4 *>(p.gx[0] + k) = make_float4(half_step(g[r][c - 1], v.y, first), half_step(v.x, v.z, row),
                                                           half_step(v.y, v.w, row), half_step(v.z, g[r][c + 4], last));
    *reinterpret_cast<float4 *>(p.gy[0] + k) = make_float4(half_step(u.x, d.x, first), half_step(u.y, d.y, row),
                                                           half_step(u.z, d.z, row), half_step(u.w, d.w, last));
}

// [1 4 6 4 1] / 16: the products with powers of two are exact, so their fused
// sums round once as separate ones do.
__device__ __forceinline__ float five_taps(float a, float b, float c, float d, float e) {
    const float s = __fadd_rn(__fmaf_rn(0.25f, b, 0.0625f * a), __fmul_rn(0.375f, c));
    return __fmaf_rn(0.0625f, e, __fmaf_rn(0.25f, d, s));
}

// Level l from level l - 1, a row per warp: the row's column sums (of columns
// outside the image too, which nothing reads), then the row.
template <int l>
__device__ __forceinline__ void down_level(const ImagePyramid &p, const PyrRegion<l - 1> &s, PyrRegion<l> &g,
                                           float (*sums)[pyr_cols(0)]) {
    constexpr int R = pyr_rows(l), S = pyr_cols(l - 1), T = kPyrTile >> l;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sx = (int)blockIdx.x * 2 * T - pyr_halo_x(l - 1), sy = (int)blockIdx.y * 2 * T - pyr_halo_y(l - 1);
    const int x = (int)blockIdx.x * T - pyr_halo_x(l) + lane, oy = (int)blockIdx.y * T - pyr_halo_y(l);
    const int sw = p.w[l - 1], sh = p.h[l - 1];
    // a last level is needed one pixel around the tile only
    const int lo = p.n == l + 1 ? pyr_halo_y(l) - 1 : 0, hi = p.n == l + 1 ? pyr_halo_y(l) + T + 1 : R;
    const bool mine = lane >= lo && lane < hi && x >= 0 && x < p.w[l];
    int col[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) col[j] = mine ? reflect101(2 * x + j - 2, sw) - sx : 0;
    for (int r = lo + warp; r < hi; r += 8) {
        const int y = oy + r;
        if (y < 0 || y >= p.h[l]) continue;
        if (2 * lane < S) {
            float2 v[5];
#pragma unroll
            for (int i = 0; i < 5; ++i)
                v[i] = *reinterpret_cast<const float2 *>(&s[reflect101(2 * y + i - 2, sh) - sy][2 * lane]);
            *reinterpret_cast<float2 *>(&sums[warp][2 * lane]) =
                make_float2(five_taps(v[0].x, v[1].x, v[2].x, v[3].x, v[4].x),
                            five_taps(v[0].y, v[1].y, v[2].y, v[3].y, v[4].y));
        }
        __syncwarp();
        if (mine) {
            const float *q = sums[warp];
            g[r][lane] = five_taps(q[col[0]], q[col[1]], q[col[2]], q[col[3]], q[col[4]]);
        }
        __syncwarp();
    }
    __syncthreads();
}

template <int kSource, bool kQuads>
__global__ void __launch_bounds__(256) image_pyramid_kernel(const __grid_constant__ ImagePyramid p) {
    __shared__ __align__(16) PyrRegion<0> g0;
    __shared__ __align__(16) PyrRegion<1> g1;
    __shared__ PyrRegion<2> g2;
    __shared__ __align__(16) float sums[8][pyr_cols(0)];
    const int ox = (int)blockIdx.x * kPyrTile - pyr_halo_x(0), oy = (int)blockIdx.y * kPyrTile - pyr_halo_y(0);
    // rows and columns around the tile that n levels reach: 1, 4 and 3, 10 and 7
    const int before = p.n == 1 ? 1 : (p.n == 2 ? 4 : 10), after = p.n == 1 ? 1 : (p.n == 2 ? 3 : 7);
    const int r0 = pyr_halo_y(0) - before, r1 = pyr_halo_y(0) + kPyrTile + after;
    if constexpr (kQuads) {
        constexpr int Q = pyr_cols(0) / 4;  // quads of a row: two rows a warp
        const int q = threadIdx.x & 15, x = ox + 4 * q;
        const bool in = q < Q && x >= 0 && x < p.w[0];
#pragma unroll
        for (int m = 0; m < (pyr_rows(0) + 15) / 16; ++m) {
            const int r = r0 + (int)(threadIdx.x >> 4) + 16 * m, y = oy + r;
            if (in && r < r1 && y >= 0 && y < p.h[0])
                *reinterpret_cast<float4 *>(&g0[r][4 * q]) = source_quad<kSource>(p, x, y);
        }
    } else {
        const int c0 = pyr_halo_x(0) - before, c1 = pyr_halo_x(0) + kPyrTile + after;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
        for (int m = 0; m < (pyr_rows(0) + 7) / 8; ++m) {
            const int r = r0 + warp + 8 * m, y = oy + r;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int c = c0 + lane + 32 * k, x = ox + c;
                if (r < r1 && c < c1 && x >= 0 && y >= 0 && x < p.w[0] && y < p.h[0])
                    g0[r][c] = source_value<kSource>(p, x, y);
            }
        }
    }
    __syncthreads();
    if constexpr (kSource != 0) {
        if constexpr (kQuads)
            store_quads(p, g0);
        else
            store_level<0>(p, g0);
    }
    if (p.n < 2) return;
    down_level<1>(p, g0, g1, sums);
    store_level<1>(p, g1);
    if (p.n < 3) return;
    down_level<2>(p, g1, g2, sums);
    store_level<2>(p, g2);
}

// The whole intensity pyramid of a gray (channels 1) or RGB (3) byte image:
// three levels a launch, the next ones from the last level stored.
void launch_image_pyramid(const uint8_t *src, int channels, int pitch, int L, const LevelCam *cam,
                          float *const *inten, float *const *gx, float *const *gy, cudaStream_t s) {
    for (int l0 = 0; l0 == 0 || l0 + 1 < L; l0 += 2) {
        ImagePyramid p;
        memset(&p, 0, sizeof(p));
        p.src = l0 == 0 ? (const void *)src : (const void *)inten[l0];
        p.pitch = l0 == 0 ? pitch : cam[l0].w * 4;
        p.n = std::min(3, L - l0);
        for (int i = 0; i < p.n; ++i) {
            p.w[i] = cam[l0 + i].w;
            p.h[i] = cam[l0 + i].h;
            p.inten[i] = inten[l0 + i];
            p.gx[i] = gx ? gx[l0 + i] : nullptr;
            p.gy[i] = gy ? gy[l0 + i] : nullptr;
        }
        const dim3 grid((p.w[0] + kPyrTile - 1) / kPyrTile, (p.h[0] + kPyrTile - 1) / kPyrTile);
        const bool quads = ((p.w[0] | pitch) & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 3u) == 0;
        if (l0 != 0)
            image_pyramid_kernel<0, false><<<grid, 256, 0, s>>>(p);
        else if (channels == 1 && quads)
            image_pyramid_kernel<1, true><<<grid, 256, 0, s>>>(p);
        else if (channels == 1)
            image_pyramid_kernel<1, false><<<grid, 256, 0, s>>>(p);
        else if (quads)
            image_pyramid_kernel<3, true><<<grid, 256, 0, s>>>(p);
        else
            image_pyramid_kernel<3, false><<<grid, 256, 0, s>>>(p);
    }
}

__device__ __forceinline__ float inv_depth_of(float z) {
    return (z > 0.2f && z < 8.0f) ? 1.0f / z : 0.0f;
}

__device__ __forceinline__ float4 vertex_of(float invz, int x, int y, const LevelCam &c) {
    float z = 1.0f / invz;
    if (invz > 0.0f && z < 3.0f)
        return make_float4(z * ((float)x - c.cx) * c.invfx, z * ((float)y - c.cy) * c.invfy, z, 1.0f);
    return make_float4(0.0f, 0.0f, 0.0f, -1.0f);
}

__device__ __forceinline__ float4 normal_of(float4 v00, float4 v01, float4 v10) {
    if (v00.w > 0.0f && v01.w > 0.0f && v10.w > 0.0f) {
        // no contraction: normals (and so their validity and the ICP gates) are
        // bit-identical to the CPU restatement's
        float ax = v10.x - v00.x, ay = v10.y - v00.y, az = v10.z - v00.z;
        float bx = v01.x - v00.x, by = v01.y - v00.y, bz = v01.z - v00.z;
        float nx = __fsub_rn(__fmul_rn(ay, bz), __fmul_rn(az, by));
        float ny = __fsub_rn(__fmul_rn(az, bx), __fmul_rn(ax, bz));
        float nz = __fsub_rn(__fmul_rn(ax, by), __fmul_rn(ay, bx));
        float nn = __fadd_rn(__fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny)), __fmul_rn(nz, nz));
        if (nn > 0.0f) {
            float inv = 1.0f / sqrtf(nn);
            nx *= inv;
            ny *= inv;
            nz *= inv;
        }
        return make_float4(nx, ny, nz, 1.0f);
    }
    return make_float4(0.0f, 0.0f, 0.0f, -1.0f);
}

// Raw depth value at level 0 in metres (u16 * scale, or float).
__device__ __forceinline__ float raw_depth(const void *src, int is_u16, int pitch, float scale, int x, int y) {
    if (is_u16) return (float)reinterpret_cast<const uint16_t *>(static_cast<const char *>(src) + (size_t)y * pitch)[x] * scale;
    return reinterpret_cast<const float *>(static_cast<const char *>(src) + (size_t)y * pitch)[x];
}

// Depth of an inverse depth as the photometric warp uses it (1 / invd, one
// IEEE division), 0 where the inverse depth is invalid.
__device__ __forceinline__ float warp_depth_of(float invz) { return invz > 0.0f ? 1.0f / invz : 0.0f; }

// The whole depth pyramid in one launch: metres (optional), and for every level
// the inverse depth, its reciprocal, the vertex and the normal map.  Level l's
// inverse depth (x, y) of the chained nearest pyr-down is level 0's (2^l x,
// 2^l y) when x < w_l - 1 and y < h_l - 1, and 0 otherwise (the inner levels'
// conditions follow from the outer one), so every level reads the source and
// none waits for another.  A CTA owns 64 x 16 pixels of a level and makes each
// vertex once, for its three normals, in shared memory (65 x 17): divisions
// bound the large images, launches the small ones.  Calls one after another, a
// launch per level and three vertices a normal before and this: 320x240 12.4 /
// 5.9 us, 640x480 15.4 / 8.2, 1280x720 22.6 / 12.4; five levels 23.6 / 8.2.
struct DepthPyramid {
    const void *src;
    int is_u16, pitch, L;
    float scale;
    LevelCam c[kMaxLevels];
    int tiles_x[kMaxLevels], first[kMaxLevels + 1];  // CTAs of the levels laid end to end
    float *depth_m, *invd[kMaxLevels], *zmap[kMaxLevels];
    float4 *vmap[kMaxLevels], *nmap[kMaxLevels];
};

constexpr int kDepthTileX = 64, kDepthTileY = 16;

__global__ void __launch_bounds__(256) depth_pyramid_kernel(const __grid_constant__ DepthPyramid p) {
    __shared__ float4 sv[kDepthTileY + 1][kDepthTileX + 1];
    int l = 0;
    while (l + 1 < p.L && (int)blockIdx.x >= p.first[l + 1]) ++l;
    const LevelCam &c = p.c[l];
    const int b = (int)blockIdx.x - p.first[l], by = b / p.tiles_x[l], bx = b - by * p.tiles_x[l];
    const int x0 = bx * kDepthTileX, y0 = by * kDepthTileY;
    const int xe = l == 0 ? c.w : c.w - 1, ye = l == 0 ? c.h : c.h - 1;
    // a thread's pixels: two rows, two columns; then one of the tile's last row
    // and column of vertices
    const int t = (int)threadIdx.x, warp = t >> 5, lane = t & 31;
    int r[5], cx[5];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        r[q] = warp + 8 * (q >> 1);
        cx[q] = lane + 32 * (q & 1);
    }
    r[4] = t <= kDepthTileX ? kDepthTileY : t - kDepthTileX - 1;
    cx[4] = t <= kDepthTileX ? t : kDepthTileX;
    float z[5];
    float4 v[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const int x = x0 + cx[q], y = y0 + r[q];
        z[q] = r[q] <= kDepthTileY && x < xe && y < ye
                   ? raw_depth(p.src, p.is_u16, p.pitch, p.scale, x << l, y << l)
                   : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const int x = x0 + cx[q], y = y0 + r[q];
        if (q == 4 && t > kDepthTileX + kDepthTileY) break;
        const float iz = inv_depth_of(z[q]);
        v[q] = vertex_of(iz, x, y, c);
        sv[r[q]][cx[q]] = v[q];
        if (q < 4 && x < c.w && y < c.h) {
            const int k = y * c.w + x;
            if (l == 0 && p.depth_m) p.depth_m[k] = z[q];
            p.invd[l][k] = iz;
            p.zmap[l][k] = warp_depth_of(iz);
            p.vmap[l][k] = v[q];
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int x = x0 + cx[q], y = y0 + r[q];
        if (x >= c.w || y >= c.h) continue;
        float4 n = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
        if (x < c.w - 1 && y < c.h - 1) n = normal_of(v[q], sv[r[q]][cx[q] + 1], sv[r[q] + 1][cx[q]]);
        p.nmap[l][y * c.w + x] = n;
    }
}

void launch_depth_pyramid(const void *src, int is_u16, int pitch, float scale, int L, const LevelCam *cam,
                          float *depth_m, TrackLevelBufs *out, cudaStream_t s) {
    DepthPyramid p;
    memset(&p, 0, sizeof(p));
    p.src = src;
    p.is_u16 = is_u16;
    p.pitch = pitch;
    p.scale = scale;
    p.L = L;
    p.depth_m = depth_m;
    for (int l = 0; l < L; ++l) {
        p.c[l] = cam[l];
        p.tiles_x[l] = (cam[l].w + kDepthTileX - 1) / kDepthTileX;
        p.first[l + 1] = p.first[l] + p.tiles_x[l] * ((cam[l].h + kDepthTileY - 1) / kDepthTileY);
        p.invd[l] = out[l].invd;
        p.zmap[l] = out[l].z;
        p.vmap[l] = out[l].vmap;
        p.nmap[l] = out[l].nmap;
    }
    depth_pyramid_kernel<<<p.first[L], 256, 0, s>>>(p);
}

// The whole model pyramid in one launch (RGBDTracking.cu:140-150: level 0's
// normals, then each level's nearest pyr-down vertex map and its normals).
// Level l's vertex (x, y) of the chained pyr-down is level 0's vertex
// (2^l x, 2^l y) when x < w_l - 1 and y < h_l - 1 and invalid otherwise (the
// inner levels' conditions follow from the outer one), so every level reads
// the raycast's level-0 map directly and no level waits for another: the same
// values, one launch instead of one per level.  Thread i covers pixel i of the
// levels laid end to end.
struct ModelPyramid {
    int L, w[kMaxLevels], h[kMaxLevels], first[kMaxLevels + 1];
    float4 *vmap[kMaxLevels], *nmap[kMaxLevels];
};

__device__ __forceinline__ float4 model_vertex(const ModelPyramid &mp, int l, int x, int y) {
    if (l == 0) {
        if (x >= mp.w[0] || y >= mp.h[0]) return make_float4(0.0f, 0.0f, 0.0f, -1.0f);
        return mp.vmap[0][(size_t)y * mp.w[0] + x];
    }
    if (x >= mp.w[l] - 1 || y >= mp.h[l] - 1) return make_float4(0.0f, 0.0f, 0.0f, -1.0f);
    return mp.vmap[0][(size_t)(y << l) * mp.w[0] + (x << l)];
}

__global__ void model_pyramid_kernel(const ModelPyramid mp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= mp.first[mp.L]) return;
    int l = 0;
    while (l + 1 < mp.L && i >= mp.first[l + 1]) ++l;
    const int k = i - mp.first[l], w = mp.w[l], h = mp.h[l];
    const int y = k / w, x = k - y * w;
    const float4 v00 = model_vertex(mp, l, x, y);
    if (l > 0) mp.vmap[l][k] = v00;
    float4 n = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
    if (x < w - 1 && y < h - 1) n = normal_of(v00, model_vertex(mp, l, x + 1, y), model_vertex(mp, l, x, y + 1));
    mp.nmap[l][k] = n;
}

void launch_model_pyramid(int L, const int *w, const int *h, float4 *const *vmap, float4 *const *nmap,
                          cudaStream_t s) {
    ModelPyramid mp;
    memset(&mp, 0, sizeof(mp));
    mp.L = L;
    mp.first[0] = 0;
    for (int l = 0; l < L; ++l) {
        mp.w[l] = w[l];
        mp.h[l] = h[l];
        mp.vmap[l] = vmap[l];
        mp.nmap[l] = nmap[l];
        mp.first[l + 1] = mp.first[l] + w[l] * h[l];
    }
    if (mp.first[L] == 0) return;
    model_pyramid_kernel<<<(mp.first[L] + 255) / 256, 256, 0, s>>>(mp);
}

// ---------------------------------------------------------------- shading
// RenderScene (ImageProc.cu:80-139): Phong shading of a vertex/normal map for
// display, white surface (ambient 0.3, diffuse 0.5, specular 0.2, power 20),
// point light at `light` (camera frame); a pixel without a vertex is
// (4, 2, 2, 255).  Colour bytes are the saturated intensity * 255 truncated.
__device__ __forceinline__ float3 normalised(float3 v) {
    const float n = sqrtf(v.x * v.x + v.y * v.y + v.z * v.z);
    return make_float3(v.x / n, v.y / n, v.z / n);
}

__global__ void render_scene_kernel(const float4 *__restrict__ vmap, const float4 *__restrict__ nmap, int vpitch,
                                    int w, int h, float3 light, uchar4 *__restrict__ out, int opitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const float4 p4 = vmap[(size_t)y * vpitch + x];
    const float4 n4 = nmap[(size_t)y * vpitch + x];
    uchar4 o = make_uchar4(4, 2, 2, 255);
    if (!isnan(p4.x)) {
        const float3 p = make_float3(p4.x, p4.y, p4.z), nrm = make_float3(n4.x, n4.y, n4.z);
        const float3 L = normalised(make_float3(light.x - p.x, light.y - p.y, light.z - p.z));
        const float3 V = normalised(make_float3(-p.x, -p.y, -p.z));
        const float nl = nrm.x * L.x + nrm.y * L.y + nrm.z * L.z;
        const float3 R = normalised(make_float3(2.0f * nrm.x * nl - L.x, 2.0f * nrm.y * nl - L.y, 2.0f * nrm.z * nl - L.z));
        const float rv = R.x * V.x + R.y * V.y + R.z * V.z;
        const float I = 0.3f + 0.5f * fmaxf(0.0f, nl) + 0.2f * powf(fmaxf(0.0f, rv), 20.0f);
        const unsigned char c = (unsigned char)(__saturatef(I) * 255.0f);
        o = make_uchar4(c, c, c, 255);
    }
    out[(size_t)y * opitch + x] = o;
}

void launch_render_scene(const float4 *vmap, const float4 *nmap, int vpitch, int w, int h, float3 light,
                         uchar4 *out, int opitch, cudaStream_t s) {
    dim3 block(32, 8);
    dim3 grid((w + 31) / 32, (h + 7) / 8);
    render_scene_kernel<<<grid, block, 0, s>>>(vmap, nmap, vpitch, w, h, light, out, opitch);
}

}  // namespace yas

// ---------------------------------------------------------------- free functions of ImageProc.h
// Standalone, pitched forms of the per-pixel functions the tracker fuses into
// its pyramid kernels, for callers of the reference's free functions
// (RGBDFusion/include/ImageProc.h:8-24).  One thread per pixel, 32x8 blocks.
namespace yas {

template <typename T>
__device__ __forceinline__ T *row_at(T *base, int pitch_bytes, int y) {
    return reinterpret_cast<T *>(reinterpret_cast<char *>(const_cast<typename std::remove_const<T>::type *>(base)) +
                                 (size_t)y * pitch_bytes);
}

__global__ void free_pyrdown_depth_kernel(const float *src, int spitch, float *dst, int dw, int dh, int dpitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    // PyrDownDepth_kernel: the last row and column are left as they are
    if (x >= dw - 1 || y >= dh - 1) return;
    row_at(dst, dpitch, y)[x] = row_at(src, spitch, 2 * y)[2 * x];
}

__global__ void free_inv_depth_kernel(const float *depth, int pitch, int w, int h, float *inv, int ipitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    row_at(inv, ipitch, y)[x] = inv_depth_of(row_at(depth, pitch, y)[x]);
}

__global__ void free_vertex_map_kernel(const float *invd, int pitch, int w, int h, float4 *vmap, int vpitch,
                                       float invfx, float invfy, float cx, float cy, float cut_off) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const float invz = row_at(invd, pitch, y)[x];
    const float z = 1.0f / invz;
    float4 &o = row_at(vmap, vpitch, y)[x];
    if (invz > 0.0f && z < cut_off)
        o = make_float4(z * ((float)x - cx) * invfx, z * ((float)y - cy) * invfy, z, 1.0f);
    else
        o.w = -1.0f;  // ComputeVertexMap_kernel leaves x, y, z as they are
}

__global__ void free_normal_map_kernel(const float4 *vmap, int pitch, int w, int h, float4 *nmap, int npitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    float4 &o = row_at(nmap, npitch, y)[x];
    if (x == w - 1 || y == h - 1) {
        o.w = -1.0f;
        return;
    }
    const float4 n = normal_of(row_at(vmap, pitch, y)[x], row_at(vmap, pitch, y)[x + 1], row_at(vmap, pitch, y + 1)[x]);
    if (n.w > 0.0f)
        o = n;
    else
        o.w = -1.0f;
}

__global__ void free_gradient_kernel(const float *src, int pitch, int w, int h, float *gx, float *gy, int gpitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    float *ox = row_at(gx, gpitch, y) + x, *oy = row_at(gy, gpitch, y) + x;
    if (x < 1 || y < 1 || x > w - 2 || y > h - 2) {
        *ox = *oy = 0.0f;
    } else {
        const float *r = row_at(src, pitch, y);
        *ox = (r[x + 1] - r[x - 1]) * 0.5f;
        *oy = (row_at(src, pitch, y + 1)[x] - row_at(src, pitch, y - 1)[x]) * 0.5f;
    }
}

// TransformReferencePoint_kernel: RKinv (x, y, 1) z + t in FP32, Eigen's
// row-by-row product order, one rounding per operation.
__global__ void free_transform_points_kernel(const float *invd, int pitch, int w, int h, float4 *out, int opitch,
                                             Rigid32 RK) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const float zinv = row_at(invd, pitch, y)[x];
    float4 &o = row_at(out, opitch, y)[x];
    if (zinv > 0.0f) {
        const float z = 1.0f / zinv, fx = (float)x, fy = (float)y;
        float p[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            p[i] = __fadd_rn(__fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(RK.r[i * 3], fx), __fmul_rn(RK.r[i * 3 + 1], fy)),
                                                 RK.r[i * 3 + 2]),
                                       z),
                             RK.t[i]);
        o = make_float4(p[0], p[1], p[2], 1.0f);
    } else {
        o = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
    }
}

}  // namespace yas

using namespace yas;

namespace {
inline dim3 grid_of(int w, int h) { return dim3((unsigned)((w + 31) / 32), (unsigned)((h + 7) / 8)); }
inline bool bad_img(const void *p, int w, int h, int pitch, int elem) {
    return !p || w <= 0 || h <= 0 || pitch < w * elem || (pitch % elem) != 0;
}
}  // namespace

extern "C" {

YAS_API int yas_pyr_down_depth(const float *src, int src_w, int src_h, int src_pitch, float *dst, int dst_w,
                               int dst_h, int dst_pitch, void *stream) {
    if (bad_img(src, src_w, src_h, src_pitch, 4) || bad_img(dst, dst_w, dst_h, dst_pitch, 4) ||
        2 * (dst_w - 2) >= src_w || 2 * (dst_h - 2) >= src_h)
        return YAS_ERR_BAD_ARG;
    free_pyrdown_depth_kernel<<<grid_of(dst_w, dst_h), dim3(32, 8), 0, (cudaStream_t)stream>>>(
        src, src_pitch, dst, dst_w, dst_h, dst_pitch);
    YAS_TRY_CUDA(cudaGetLastError());
    return YAS_OK;
}

YAS_API int yas_depth_to_inv_depth(const float *depth, int w, int h, int pitch, float *inv_depth, int inv_pitch,
                                   void *stream) {
    if (bad_img(depth, w, h, pitch, 4) || bad_img(inv_depth, w, h, inv_pitch, 4)) return YAS_ERR_BAD_ARG;
    free_inv_depth_kernel<<<grid_of(w, h), dim3(32, 8), 0, (cudaStream_t)stream>>>(depth, pitch, w, h, inv_depth,
                                                                                   inv_pitch);
    YAS_TRY_CUDA(cudaGetLastError());
    return YAS_OK;
}

YAS_API int yas_compute_vertex_map(const float *inv_depth, int w, int h, int pitch, float *vmap, int vmap_pitch,
                                   float invfx, float invfy, float cx, float cy, float cut_off, void *stream) {
    if (bad_img(inv_depth, w, h, pitch, 4) || bad_img(vmap, w, h, vmap_pitch, 16)) return YAS_ERR_BAD_ARG;
    free_vertex_map_kernel<<<grid_of(w, h), dim3(32, 8), 0, (cudaStream_t)stream>>>(
        inv_depth, pitch, w, h, reinterpret_cast<float4 *>(vmap), vmap_pitch, invfx, invfy, cx, cy, cut_off);
    YAS_TRY_CUDA(cudaGetLastError());
    return YAS_OK;
}

YAS_API int yas_compute_normal_map(const float *vmap, int w, int h, int pitch, float *nmap, int nmap_pitch,
                                   void *stream) {
    if (bad_img(vmap, w, h, pitch, 16) || bad_img(nmap, w, h, nmap_pitch, 16)) return YAS_ERR_BAD_ARG;
    free_normal_map_kernel<<<grid_of(w, h), dim3(32, 8), 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const float4 *>(vmap), pitch, w, h, reinterpret_cast<float4 *>(nmap), nmap_pitch);
    YAS_TRY_CUDA(cudaGetLastError());
    return YAS_OK;
}

YAS_API int yas_image_gradient(const float *image, int w, int h, int pitch, float *gx, float *gy, int grad_pitch,
                               void *stream) {
    if (bad_img(image, w, h, pitch, 4) || bad_img(gx, w, h, grad_pitch, 4) || bad_img(gy, w, h, grad_pitch, 4))
        return YAS_ERR_BAD_ARG;
    free_gradient_kernel<<<grid_of(w, h), dim3(32, 8), 0, (cudaStream_t)stream>>>(image, pitch, w, h, gx, gy,
                                                                                  grad_pitch);
    YAS_TRY_CUDA(cudaGetLastError());
    return YAS_OK;
}

YAS_API int yas_transform_reference_point(const float *inv_depth, int w, int h, int pitch, float *vmap,
                                          int vmap_pitch, const double *K, const yas_pose *T, void *stream) {
    if (bad_img(inv_depth, w, h, pitch, 4) || bad_img(vmap, w, h, vmap_pitch, 16) || !K || !T) return YAS_ERR_BAD_ARG;
    // R * K^-1 in FP64, then rounded to FP32 (TransformReferencePoint, ImageProc.cu:64-78)
    const double fx = K[0], fy = K[4], cx = K[2], cy = K[5];
    if (!(fx != 0.0 && fy != 0.0)) return YAS_ERR_BAD_ARG;
    const double Ki[9] = {1.0 / fx, 0.0, -cx / fx, 0.0, 1.0 / fy, -cy / fy, 0.0, 0.0, 1.0};
    Rigid32 RK;
    for (int i = 0; i < 3; ++i) {
        for (int j = 0; j < 3; ++j)
            RK.r[i * 3 + j] = (float)((T->m[i * 4 + 0] * Ki[0 * 3 + j] + T->m[i * 4 + 1] * Ki[1 * 3 + j]) +
                                      T->m[i * 4 + 2] * Ki[2 * 3 + j]);
        RK.t[i] = (float)T->m[i * 4 + 3];
    }
    free_transform_points_kernel<<<grid_of(w, h), dim3(32, 8), 0, (cudaStream_t)stream>>>(
        inv_depth, pitch, w, h, reinterpret_cast<float4 *>(vmap), vmap_pitch, RK);
    YAS_TRY_CUDA(cudaGetLastError());
    return YAS_OK;
}

YAS_API int yas_vmap_to_depth(const float *vmap, int w, int h, int pitch, float *depth, int depth_pitch,
                              void *stream) {
    if (bad_img(vmap, w, h, pitch, 16) || bad_img(depth, w, h, depth_pitch, 4)) return YAS_ERR_BAD_ARG;
    launch_vmap_to_depth(reinterpret_cast<const float4 *>(vmap), pitch / 16, depth, depth_pitch / 4, w, h,
                         (cudaStream_t)stream);
    YAS_TRY_CUDA(cudaGetLastError());
    return YAS_OK;
}

}  // extern "C"
