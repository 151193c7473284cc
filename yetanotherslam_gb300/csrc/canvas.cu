// canvas.cu — headless drawing of submap meshes into an RGBA image.
//
// The reference draws every inactive submap's marching-cubes mesh with a GLSL
// program (FullSystem/src/MapDrawer.cpp:13-58 shaders, :159-234 draw loop):
// the vertex shader shades each vertex in the submap's own frame with a
// light at (5, 5, 5) and the viewer at the origin,
//     I = 0.3 + 0.5 max(0, n.L) + 0.2 max(0, R.V)^20,
//     L = normalize(light - p), V = normalize(-p), R = normalize(2 n (n.L) - L),
// places it with mvpMat * Tmw, and OpenGL interpolates the colour over the
// triangle.  There is no GL here: a CUDA rasteriser restates it into a device
// buffer.  Each triangle is moved by Tmw (submap -> world) and Tcw (world ->
// camera), projected with pinhole intrinsics (pixel centres at integer
// coordinates), and every covered pixel takes the perspective-correct
// interpolated intensity.  The depth test is one 64-bit atomicMin per
// fragment on (depth bits << 32 | RGBA), so meshes drawn one after another
// share the z-buffer and equal depths resolve the same way in any order.
// Triangles with a vertex nearer than 5 cm are not drawn (no clipping).
// All arithmetic is one rounding per operation in a fixed order, so the image
// is reproducible bit for bit by a CPU restatement.
#include <mutex>

#include "yas_internal.h"

struct yas_canvas {
    int w = 0, h = 0;
    yas::Cam cam;
    cudaStream_t stream = nullptr;
    unsigned long long *keys = nullptr;  // w * h
    // w * h colours, then w * h depths: what a host read copies.  Kept: memory
    // allocated for one read goes back to the system at its synchronisation, and
    // a 640x480 read took 213 us for the 45 that its copies take.
    uchar4 *image = nullptr;
    std::mutex image_mutex;  // one host read at a time: its colours and depths are of one moment
};

namespace yas {

constexpr float kCanvasNear = 0.05f;
constexpr unsigned long long kCanvasEmpty = ~0ull;

struct Affine {
    float m[12];  // row-major [R | t]
};

__device__ __forceinline__ float3 affine_apply(const Affine &A, float x, float y, float z) {
    float3 o;
    o.x = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(A.m[0], x), __fmul_rn(A.m[1], y)), __fmul_rn(A.m[2], z)), A.m[3]);
    o.y = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(A.m[4], x), __fmul_rn(A.m[5], y)), __fmul_rn(A.m[6], z)), A.m[7]);
    o.z = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(A.m[8], x), __fmul_rn(A.m[9], y)), __fmul_rn(A.m[10], z)),
                    A.m[11]);
    return o;
}

__device__ __forceinline__ float dot3(float3 a, float3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}

__device__ __forceinline__ float3 normalize3(float3 v) {
    const float l = __fsqrt_rn(dot3(v, v));
    if (!(l > 0.0f)) return make_float3(0.0f, 0.0f, 0.0f);
    return make_float3(__fdiv_rn(v.x, l), __fdiv_rn(v.y, l), __fdiv_rn(v.z, l));
}

// The vertex shader's intensity (MapDrawer.cpp:26-44), in [0, 1].
__device__ __forceinline__ float mesh_shade(float3 p, float3 n) {
    const float3 L = normalize3(make_float3(__fsub_rn(5.0f, p.x), __fsub_rn(5.0f, p.y), __fsub_rn(5.0f, p.z)));
    const float3 V = normalize3(make_float3(-p.x, -p.y, -p.z));
    const float nl = dot3(n, L);
    const float k = __fmul_rn(2.0f, nl);
    const float3 R = normalize3(make_float3(__fsub_rn(__fmul_rn(k, n.x), L.x), __fsub_rn(__fmul_rn(k, n.y), L.y),
                                            __fsub_rn(__fmul_rn(k, n.z), L.z)));
    const float rv = fmaxf(0.0f, dot3(R, V));
    const float r2 = __fmul_rn(rv, rv), r4 = __fmul_rn(r2, r2), r8 = __fmul_rn(r4, r4), r16 = __fmul_rn(r8, r8);
    const float r20 = __fmul_rn(r16, r4);
    const float i = __fadd_rn(__fadd_rn(0.3f, __fmul_rn(0.5f, fmaxf(0.0f, nl))), __fmul_rn(0.2f, r20));
    return fminf(1.0f, fmaxf(0.0f, i));
}

// Twice the signed area of (a, b, p).
__device__ __forceinline__ float edge_fn(float ax, float ay, float bx, float by, float px, float py) {
    return __fsub_rn(__fmul_rn(__fsub_rn(bx, ax), __fsub_rn(py, ay)), __fmul_rn(__fsub_rn(by, ay), __fsub_rn(px, ax)));
}

// A projected triangle: image coordinates and inverse depths of its vertices.
struct Projected {
    float u[3], v[3], iz[3];
};

// Pixels of its bounding box, clamped before the conversion to int (a vertex at
// 5 cm can project far out).
struct PixelBox {
    int x0, x1, y0, y1;
    __device__ __forceinline__ PixelBox(const Projected &p, int w, int h) {
        const float lim = 1.0e7f;
        x0 = max(0, (int)ceilf(fmaxf(-lim, fminf(fminf(p.u[0], p.u[1]), p.u[2]))));
        x1 = min(w - 1, (int)floorf(fminf(lim, fmaxf(fmaxf(p.u[0], p.u[1]), p.u[2]))));
        y0 = max(0, (int)ceilf(fmaxf(-lim, fminf(fminf(p.v[0], p.v[1]), p.v[2]))));
        y1 = min(h - 1, (int)floorf(fminf(lim, fmaxf(fmaxf(p.v[0], p.v[1]), p.v[2]))));
    }
};

// The three edge functions at pixel (x, y); true when it is covered.
__device__ __forceinline__ bool covered(const Projected &p, float area, int x, int y, float e[3]) {
    const float px = (float)x, py = (float)y;
    e[0] = edge_fn(p.u[1], p.v[1], p.u[2], p.v[2], px, py);
    e[1] = edge_fn(p.u[2], p.v[2], p.u[0], p.v[0], px, py);
    e[2] = edge_fn(p.u[0], p.v[0], p.u[1], p.v[1], px, py);
    return area > 0.0f ? (e[0] >= 0.0f && e[1] >= 0.0f && e[2] >= 0.0f) : (e[0] <= 0.0f && e[1] <= 0.0f && e[2] <= 0.0f);
}

__device__ __forceinline__ float area_of(const Projected &p) {
    return edge_fn(p.u[0], p.v[0], p.u[1], p.v[1], p.u[2], p.v[2]);
}

// True when triangle t can cover a pixel; boxes of up to kSmallBox pixels are
// tried, larger ones pass.
constexpr int kSmallBox = 6;
__device__ __forceinline__ bool project_triangle(const float *__restrict__ pts, unsigned t, const Affine &model,
                                                 const Affine &view, const Cam &cam, int w, int h, Projected &o) {
    bool near = false;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float *p = pts + (size_t)t * 9 + k * 3;
        const float3 pw = affine_apply(model, p[0], p[1], p[2]);
        const float3 pc = affine_apply(view, pw.x, pw.y, pw.z);
        near = near || !(pc.z >= kCanvasNear);
        o.u[k] = __fadd_rn(__fdiv_rn(__fmul_rn(cam.fx, pc.x), pc.z), cam.cx);
        o.v[k] = __fadd_rn(__fdiv_rn(__fmul_rn(cam.fy, pc.y), pc.z), cam.cy);
        o.iz[k] = __fdiv_rn(1.0f, pc.z);
    }
    const float area = area_of(o);
    if (near || !(area != 0.0f)) return false;
    const PixelBox box(o, w, h);
    if (box.x0 > box.x1 || box.y0 > box.y1) return false;
    if (box.x1 - box.x0 >= kSmallBox || (box.x1 - box.x0 + 1) * (box.y1 - box.y0 + 1) > kSmallBox) return true;
    bool any = false;
    float e[3];
    for (int y = box.y0; y <= box.y1; ++y)
        for (int x = box.x0; x <= box.x1; ++x) any = any || covered(o, area, x, y, e);
    return any;
}

__device__ __forceinline__ void draw_triangle(const float *__restrict__ pts, const float *__restrict__ nrm, unsigned t,
                                              const Projected &p, unsigned long long *keys, int w, int h) {
    float ioz[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float *a = pts + (size_t)t * 9 + k * 3, *q = nrm + (size_t)t * 9 + k * 3;
        ioz[k] = __fmul_rn(mesh_shade(make_float3(a[0], a[1], a[2]), make_float3(q[0], q[1], q[2])), p.iz[k]);
    }
    const float area = area_of(p);
    const PixelBox box(p, w, h);
    for (int y = box.y0; y <= box.y1; ++y)
        for (int x = box.x0; x <= box.x1; ++x) {
            float e[3];
            if (!covered(p, area, x, y, e)) continue;
            const float b0 = __fdiv_rn(e[0], area), b1 = __fdiv_rn(e[1], area), b2 = __fdiv_rn(e[2], area);
            const float wz =
                __fadd_rn(__fadd_rn(__fmul_rn(b0, p.iz[0]), __fmul_rn(b1, p.iz[1])), __fmul_rn(b2, p.iz[2]));
            if (!(wz > 0.0f)) continue;
            const float z = __fdiv_rn(1.0f, wz);
            const float wi = __fadd_rn(__fadd_rn(__fmul_rn(b0, ioz[0]), __fmul_rn(b1, ioz[1])), __fmul_rn(b2, ioz[2]));
            const float in01 = fminf(1.0f, fmaxf(0.0f, __fmul_rn(wi, z)));
            const unsigned c = (unsigned)floorf(__fadd_rn(__fmul_rn(in01, 255.0f), 0.5f));
            const unsigned rgba = c | (c << 8) | (c << 16) | (255u << 24);
            const unsigned long long key = ((unsigned long long)__float_as_uint(z) << 32) | rgba;
            atomicMin(keys + (size_t)y * w + x, key);
        }
}

// A mesh's triangles are about a pixel in size, so many cover none, and shading
// (27 divisions, 9 square roots) is most of a triangle's work.  A warp projects
// 32 triangles at a time, queues those that cover a pixel, and shades and draws
// the queue 32 at a time, every lane with a triangle.  1.03 M triangles of 6 mm
// at 640x480: 54.5 us shading each triangle first, 33.1 here (bound by the
// exact divisions and square roots; more warps in flight are no faster).
constexpr int kDrawThreads = 128;

__global__ void __launch_bounds__(kDrawThreads) canvas_draw_kernel(const float *__restrict__ pts, const float *__restrict__ nrm,
                                                                   unsigned ntris, Affine model, Affine view, Cam cam,
                                                                   unsigned long long *keys, int w, int h) {
    __shared__ float queue_p[kDrawThreads / 32][9][64];
    __shared__ unsigned queue_t[kDrawThreads / 32][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float(*qp)[64] = queue_p[warp];
    unsigned *qt = queue_t[warp];
    int n = 0;  // queued, at most 31 + 32
    bool last;
    long long t0 = (long long)blockIdx.x * kDrawThreads + warp * 32;
    do {
        Projected p;
        const long long t = t0 + lane;
        const bool hit = t < ntris && project_triangle(pts, (unsigned)t, model, view, cam, w, h, p);
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        if (hit) {
            const int k = n + __popc(hits & ((1u << lane) - 1u));
            qt[k] = (unsigned)t;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                qp[i][k] = p.u[i];
                qp[3 + i][k] = p.v[i];
                qp[6 + i][k] = p.iz[i];
            }
        }
        n += __popc(hits);
        __syncwarp();
        t0 += (long long)gridDim.x * kDrawThreads;
        last = t0 >= ntris;
        while (n >= 32 || (last && n > 0)) {
            const int m = min(n, 32);
            n -= m;
            if (lane < m) {
                const int k = n + lane;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    p.u[i] = qp[i][k];
                    p.v[i] = qp[3 + i][k];
                    p.iz[i] = qp[6 + i][k];
                }
                draw_triangle(pts, nrm, qt[k], p, keys, w, h);
            }
            __syncwarp();
        }
    } while (!last);
}

__global__ void canvas_resolve_kernel(const unsigned long long *keys, int w, int h, uchar4 *rgba, int rpitch,
                                      float *depth, int dpitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const unsigned long long k = keys[(size_t)y * w + x];
    const bool empty = k == kCanvasEmpty;
    if (rgba) {
        const unsigned c = empty ? 0xffffffffu : (unsigned)k;  // the viewer clears to white
        rgba[(size_t)y * rpitch + x] = make_uchar4(c & 255u, (c >> 8) & 255u, (c >> 16) & 255u, c >> 24);
    }
    if (depth) depth[(size_t)y * dpitch + x] = empty ? 0.0f : __uint_as_float((unsigned)(k >> 32));
}

static Affine affine_of(const yas_pose &p) {
    Affine a;
    for (int i = 0; i < 12; ++i) a.m[i] = (float)p.m[i];
    return a;
}

// h rows of w words to a host image of that pitch: one copy where the rows adjoin.
static cudaError_t copy_rows(void *dst, int pitch, const void *src, const yas_canvas *c) {
    const size_t row = (size_t)c->w * 4;
    if ((size_t)pitch == row) return cudaMemcpyAsync(dst, src, row * c->h, cudaMemcpyDeviceToHost, c->stream);
    return cudaMemcpy2DAsync(dst, pitch, src, row, row, c->h, cudaMemcpyDeviceToHost, c->stream);
}

}  // namespace yas

using namespace yas;

extern "C" {

YAS_API int yas_canvas_destroy(yas_canvas *c) {
    if (!c) return YAS_ERR_BAD_ARG;
    if (c->stream) cudaStreamSynchronize(c->stream);
    cudaFree(c->keys);
    cudaFree(c->image);
    delete c;
    return YAS_OK;
}

YAS_API int yas_canvas_create(yas_canvas **out, int width, int height, const yas_intrinsics *K, void *stream) {
    if (!out || !K || width <= 0 || height <= 0 || width > 16384 || height > 16384) return YAS_ERR_BAD_ARG;
    yas_canvas *c = new yas_canvas();
    c->w = width;
    c->h = height;
    c->cam = make_cam(K->fx, K->fy, K->cx, K->cy, width, height);
    c->stream = (cudaStream_t)stream;
    if (cudaMalloc(&c->keys, (size_t)width * height * sizeof(unsigned long long)) != cudaSuccess ||
        cudaMalloc(&c->image, (size_t)width * height * (sizeof(uchar4) + sizeof(float))) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(c->keys);
        delete c;
        return YAS_ERR_OOM;
    }
    *out = c;
    return yas_canvas_clear(c);
}

YAS_API int yas_canvas_clear(yas_canvas *c) {
    if (!c) return YAS_ERR_BAD_ARG;
    YAS_TRY_CUDA(cudaMemsetAsync(c->keys, 0xff, (size_t)c->w * c->h * sizeof(unsigned long long), c->stream));
    return YAS_OK;
}

YAS_API int yas_canvas_draw_triangles(yas_canvas *c, const float *points, const float *normals, unsigned n_tris,
                                      int on_device, const yas_pose *Tmw, const yas_pose *Tcw) {
    if (!c || !Tmw || !Tcw || (n_tris && (!points || !normals))) return YAS_ERR_BAD_ARG;
    if (!n_tris) return YAS_OK;
    const float *p = points, *n = normals;
    float *tmp = nullptr;
    if (!on_device) {
        const size_t bytes = (size_t)n_tris * 9 * sizeof(float);
        if (cudaMallocAsync(&tmp, 2 * bytes, c->stream) != cudaSuccess) {
            cudaGetLastError();
            return YAS_ERR_OOM;
        }
        YAS_TRY_CUDA(cudaMemcpyAsync(tmp, points, bytes, cudaMemcpyHostToDevice, c->stream));
        YAS_TRY_CUDA(cudaMemcpyAsync(tmp + (size_t)n_tris * 9, normals, bytes, cudaMemcpyHostToDevice, c->stream));
        p = tmp;
        n = tmp + (size_t)n_tris * 9;
    }
    const int grid = (int)std::min<unsigned>((n_tris + kDrawThreads - 1) / kDrawThreads, (unsigned)kSMs * 16u);
    canvas_draw_kernel<<<grid, kDrawThreads, 0, c->stream>>>(p, n, n_tris, affine_of(*Tmw), affine_of(*Tcw), c->cam, c->keys,
                                                    c->w, c->h);
    cudaError_t e = cudaGetLastError();
    if (tmp) {
        cudaFreeAsync(tmp, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    }
    YAS_TRY_CUDA(e);
    return YAS_OK;
}

YAS_API int yas_canvas_draw_mesh(yas_canvas *c, yas_mesher *me, const yas_pose *Tmw, const yas_pose *Tcw) {
    if (!c || !me) return YAS_ERR_BAD_ARG;
    const unsigned n = std::min<unsigned>(me->last_tris, (unsigned)me->mb.max_tris);
    if (me->stream != c->stream) YAS_TRY_CUDA(cudaStreamSynchronize(me->stream));
    return yas_canvas_draw_triangles(c, me->mb.points, me->mb.normals, n, 1, Tmw, Tcw);
}

YAS_API int yas_canvas_read(yas_canvas *c, uint8_t *rgba, int rgba_pitch, float *depth, int depth_pitch,
                            int on_device) {
    if (!c || (!rgba && !depth)) return YAS_ERR_BAD_ARG;
    if ((rgba && (rgba_pitch < c->w * 4 || rgba_pitch % 4)) || (depth && (depth_pitch < c->w * 4 || depth_pitch % 4)))
        return YAS_ERR_BAD_ARG;
    uchar4 *drgba = reinterpret_cast<uchar4 *>(rgba);
    float *ddepth = depth;
    if (!on_device) {
        drgba = rgba ? c->image : nullptr;
        ddepth = depth ? reinterpret_cast<float *>(c->image + (size_t)c->w * c->h) : nullptr;
    }
    std::unique_lock<std::mutex> lk(c->image_mutex, std::defer_lock);
    if (!on_device) lk.lock();
    const int rp = on_device ? rgba_pitch / 4 : c->w, dp = on_device ? depth_pitch / 4 : c->w;
    dim3 grid((c->w + 31) / 32, (c->h + 7) / 8);
    canvas_resolve_kernel<<<grid, dim3(32, 8), 0, c->stream>>>(c->keys, c->w, c->h, drgba, rp, ddepth, dp);
    cudaError_t e = cudaGetLastError();
    if (!on_device) {
        if (e == cudaSuccess && rgba) e = copy_rows(rgba, rgba_pitch, drgba, c);
        if (e == cudaSuccess && depth) e = copy_rows(depth, depth_pitch, ddepth, c);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    }
    YAS_TRY_CUDA(e);
    return YAS_OK;
}

}  // extern "C"
