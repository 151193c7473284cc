// map.cu — voxel-hash TSDF map: block allocation, visibility compaction,
// depth integration, reset and host export/import.
//
// Reference semantics (paths relative to the reference project root):
//   allocation   RGBDFusion/src/VoxelMap.cu:517-652 (CreateBlockLineTracingFunctor)
//   visibility   RGBDFusion/src/VoxelMap.cu:654-717, RGBDFusion/utils/VoxelStructUtils.h:112-147
//   integration  RGBDFusion/src/VoxelMap.cu:719-786 (DepthFusionFunctor)
//   reset        RGBDFusion/src/VoxelMap.cu:24-58
//
// GB300 layout: 16-byte open-addressing slots with packed 64-bit keys; the
// voxel pool is bump-allocated so pool index i <-> block_keys[i] is itself
// the allocated-block list (no full-table scans); new blocks are zeroed by the
// warp that allocated them.
#include <atomic>

#include "yas_internal.h"

namespace yas {

// f2i_floor: floor to int with NaN/out-of-range mapped to INT_MIN; the CPU
// oracle uses the same rule so that degenerate projections agree.
__device__ __forceinline__ int f2i_floor(float x) {
    if (!(x >= -2147483648.0f && x < 2147483648.0f)) return (int)0x80000000;
    return (int)floorf(x);
}

// ---------------------------------------------------------------- allocation
// Block coordinate of a camera-ray point at metric depth z (FP32 canonical):
// UnProjectWorld (VoxelStructUtils.h:100-110) -> WorldPtToVoxelPos -> VoxelPosToBlockPos.
__device__ __forceinline__ void ray_block(const Cam &c, const Rigid32 &T, float vs, int x, int y,
                                          float z, int b[3]) {
    float px = cmul(cmul(c.invfx, csub((float)x, c.cx)), z);
    float py = cmul(cmul(c.invfy, csub((float)y, c.cy)), z);
    float3 q = rigid_exact(T, px, py, z);
    b[0] = floor_div8(f2i_floor(cdiv(q.x, vs)));
    b[1] = floor_div8(f2i_floor(cdiv(q.y, vs)));
    b[2] = floor_div8(f2i_floor(cdiv(q.z, vs)));
}

// 3-D Bresenham walker over block coordinates with the reference's major-axis
// choice and error terms (VoxelMap.cu:568-650).
struct BlockLine {
    // components in the order major axis, a1, a2 (no indexing by axis, which
    // would put them in local memory)
    int cur[3], inc[3], d2[3];  // d2: 2 * |d|
    int major;
    int err1, err2;
    int count;  // number of blocks on the line (|d_major| + 1)

    // (m, a1, a2) = (0, 1, 2), (1, 0, 2) or (2, 1, 0)
    __device__ __forceinline__ void init(const int s[3], const int e[3]) {
        const int ax = abs(e[0] - s[0]), ay = abs(e[1] - s[1]), az = abs(e[2] - s[2]);
        major = ax >= ay && ax >= az ? 0 : (ay >= ax && ay >= az ? 1 : 2);
        const int sm = major == 0 ? s[0] : (major == 1 ? s[1] : s[2]), em = major == 0 ? e[0] : (major == 1 ? e[1] : e[2]);
        const int s1 = major == 1 ? s[0] : s[1], e1 = major == 1 ? e[0] : e[1];
        const int s2 = major == 2 ? s[0] : s[2], e2 = major == 2 ? e[0] : e[2];
        cur[0] = sm, cur[1] = s1, cur[2] = s2;
        inc[0] = em < sm ? -1 : 1, inc[1] = e1 < s1 ? -1 : 1, inc[2] = e2 < s2 ? -1 : 1;
        d2[0] = abs(em - sm) << 1, d2[1] = abs(e1 - s1) << 1, d2[2] = abs(e2 - s2) << 1;
        err1 = d2[1] - 1;
        err2 = d2[2] - 1;
        count = (d2[0] >> 1) + 1;
    }
    __device__ __forceinline__ void step() {
        if (err1 > 0) {
            cur[1] += inc[1];
            err1 -= d2[0];
        }
        if (err2 > 0) {
            cur[2] += inc[2];
            err2 -= d2[0];
        }
        err1 += d2[1];
        err2 += d2[2];
        cur[0] += inc[0];
    }
    __device__ __forceinline__ int3 block() const {
        return make_int3(major == 0 ? cur[0] : (major == 1 ? cur[1] : cur[2]), major == 1 ? cur[0] : cur[1],
                         major == 2 ? cur[0] : cur[2]);
    }
};

constexpr int kMaxLineBlocks = 1024;

// Opens a call at a pose given by the host: one launch for a pose copy and a
// memset.  With the call's kernels as dependents, one Fuse after another 160x120
// 23.1 / 16.9 us, 640x480 43.0 / 36.0.
__global__ void pose_begin_kernel(PosePair pose, PosePair *P, MapHeader *hdr) {
    release_dependents();
    if (threadIdx.x == 0) {
        *P = pose;
        hdr->n_visible = 0u;
    }
}

void launch_pose_begin(const MapDev &m, const PosePair &pose, PosePair *P, cudaStream_t s) {
    pose_begin_kernel<<<1, 32, 0, s>>>(pose, P, m.hdr);
}

template <int VBYTES>
__global__ void __launch_bounds__(256) allocate_kernel(MapDev m, const float *__restrict__ depth,
                                                       int pitch, Cam cam, const PosePair *P,
                                                       const int *skip) {
    dependent_wait();
    release_dependents();
    if (skip && *skip) return;
    const int x = blockIdx.x * 32 + (threadIdx.x & 31);
    const int y = blockIdx.y * 8 + (threadIdx.x >> 5);
    const Rigid32 T = P->T;

    BlockLine line;
    int n = 0;
    if (x < cam.w && y < cam.h) {
        float dist = depth[(size_t)y * pitch + x];
        if (!(isnan(dist) || dist < m.depth_min || dist > m.depth_max)) {
            const float half = m.trunc * 0.5f;
            float dnear = fmaxf(m.depth_min, csub(dist, half));
            float dfar = fminf(m.depth_max, cadd(dist, half));
            if (dnear < dfar) {
                int bs[3], be[3];
                ray_block(cam, T, m.voxel_size, x, y, dnear, bs);
                ray_block(cam, T, m.voxel_size, x, y, dfar, be);
                line.init(bs, be);
                n = line.count;
                if (n > kMaxLineBlocks) {
                    raise_error(m, YAS_ERR_COORD_RANGE);
                    n = 0;
                }
            }
        }
    }
    // Nearly all blocks of a frame are allocated already, so a step first looks
    // them up (two at a time: their first probes are in flight together); only
    // a warp with a lane whose block is missing goes through the insertion,
    // which matches the lanes' keys and takes two counters' round trips.  A
    // tracked frame at 640x480, 5 mm: 14 -> 9 us, 1280x720, 4 mm: 22 -> 16.
    const int nmax = __reduce_max_sync(0xffffffffu, n);
    for (int s = 0; s < nmax; s += 2) {
        unsigned long long key[2] = {kEmptyKey, kEmptyKey}, found[2] = {kEmptyKey, kEmptyKey};
        unsigned slot[2] = {0u, 0u};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (s + i >= n) continue;
            if (s + i > 0) line.step();
            const int3 b = line.block();
            if (coord_in_range(b.x, b.y, b.z)) {
                key[i] = pack_key(b.x, b.y, b.z);
                slot[i] = hash_key(key[i]) & m.slot_mask;
                found[i] = __ldcg(&m.slots[slot[i]].key);
            } else {
                raise_error(m, YAS_ERR_COORD_RANGE);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            bool missing = found[i] != key[i];
            if (missing && found[i] != kEmptyKey) missing = !probe_key(m, key[i], slot[i]);
            if (__any_sync(0xffffffffu, missing)) warp_insert<VBYTES>(m, key[i], missing);
        }
    }
}

void launch_allocate(const MapDev &m, int fmt, const float *depth, int pitch_elems, const Cam &cam,
                     const PosePair *P, const int *skip, cudaStream_t s, bool dependent) {
    dim3 block(256);
    dim3 grid((cam.w + 31) / 32, (cam.h + 7) / 8);
    launch_kernel(fmt == YAS_VOXEL_F32 ? allocate_kernel<8> : allocate_kernel<4>, grid, block, s, dependent, m,
                  depth, pitch_elems, cam, P, skip);
}

// ---------------------------------------------------------------- visibility
// CheckBlockVisibility (VoxelStructUtils.h:112-147), FP32 canonical.
__device__ __forceinline__ bool block_visible(const Cam &c, const Rigid32 &Tinv, float vs, float dmin,
                                              float dmax, int bx, int by, int bz) {
    const float scale = cmul(vs, 8.0f);
#pragma unroll
    for (int corner = 0; corner < 8; ++corner) {
        float wx = cmul((float)(bx + (corner & 1)), scale);
        float wy = cmul((float)(by + ((corner >> 1) & 1)), scale);
        float wz = cmul((float)(bz + ((corner >> 2) & 1)), scale);
        float3 p = rigid_exact(Tinv, wx, wy, wz);
        float u = cadd(cdiv(cmul(c.fx, p.x), p.z), c.cx);
        float v = cadd(cdiv(cmul(c.fy, p.y), p.z), c.cy);
        if (!(u < 0.0f || v < 0.0f || u > (float)(c.w - 1) || v > (float)(c.h - 1) || p.z < dmin ||
              p.z > dmax))
            return true;
    }
    return false;
}

__global__ void __launch_bounds__(256) visible_kernel(MapDev m, Cam cam, const PosePair *P,
                                                      const int *skip) {
    dependent_wait();
    release_dependents();
    if (skip && *skip) return;
    const unsigned n = num_blocks(m);
    const Rigid32 Tinv = P->Tinv;
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
        unsigned i = base + lane_id();
        bool vis = false;
        if (i < n) {
            int bx, by, bz;
            unpack_key(m.block_keys[i], bx, by, bz);
            vis = block_visible(cam, Tinv, m.voxel_size, m.depth_min, m.depth_max, bx, by, bz);
        }
        unsigned slot = warp_append(&m.hdr->n_visible, vis);
        if (vis) m.visible[slot] = (int)i;
    }
}

void launch_visible(const MapDev &m, const Cam &cam, const PosePair *P, const int *skip,
                    cudaStream_t s, bool dependent) {
    launch_kernel(visible_kernel, dim3(kSMs * 4), dim3(256), s, dependent, m, cam, P, skip);
}

// ---------------------------------------------------------------- integration
// Pixel index floor(((a / z) + c) + 0.5) with the IEEE quotient a / z, as the
// canonical FP32 order defines it: the exact form.
__device__ __forceinline__ int project_exact(float a, float z, float c) {
    return f2i_floor(cadd(cadd(cdiv(a, z), c), 0.5f));
}

// Approximate FP32 reciprocal (relative error at most 2^-23).
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Largest distance of the coordinate s = a rcp_approx(z) + c from an integer at
// which rint(s) is still the exact form's pixel, in an image `n` pixels wide.
// The approximate quotient is within 2^-22 of a / z (reciprocal 2^-23, product
// and IEEE quotient 2^-24 each) and the sums on either side round to within
// 2^-24 of their results, so s + 0.5 differs from the exact form's last sum by
// at most 2^-22 (2 |s| + |c| + 2); nearer than that to a pixel's edge, the
// exact form is evaluated (about one voxel in 500 at 640x480).  Outside the
// image the difference grows with |s| but stays far below its distance to the
// image, up to 2^18 pixels; beyond (-1) every coordinate is evaluated exactly.
__device__ __forceinline__ float project_margin(int n, float c) {
    const float m = 2.0f * (float)n + fabsf(c) + 4.0f;
    return m < 262144.0f ? 0.5f - m * 0x1p-22f : -1.0f;
}

// rint(s) of a pair by adding 1.5 * 2^23, and s's distance from it: no
// conversion, which would take the quarter-rate pipe.  |s| < 2^22; a larger one
// (or a NaN) comes back as a pixel outside every image or with a NaN distance.
__device__ __forceinline__ int2 nearest_pixel2(float2 s, float2 &off) {
    const float2 k = cadd2(s, pair(12582912.0f));
    off = csub2(s, cadd2(k, pair(-12582912.0f)));
    return make_int2(__float_as_int(k.x) - 0x4b400000, __float_as_int(k.y) - 0x4b400000);
}

// Each 128-thread group owns one block; thread t updates voxels 4t..4t+3
// (z = t/16, y = (t/2)%8, x = 4*(t%2) .. +3), one 16-byte (or 32-byte) access.
// SIGN = +1: DepthFusionFunctor (VoxelMap.cu:719-786).  SIGN = -1: the same
// observation removed again (de-integration, for re-integration after a pose
// correction): s <- (s w - d) / (w - 1), w <- w - 1; exact while the weight
// stayed below the cap, as the reference's running average is then invertible.
// Bound by instruction issue and by the latency of its reads (the depth image and
// the blocks are in L2): a thread projects its four voxels two at a time with
// packed FP32, starts their depth reads, and then updates all four under one
// branch.  13 k visible blocks at 640x480, 5 mm F16: 37.8 -> 25.6 us (before, a
// correctly rounded reciprocal, conversions and a branch per voxel; now 16.2 M warp
// instructions for 30.9 M, 65 % of the issue slots for 75 %, 29 warps an SM),
// 1280x720, 4 mm F16: 59.8 -> 39.7, 320x240, 8 mm F32: 15.7 -> 12.6.
template <int FMT, int SIGN>
__global__ void __launch_bounds__(256) integrate_kernel(MapDev m, const float *__restrict__ depth,
                                                        int pitch, Cam cam, const PosePair *P,
                                                        const int *skip) {
    typedef VoxelIO<FMT> IO;
    typedef typename IO::T V;
    dependent_wait();
    if (skip && *skip) return;
    const unsigned nvis = *(volatile unsigned *)&m.hdr->n_visible;
    const Rigid32 Tinv = P->Tinv;
    const int t = threadIdx.x & 127;
    const int lz = t >> 4, ly = (t >> 1) & 7, lx0 = (t & 1) * 4;
    const float vs = m.voxel_size, inv_trunc = 1.0f / m.trunc, ntrunc = -m.trunc;
    const float mar_u = project_margin(cam.w, cam.cx), mar_v = project_margin(cam.h, cam.cy);
    V *vox = static_cast<V *>(m.voxels);
    for (unsigned j = blockIdx.x * 2 + (threadIdx.x >> 7); j < nvis; j += gridDim.x * 2) {
        const int b = m.visible[j];
        int bx, by, bz;
        unpack_key(m.block_keys[b], bx, by, bz);
        V *p = vox + (size_t)b * kBlockVoxels + t * 4;
        V v[4];
        if (sizeof(V) == 4) {
            uint4 q = *reinterpret_cast<const uint4 *>(p);
            v[0] = *reinterpret_cast<V *>(&q.x);
            v[1] = *reinterpret_cast<V *>(&q.y);
            v[2] = *reinterpret_cast<V *>(&q.z);
            v[3] = *reinterpret_cast<V *>(&q.w);
        } else {
            float4 q0 = reinterpret_cast<const float4 *>(p)[0];
            float4 q1 = reinterpret_cast<const float4 *>(p)[1];
            v[0] = *reinterpret_cast<V *>(&q0.x);
            v[1] = *reinterpret_cast<V *>(&q0.z);
            v[2] = *reinterpret_cast<V *>(&q1.x);
            v[3] = *reinterpret_cast<V *>(&q1.z);
        }
        const float wy = cmul((float)(by * 8 + ly), vs);
        const float wz = cmul((float)(bz * 8 + lz), vs);
        const float x0 = (float)(bx * 8 + lx0);
        // the products of the rows with wy and wz are the same for all four
        const float xy = cmul(Tinv.r[1], wy), xz = cmul(Tinv.r[2], wz), yy = cmul(Tinv.r[4], wy), yz = cmul(Tinv.r[5], wz);
        const float zy = cmul(Tinv.r[7], wy), zz = cmul(Tinv.r[8], wz);
        float au[4], av[4], zc[4], dist[4];
        int u[4], w[4];
        bool edge[4];
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            // rigid_exact and the projection of a pair
            const float2 wx = cmul2(cadd2(pair(x0), make_float2((float)q, (float)(q + 1))), pair(vs));  // x0 + q is exact
            const float2 cx = cadd2(cadd2(cadd2(cmul_each(pair(Tinv.r[0]), wx), pair(xy)), pair(xz)), pair(Tinv.t[0]));
            const float2 cy = cadd2(cadd2(cadd2(cmul_each(pair(Tinv.r[3]), wx), pair(yy)), pair(yz)), pair(Tinv.t[1]));
            const float2 cz = cadd2(cadd2(cadd2(cmul_each(pair(Tinv.r[6]), wx), pair(zy)), pair(zz)), pair(Tinv.t[2]));
            const float2 a = cmul2(pair(cam.fx), cx), b2 = cmul2(pair(cam.fy), cy);
            const float2 rz = make_float2(rcp_approx(cz.x), rcp_approx(cz.y));
            float2 off_u, off_v;
            const int2 iu = nearest_pixel2(cadd2(cmul_each(a, rz), pair(cam.cx)), off_u);
            const int2 iv = nearest_pixel2(cadd2(cmul_each(b2, rz), pair(cam.cy)), off_v);
            edge[q] = !(fabsf(off_u.x) < mar_u && fabsf(off_v.x) < mar_v);
            edge[q + 1] = !(fabsf(off_u.y) < mar_u && fabsf(off_v.y) < mar_v);
            au[q] = a.x, au[q + 1] = a.y, av[q] = b2.x, av[q + 1] = b2.y;
            zc[q] = cz.x, zc[q + 1] = cz.y;
            u[q] = iu.x, u[q + 1] = iu.y, w[q] = iv.x, w[q + 1] = iv.y;
        }
        if (edge[0] || edge[1] || edge[2] || edge[3]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (!edge[q]) continue;
                u[q] = project_exact(au[q], zc[q], cam.cx);
                w[q] = project_exact(av[q], zc[q], cam.cy);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            dist[q] = __int_as_float(0x7fffffff);
            if ((unsigned)u[q] < (unsigned)cam.w && (unsigned)w[q] < (unsigned)cam.h)
                dist[q] = __ldg(depth + (size_t)w[q] * pitch + u[q]);
        }
        float d[4];
        bool ok[4], any = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            d[q] = csub(dist[q], zc[q]);
            ok[q] = dist[q] >= m.depth_min && dist[q] <= m.depth_max && !(d[q] < ntrunc);
            if (SIGN < 0) ok[q] = ok[q] && IO::wt(v[q]) != 0;
            any = any || ok[q];
        }
        if (!any) continue;
        float ns[4];
        int nw[4];
        bool plain = true;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            // (the approximate quotient's error is two ulps)
            const float sdf = fminf(1.0f, d[q] * inv_trunc), wf = IO::wtf(v[q]);
            const int wt = IO::wt(v[q]);
            const float up = SIGN > 0 ? fmaf(IO::sdf(v[q]), wf, sdf) * rcp_approx(wf + 1.0f)
                                      : fmaf(IO::sdf(v[q]), wf, -sdf) * rcp_approx(wf - 1.0f);
            if (SIGN > 0) {
                ns[q] = wt == 0 ? sdf : up;
                nw[q] = wt == 0 ? 1 : min(m.max_weight, wt + 1);
            } else {
                ns[q] = wt == 1 ? 0.0f : up;
                nw[q] = wt - 1;
            }
            plain = plain && (!ok[q] || IO::plain(ns[q]));
        }
        if (plain) {
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = ok[q] ? IO::make_plain(ns[q], nw[q]) : v[q];
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (ok[q]) v[q] = IO::make(ns[q], nw[q]);
        }
        if (sizeof(V) == 4) {
            uint4 q;
            q.x = *reinterpret_cast<unsigned *>(&v[0]);
            q.y = *reinterpret_cast<unsigned *>(&v[1]);
            q.z = *reinterpret_cast<unsigned *>(&v[2]);
            q.w = *reinterpret_cast<unsigned *>(&v[3]);
            *reinterpret_cast<uint4 *>(p) = q;
        } else {
            float4 q0, q1;
            *reinterpret_cast<V *>(&q0.x) = v[0];
            *reinterpret_cast<V *>(&q0.z) = v[1];
            *reinterpret_cast<V *>(&q1.x) = v[2];
            *reinterpret_cast<V *>(&q1.z) = v[3];
            reinterpret_cast<float4 *>(p)[0] = q0;
            reinterpret_cast<float4 *>(p)[1] = q1;
        }
    }
}

template <int SIGN>
static void launch_integrate_sign(const MapDev &m, int fmt, const float *depth, int pitch_elems, const Cam &cam,
                                  const PosePair *P, const int *skip, cudaStream_t s, int grid_ctas = 0,
                                  bool dependent = false) {
    const dim3 grid(grid_ctas > 0 ? grid_ctas : kSMs * 8);
    switch (fmt) {
        case YAS_VOXEL_F32:
            launch_kernel(integrate_kernel<YAS_VOXEL_F32, SIGN>, grid, dim3(256), s, dependent, m, depth, pitch_elems,
                          cam, P, skip);
            break;
        case YAS_VOXEL_F16:
            launch_kernel(integrate_kernel<YAS_VOXEL_F16, SIGN>, grid, dim3(256), s, dependent, m, depth, pitch_elems,
                          cam, P, skip);
            break;
        case YAS_VOXEL_S16:
            launch_kernel(integrate_kernel<YAS_VOXEL_S16, SIGN>, grid, dim3(256), s, dependent, m, depth, pitch_elems,
                          cam, P, skip);
            break;
        default:
            launch_kernel(integrate_kernel<YAS_VOXEL_S24, SIGN>, grid, dim3(256), s, dependent, m, depth, pitch_elems,
                          cam, P, skip);
            break;
    }
}

void launch_integrate(const MapDev &m, int fmt, const float *depth, int pitch_elems, const Cam &cam,
                      const PosePair *P, const int *skip, cudaStream_t s, int grid_ctas, bool dependent) {
    launch_integrate_sign<1>(m, fmt, depth, pitch_elems, cam, P, skip, s, grid_ctas, dependent);
}

void launch_deintegrate(const MapDev &m, int fmt, const float *depth, int pitch_elems, const Cam &cam,
                        const PosePair *P, cudaStream_t s, bool dependent) {
    launch_integrate_sign<-1>(m, fmt, depth, pitch_elems, cam, P, nullptr, s, 0, dependent);
}

// ---------------------------------------------------------------- reset
__global__ void reset_slots_kernel(MapDev m, unsigned block_set) {
    const unsigned n = m.slot_mask + 1;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        HashSlot s;
        s.key = kEmptyKey;
        s.ptr = -1;
        s.pad = 0;
        m.slots[i] = s;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        MapHeader h = {};
        h.block_set = block_set;
        *m.hdr = h;
    }
}

void launch_map_reset(const MapDev &m, cudaStream_t s) {
    static std::atomic<unsigned> drawn{0};
    unsigned block_set = ++drawn;
    if (block_set == 0u) block_set = ++drawn;
    reset_slots_kernel<<<kSMs * 4, 256, 0, s>>>(m, block_set);
}

// ---------------------------------------------------------------- export/import
template <int FMT>
__global__ void export_kernel(MapDev m, int *coords, float *sdf, float *wt, unsigned first,
                              unsigned count) {
    typedef VoxelIO<FMT> IO;
    const typename IO::T *vox = static_cast<const typename IO::T *>(m.voxels);
    for (unsigned j = blockIdx.x; j < count; j += gridDim.x) {
        unsigned b = first + j;
        if (threadIdx.x == 0) {
            int x, y, z;
            unpack_key(m.block_keys[b], x, y, z);
            coords[3 * j + 0] = x;
            coords[3 * j + 1] = y;
            coords[3 * j + 2] = z;
        }
        for (int i = threadIdx.x; i < kBlockVoxels; i += blockDim.x) {
            typename IO::T v = vox[(size_t)b * kBlockVoxels + i];
            sdf[(size_t)j * kBlockVoxels + i] = IO::sdf(v);
            wt[(size_t)j * kBlockVoxels + i] = (float)IO::wt(v);
        }
    }
}

void launch_map_export(const MapDev &m, int fmt, int *coords, float *sdf, float *wt, unsigned first,
                       unsigned count, cudaStream_t s) {
    if (count == 0) return;
    unsigned grid = count < 4096 ? count : 4096;
    if (fmt == YAS_VOXEL_F32)
        export_kernel<YAS_VOXEL_F32><<<grid, 128, 0, s>>>(m, coords, sdf, wt, first, count);
    else if (fmt == YAS_VOXEL_F16)
        export_kernel<YAS_VOXEL_F16><<<grid, 128, 0, s>>>(m, coords, sdf, wt, first, count);
    else if (fmt == YAS_VOXEL_S16)
        export_kernel<YAS_VOXEL_S16><<<grid, 128, 0, s>>>(m, coords, sdf, wt, first, count);
    else
        export_kernel<YAS_VOXEL_S24><<<grid, 128, 0, s>>>(m, coords, sdf, wt, first, count);
}

// One warp per imported block: lane 0 claims the slot and a pool index.
template <int FMT>
__global__ void import_kernel(MapDev m, const int *coords, const float *sdf, const float *wt,
                              unsigned count) {
    typedef VoxelIO<FMT> IO;
    typename IO::T *vox = static_cast<typename IO::T *>(m.voxels);
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;
    for (unsigned j = warp; j < count; j += nwarps) {
        int x = coords[3 * j], y = coords[3 * j + 1], z = coords[3 * j + 2];
        int b = -1;
        if (lane_id() == 0) {
            if (!coord_in_range(x, y, z)) {
                raise_error(m, YAS_ERR_COORD_RANGE);
            } else {
                unsigned long long key = pack_key(x, y, z);
                unsigned slot;
                int c = claim_slot(m, key, &slot);
                if (c == 1) {
                    unsigned idx = atomicAdd(&m.hdr->n_alloc, 1u);
                    if (idx < (unsigned)m.max_blocks) {
                        m.block_keys[idx] = key;
                        m.slots[slot].ptr = (int)idx;
                        b = (int)idx;
                    } else {
                        raise_error(m, YAS_ERR_POOL_FULL);
                    }
                } else if (c == 0) {
                    // Existing block: overwrite its contents. Its ptr was set by an
                    // earlier kernel, so the plain read is complete.
                    b = find_block(m, key);
                } else {
                    raise_error(m, YAS_ERR_TABLE_FULL);
                }
            }
        }
        b = __shfl_sync(0xffffffffu, b, 0);
        if (b < 0) continue;
        for (int i = lane_id(); i < kBlockVoxels; i += 32) {
            float s = sdf[(size_t)j * kBlockVoxels + i];
            int w = (int)wt[(size_t)j * kBlockVoxels + i];
            vox[(size_t)b * kBlockVoxels + i] = IO::make(s, w);
        }
    }
}

void launch_map_import(const MapDev &m, int fmt, const int *coords, const float *sdf, const float *wt,
                       unsigned count, cudaStream_t s) {
    if (count == 0) return;
    if (fmt == YAS_VOXEL_F32)
        import_kernel<YAS_VOXEL_F32><<<256, 256, 0, s>>>(m, coords, sdf, wt, count);
    else if (fmt == YAS_VOXEL_F16)
        import_kernel<YAS_VOXEL_F16><<<256, 256, 0, s>>>(m, coords, sdf, wt, count);
    else if (fmt == YAS_VOXEL_S16)
        import_kernel<YAS_VOXEL_S16><<<256, 256, 0, s>>>(m, coords, sdf, wt, count);
    else
        import_kernel<YAS_VOXEL_S24><<<256, 256, 0, s>>>(m, coords, sdf, wt, count);
}

__global__ void visible_coords_kernel(MapDev m, int *coords, unsigned count) {
    for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += gridDim.x * blockDim.x) {
        int x, y, z;
        unpack_key(m.block_keys[m.visible[j]], x, y, z);
        coords[3 * j] = x;
        coords[3 * j + 1] = y;
        coords[3 * j + 2] = z;
    }
}

void launch_visible_coords(const MapDev &m, int *coords, unsigned count, cudaStream_t s) {
    if (count == 0) return;
    visible_coords_kernel<<<(count + 255) / 256, 256, 0, s>>>(m, coords, count);
}

// ---------------------------------------------------------------- device memory
MapDev map_view(const yas_map *m) {
    MapDev d;
    d.slots = m->slots;
    d.slot_mask = m->slot_mask;
    d.block_keys = m->block_keys;
    d.voxels = m->voxels;
    d.visible = m->visible;
    d.hdr = m->hdr;
    d.max_blocks = m->cfg.max_blocks;
    d.voxel_size = m->cfg.voxel_size;
    d.trunc = m->cfg.trunc_dist;
    d.depth_min = m->cfg.depth_min;
    d.depth_max = m->cfg.depth_max;
    d.max_weight = m->cfg.max_weight;
    return d;
}

int map_dev_alloc(yas_map *m) {
    const size_t nslots = (size_t)m->cfg.hash_slots;
    if (cudaMalloc(&m->slots, nslots * sizeof(HashSlot)) != cudaSuccess ||
        cudaMalloc(&m->block_keys, (size_t)m->cfg.max_blocks * sizeof(unsigned long long)) !=
            cudaSuccess ||
        cudaMalloc(&m->voxels, m->voxel_bytes()) != cudaSuccess ||
        cudaMalloc(&m->visible, (size_t)m->cfg.max_blocks * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&m->hdr, sizeof(MapHeader)) != cudaSuccess) {
        cudaGetLastError();
        map_dev_free(m);
        return YAS_ERR_OOM;
    }
    m->slot_mask = (unsigned)(nslots - 1);
    return YAS_OK;
}

void map_dev_free(yas_map *m) {
    cudaFree(m->slots);
    cudaFree(m->block_keys);
    cudaFree(m->voxels);
    cudaFree(m->visible);
    cudaFree(m->hdr);
    m->slots = nullptr;
    m->block_keys = nullptr;
    m->voxels = nullptr;
    m->visible = nullptr;
    m->hdr = nullptr;
}

}  // namespace yas
