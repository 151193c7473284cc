// raycast.cu — TSDF raycasting into a camera-frame vertex map.
//
// Reference semantics (paths relative to the reference project root):
//   z-range tiles  RGBDFusion/src/RayTraceEngine.cu:58-214 (RenderingBlockDelegate,
//                  FillRenderingBlockFunctor): every visible block's 8 corners are
//                  projected to an (W/8)x(H/8) grid; each covered cell keeps the
//                  min near / max far depth of the blocks covering it.
//   ray march      RayTraceEngine.cu:266-410 (MapRenderingDelegate): march from the
//                  cell's near to far depth in voxel units with step
//                  max(sdf * trunc/voxel, 1) (1 when the sample is unobserved),
//                  trilinear sampling when |sdf| <= 0.5, stop at sdf <= 0, then two
//                  correction moves of sdf * trunc/voxel with one trilinear
//                  re-sample between them.
//
// GB300 design: the z-range fill walks each visible block's footprint with
// integer atomicMin/atomicMax on the float bit patterns (depths are positive,
// so integer order equals float order) instead of CAS loops over split tiles;
// a ray looks its blocks up in a dense grid of pool indices made for the view
// and keeps the last one, so consecutive samples inside one 8^3 block cost one
// 4- or 8-byte load each.  Per raycast (warm, events around the kernel; before:
// hash lookups, image order, 32 rays a warp): 640x480, 5 mm F16 122 -> 79 us,
// 1280x720, 4 mm F16 241 -> 166, 320x240, 8 mm F32 77 -> 50, 160x120, 1 cm F32
// 72 -> 38.  A map that has been tracked against for long takes more: its rays
// cross the layers that drift left (at 640x480, 5 mm after 1000 frames 38
// samples a ray instead of 11, 10 of them interpolated).  There the warps are
// bound by the instructions of an iteration, whose lanes look up, jump and
// interpolate in turn (14 of 32 active, 63% of the issue slots), and the last by
// the chain of the longest rays; floors without conversion instructions, the
// neighbours of a cell read side by side, and packed lerps take such a raycast
// (its other kernels included) from 264 to 218 us, a new map's from 115 to 109,
// 1280x720, 4 mm after 600 frames from 420 to 371.  Not kept: interpolated samples
// handed round the warp four lanes each (242 us), steps until most lanes
// interpolate (286 and more), 16 or 8 rays a warp for the long ones (262, 329),
// tiles in the order of the last raycast's sample counts (213, but 91 instead
// of 84 us at 320x240).
// Deliberate differences: a missed ray writes w = -1 (the reference leaves w
// stale on its early return, RayTraceEngine.cu:338-347); the 8 trilinear
// corners are floor(p) + {0,1}^3 (the reference floors p + offset per corner).
#include <algorithm>
#include <cfloat>
#include <climits>

#include "pure.h"
#include "yas_internal.h"

namespace yas {

// Block grid of a raycast: a cell for each of the kGridSide^3 blocks around the
// middle of the view, which rays look their blocks up in instead of the hash
// table.  A cell holds epoch << 24 | pool index; one of another epoch is an
// unallocated block.  Raycast e of the 255 epochs clears slice e of the cells before
// it fills its own, so that none keeps an epoch until that comes again (all of them
// at once, every 255th raycast of 160x120 took 107 us instead of 57).
// Most lookups of a long ray are of unallocated blocks (59 of 74 samples of the
// longest 2000 rays at 640x480, 5 mm): in the table each a 64-bit hash and a read
// of a random line of 16-32 MB, here a few index instructions and a line that
// neighbouring rays share.  (A bit per block in
// front of the cells, kept by the ray per 4x4x4 blocks, saved reads but cost
// more in instructions: 174 against 161 us at 1280x720, 4 mm.)  Blocks outside
// the grid, and those whose index does not fit 24 bits (kGridAsk), are looked
// up in the table; all of them where there is no grid (no memory for one).
// info: first block x, y, z; epoch; epoch of the next raycast; the map's block_set
// and n_alloc when it was filled.  A march that finds another set in the map,
// as after an import, a Fuse or a reset between a session's frames, looks all its
// blocks up in the table: the comparison is made on the GPU, in the stream's order,
// whoever changed the map (640x480, 5 mm, a frame after a block was imported: 456 us
// by the table, 425 by a new grid).
constexpr int kGridInfo = 8;
constexpr int kGridEpochs = 255;
constexpr int kGridSlice = (kGridCells / 4 + kGridEpochs - 1) / kGridEpochs;  // 16-byte words

__device__ __forceinline__ int grid_cell(int x, int y, int z) { return (z * kGridSide + y) * kGridSide + x; }
__device__ __forceinline__ bool grid_holds(int x, int y, int z) {
    return max(max((unsigned)x, (unsigned)y), (unsigned)z) < (unsigned)kGridSide;
}

// Opens an epoch: the grid is centred half way along the depth range, at most
// 64 blocks ahead of the camera.  (grid_fill, the next kernel, writes info[4].)
__device__ __forceinline__ void grid_begin(const MapDev &m, const Rigid32 &T, const BlockGrid &g) {
    if (!g.cells) return;
    const int next = g.info[4], epoch = next < 1 || next > kGridEpochs ? 1 : next;
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    const int end = min(epoch * kGridSlice, kGridCells / 4);
    for (int i = (epoch - 1) * kGridSlice + i0; i < end; i += stride)
        reinterpret_cast<uint4 *>(g.cells)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (i0 == 0) {
        const float side = m.voxel_size * (float)kBlockSide;
        const float3 c = rigid_fast(T, 0.0f, 0.0f, fminf(0.5f * m.depth_max, 64.0f * side));
        const float lim = 1.0e8f;  // far outside the key range
        g.info[0] = (int)floorf(fmaxf(-lim, fminf(lim, c.x / side))) - kGridSide / 2;
        g.info[1] = (int)floorf(fmaxf(-lim, fminf(lim, c.y / side))) - kGridSide / 2;
        g.info[2] = (int)floorf(fmaxf(-lim, fminf(lim, c.z / side))) - kGridSide / 2;
        g.info[3] = epoch;
        g.info[5] = 0;  // of no block set until it is filled
    }
}

__device__ __forceinline__ void grid_fill(const MapDev &m, const BlockGrid &g) {
    if (!g.cells) return;
    const int ox = g.info[0], oy = g.info[1], oz = g.info[2];
    const unsigned epoch = (unsigned)g.info[3] << 24, n = num_blocks(m);
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int x, y, z;
        unpack_key(m.block_keys[i], x, y, z);
        x -= ox, y -= oy, z -= oz;
        if (grid_holds(x, y, z)) g.cells[grid_cell(x, y, z)] = epoch | min(i, kGridAsk);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        g.info[4] = g.info[3] + 1;
        g.info[5] = (int)m.hdr->block_set;
        g.info[6] = (int)m.hdr->n_alloc;
    }
}

__device__ __forceinline__ void zrange_reset(const MapDev &m, const Rigid32 &T, float *znear, float *zfar, int n,
                                             unsigned *queue, float *fnear, int nf, const BlockGrid &g) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        znear[i] = 100.0f;
        zfar[i] = 0.0f;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x) fnear[i] = 100.0f;
    if (blockIdx.x == 0 && threadIdx.x == 0) *queue = 0u;
    grid_begin(m, T, g);
}

__global__ void zrange_reset_kernel(MapDev m, const PosePair *P, float *znear, float *zfar, int n, unsigned *queue,
                                    float *fnear, int nf, BlockGrid g) {
    zrange_reset(m, P->T, znear, zfar, n, queue, fnear, nf, g);
}

// zrange_reset and pose_begin (map.cu) in one launch.
__global__ void raycast_begin_kernel(MapDev m, PosePair pose, PosePair *P, float *znear, float *zfar, int n,
                                     unsigned *queue, float *fnear, int nf, BlockGrid g) {
    release_dependents();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *P = pose;
        m.hdr->n_visible = 0u;
    }
    zrange_reset(m, pose.T, znear, zfar, n, queue, fnear, nf, g);
}

__global__ void __launch_bounds__(256) grid_begin_kernel(MapDev m, const PosePair *P, BlockGrid g) {
    grid_begin(m, P->T, g);
}

__global__ void __launch_bounds__(256) grid_fill_kernel(MapDev m, BlockGrid g) {
    grid_fill(m, g);
}

__device__ __forceinline__ int clamp_floor(float v) {
    if (!(v > -1.0e6f)) return -1000000;
    if (v > 1.0e6f) return 1000000;
    return (int)floorf(v);
}
__device__ __forceinline__ int clamp_ceil(float v) {
    if (!(v > -1.0e6f)) return -1000000;
    if (v > 1.0e6f) return 1000000;
    return (int)ceilf(v);
}

// The tiles of every visible block: eight lanes a block, one corner each, which
// then share the block's cells (4x2 at a time).  Bound by its chain of
// latencies and atomics; one thread a block did 8 projections and some 40
// atomics one after the other, and counted its tiles on one shared counter
// (with the reset, 13 k blocks at 640x480, 5 mm: 15.5 -> 12.5 us, with the
// block grid's fill in it now).
__global__ void __launch_bounds__(128) zrange_fill_kernel(MapDev m, Cam cam, const PosePair *P,
                                                          float *znear, float *zfar, int zw, int zh,
                                                          const int *skip, float *fnear, int fw, int fh,
                                                          BlockGrid g, unsigned *host_visible) {
    dependent_wait();
    release_dependents();
    if (skip && *skip) return;
    grid_fill(m, g);
    const unsigned nvis = *(volatile unsigned *)&m.hdr->n_visible;
    if (host_visible && blockIdx.x == 0 && threadIdx.x == 0) *host_visible = nvis;
    const Rigid32 Tinv = P->Tinv;
    const float scale = m.voxel_size * 8.0f;
    const unsigned lane = lane_id(), c = lane & 7u, shift = lane & ~7u;
    const int lx = (int)(c & 3u), ly = (int)(c >> 2);
    for (unsigned base = (blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) / 8u; base < nvis;
         base += gridDim.x * blockDim.x / 8u) {
        const unsigned j = base + lane / 8u;
        const bool have = j < nvis;
        int bx, by, bz;
        unpack_key(m.block_keys[m.visible[have ? j : base]], bx, by, bz);
        const float3 p = rigid_exact(Tinv, (float)(bx + (int)(c & 1u)) * scale, (float)(by + (int)((c >> 1) & 1u)) * scale,
                                     (float)(bz + (int)(c >> 2)) * scale);
        const float pu = cam.fx * p.x / p.z + cam.cx, pv = cam.fy * p.y / p.z + cam.cy;
        const bool behind = ((__ballot_sync(0xffffffffu, !(p.z > 1e-3f)) >> shift) & 0xffu) != 0u;
        // a NaN coordinate counts as far to the left and up, as clamp_floor has it
        const bool nan_u = ((__ballot_sync(0xffffffffu, isnan(pu)) >> shift) & 0xffu) != 0u;
        const bool nan_v = ((__ballot_sync(0xffffffffu, isnan(pv)) >> shift) & 0xffu) != 0u;
        float pu0 = fminf(pu, 1e30f), pu1 = fmaxf(pu, -1e30f), pv0 = fminf(pv, 1e30f), pv1 = fmaxf(pv, -1e30f);
        float zmin = fminf(m.depth_max, p.z), zmax = fmaxf(m.depth_min, p.z);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            pu0 = fminf(pu0, __shfl_xor_sync(0xffffffffu, pu0, o));
            pu1 = fmaxf(pu1, __shfl_xor_sync(0xffffffffu, pu1, o));
            pv0 = fminf(pv0, __shfl_xor_sync(0xffffffffu, pv0, o));
            pv1 = fmaxf(pv1, __shfl_xor_sync(0xffffffffu, pv1, o));
            zmin = fminf(zmin, __shfl_xor_sync(0xffffffffu, zmin, o));
            zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
        }
        if (!have || !(zmax >= m.depth_min)) continue;
        // Fine near bound (not a reference quantity; the march uses it only to
        // jump over samples that lie before every visible block along the ray):
        // the block's projected box widened by a pixel, or the whole image when a
        // corner is not in front of the camera.
        int fx0 = 0, fy0 = 0, fx1 = fw - 1, fy1 = fh - 1;
        if (!behind) {
            constexpr float kInvCell = 1.0f / (float)(1 << kFineShift);
            fx0 = max(fx0, clamp_floor((pu0 - 1.0f) * kInvCell));
            fy0 = max(fy0, clamp_floor((pv0 - 1.0f) * kInvCell));
            fx1 = min(fx1, clamp_floor((pu1 + 1.0f) * kInvCell));
            fy1 = min(fy1, clamp_floor((pv1 + 1.0f) * kInvCell));
        }
        const int fz = __float_as_int(fmaxf(fminf(zmin, m.depth_max), 0.0f));
        for (int y = fy0 + ly; y <= fy1; y += 2)
            for (int x = fx0 + lx; x <= fx1; x += 4) atomicMin(reinterpret_cast<int *>(fnear) + y * fw + x, fz);
        const int ulx = max(nan_u ? 0 : clamp_floor(pu0 / 8.0f), 0), uly = max(nan_v ? 0 : clamp_floor(pv0 / 8.0f), 0);
        const int lrx = min(clamp_ceil(pu1 / 8.0f), zw - 1), lry = min(clamp_ceil(pv1 / 8.0f), zh - 1);
        const int inear = __float_as_int(fmaxf(zmin, m.depth_min)), ifar = __float_as_int(zmax);
        for (int y = uly + ly; y <= lry; y += 2)
            for (int x = ulx + lx; x <= lrx; x += 4) {
                atomicMin(reinterpret_cast<int *>(znear) + y * zw + x, inear);
                atomicMax(reinterpret_cast<int *>(zfar) + y * zw + x, ifar);
            }
    }
}

// No epoch and no block set: the next raycast begins with epoch 1.  (The fill runs on
// the legacy stream, which the raycaster's non-blocking stream does not wait for.)
static bool grid_forget(const BlockGrid &g) {
    return cudaMemset(g.info, 0, kGridInfo * sizeof(int)) == cudaSuccess &&
           cudaStreamSynchronize(cudaStreamLegacy) == cudaSuccess;
}

int raycast_buffers_alloc(RaycastBuffers &rb, int width, int height) {
    rb.w = width;
    rb.h = height;
    rb.zw = (width + 7) / 8;
    rb.zh = (height + 7) / 8;
    rb.fw = (width + (1 << kFineShift) - 1) >> kFineShift;
    rb.fh = (height + (1 << kFineShift) - 1) >> kFineShift;
    const size_t nz = (size_t)rb.zw * rb.zh;
    if (cudaMalloc(&rb.znear, nz * 4) != cudaSuccess || cudaMalloc(&rb.zfar, nz * 4) != cudaSuccess ||
        cudaMalloc(&rb.queue, sizeof(unsigned)) != cudaSuccess ||
        cudaMalloc(&rb.fnear, (size_t)rb.fw * rb.fh * 4) != cudaSuccess ||
        cudaMalloc(&rb.grid.info, kGridInfo * sizeof(int)) != cudaSuccess) {
        cudaGetLastError();
        return YAS_ERR_OOM;
    }
    return grid_forget(rb.grid) ? YAS_OK : YAS_ERR_CUDA;
}

void block_grid_alloc(BlockGrid &g) {
    if (g.cells) return;
    unsigned *cells = nullptr;
    if (cudaMalloc(&cells, kGridBytes) != cudaSuccess || cudaMemset(cells, 0, kGridBytes) != cudaSuccess ||
        !grid_forget(g)) {
        cudaGetLastError();
        cudaFree(cells);
        return;
    }
    g.cells = cells;
}

void block_grid_free(BlockGrid &g) {
    cudaFree(g.cells);
    g.cells = nullptr;
}

void raycast_buffers_free(RaycastBuffers &rb) {
    cudaFree(rb.znear);
    cudaFree(rb.zfar);
    cudaFree(rb.queue);
    cudaFree(rb.fnear);
    cudaFree(rb.grid.cells);
    cudaFree(rb.grid.info);
    rb = RaycastBuffers{};
}

void launch_zrange(const MapDev &m, const Cam &cam, const PosePair *P, RaycastBuffers &rb,
                   const int *skip, cudaStream_t s) {
    const int n = rb.zw * rb.zh, nf = rb.fw * rb.fh;
    zrange_reset_kernel<<<(std::max({n, nf, kGridSlice}) + 255) / 256, 256, 0, s>>>(m, P, rb.znear, rb.zfar, n, rb.queue, rb.fnear,
                                                                      nf, rb.grid);
    zrange_fill_kernel<<<kSMs * 8, 128, 0, s>>>(m, cam, P, rb.znear, rb.zfar, rb.zw, rb.zh, skip, rb.fnear, rb.fw,
                                               rb.fh, rb.grid, nullptr);
}

void launch_block_grid(const MapDev &m, const PosePair *P, const RaycastBuffers &rb, cudaStream_t s) {
    grid_begin_kernel<<<kSMs, 256, 0, s>>>(m, P, rb.grid);
    grid_fill_kernel<<<kSMs, 256, 0, s>>>(m, rb.grid);
}

// floor(x) and its integer.  NEAR: |x| < 2^22, by one sum rounded down (the
// conversion instructions run at a quarter of the rate).
constexpr float kFloorShift = 12582912.0f;  // 1.5 x 2^23
template <bool NEAR>
__device__ __forceinline__ float floor_of(float x, int &i) {
    if (NEAR) {
        const float k = __fadd_rd(x, kFloorShift);
        i = __float_as_int(k) - 0x4b400000;
        return __fsub_rn(k, kFloorShift);
    }
    const float f = floorf(x);
    i = (int)f;
    return f;
}
template <bool NEAR>
__device__ __forceinline__ int ifloor_of(float x) {
    int i;
    floor_of<NEAR>(x, i);
    return i;
}

// The reference's lerp (1 - t) a + t b of a pair.
__device__ __forceinline__ float2 mix2(float2 a, float2 b, float t) {
    return cfma2(pair(1.0f - t), a, cmul2(pair(t), b));
}

// Reads of one ray.  What the kernels of the same raycast write (grid, z-range
// tiles) is read by plain loads: a march that starts beside the last of them
// (dependent_wait) may not read it through the read-only path, which is for memory
// that nothing writes while the kernel lasts.  Voxels and the table are older.
template <int FMT>
struct RayReader {
    typedef VoxelIO<FMT> IO;
    typedef typename IO::T V;
    const MapDev &m;
    const BlockGrid &g;
    const V *vox;
    int ox, oy, oz;  // the grid's first block (ox: far below every block when it shows another block set)
    unsigned epoch;  // and its epoch << 24

    __device__ __forceinline__ RayReader(const MapDev &mm, const BlockGrid &gg)
        : m(mm), g(gg), vox(static_cast<const V *>(mm.voxels)) {
        const int4 at = reinterpret_cast<const int4 *>(gg.info)[0], of = reinterpret_cast<const int4 *>(gg.info)[1];
        const uint2 now = *reinterpret_cast<const uint2 *>(mm.hdr);  // n_alloc, block_set
        const bool same = gg.cells && (unsigned)of.z == now.x && (unsigned)of.y == now.y;
        ox = same ? at.x : INT_MIN / 2;
        oy = at.y;
        oz = at.z;
        epoch = (unsigned)at.w << 24;
    }

    // Pool index of block (x, y, z), or -1.
    __device__ __forceinline__ int lookup(int x, int y, int z) const {
        const int gx = x - ox, gy = y - oy, gz = z - oz;
        if (grid_holds(gx, gy, gz)) {
            const unsigned w = g.cells[grid_cell(gx, gy, gz)] - epoch;  // below 2^24 in this epoch only
            if (w != kGridAsk) return w < kGridAsk ? (int)w : -1;
        }
        return find_block_xyz(m, x, y, z);
    }
    // voxel (vx,vy,vz) of pool block b
    __device__ __forceinline__ V at(int b, int vx, int vy, int vz) const {
        return __ldg(vox + (size_t)b * kBlockVoxels + ((vz & 7) << 6) + ((vy & 7) << 3) + (vx & 7));
    }
    // sdf of a voxel word; ok is cleared when it is unobserved (weight 0)
    __device__ __forceinline__ float value(V v, bool &ok) const {
        if (IO::wt(v) == 0) {
            ok = false;
            return 1.0f;
        }
        return IO::sdf(v);
    }
    // Trilinear sample at p, whose block (bx, by, bz) has pool index b, with the
    // reference's lerp order (RayTraceEngine.cu:297-329).  Corner c of the 2x2x2
    // cell lies in neighbour c & across, across the set of axes on which the cell
    // straddles a block face (a third of the cells straddle one): their lanes read
    // the seven corners' grid words side by side; only at the grid's border, or
    // for a block that the grid leaves to the table, they look up one by one.
    template <bool NEAR>
    __device__ __forceinline__ float interp(float3 p, int bx, int by, int bz, int b, bool &valid) const {
        int x0, y0, z0;
        const float ax = p.x - floor_of<NEAR>(p.x, x0), ay = p.y - floor_of<NEAR>(p.y, y0);
        const float az = p.z - floor_of<NEAR>(p.z, z0);
        const unsigned across = ((x0 & 7) == 7 ? 1u : 0u) | ((y0 & 7) == 7 ? 2u : 0u) | ((z0 & 7) == 7 ? 4u : 0u);
        unsigned q[8], lim = 0x80000000u;  // pool index of each corner's block (lim or above: unallocated)
#pragma unroll
        for (int c = 0; c < 8; ++c) q[c] = (unsigned)b;
        if (across != 0u) {
            const int gx = bx - ox, gy = by - oy, gz = bz - oz;
            const bool inner = max(max((unsigned)gx, (unsigned)gy), (unsigned)gz) < (unsigned)(kGridSide - 1);
            const unsigned *cell = g.cells + (inner ? grid_cell(gx, gy, gz) : 0);
            const int sx = across & 1u, sy = across & 2u ? kGridSide : 0, sz = across & 4u ? kGridSide * kGridSide : 0;
            lim = corner_blocks(
                across, b, inner,
                [&](unsigned c) { return cell[(c & 1 ? sx : 0) + (c & 2 ? sy : 0) + (c & 4 ? sz : 0)] - epoch; },
                [&](unsigned d) { return lookup(bx + (int)(d & 1u), by + (int)((d >> 1) & 1u), bz + (int)(d >> 2)); }, q);
        }
        const int xo[2] = {x0 & 7, (x0 + 1) & 7}, yo[2] = {(y0 & 7) << 3, ((y0 + 1) & 7) << 3};
        const int zo[2] = {(z0 & 7) << 6, ((z0 + 1) & 7) << 6};
        V v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c)
            v[c] = q[c] < lim ? __ldg(vox + (size_t)q[c] * kBlockVoxels + (zo[c >> 2] + yo[(c >> 1) & 1] + xo[c & 1]))
                                : IO::make(1.0f, 0);
        bool ok = true;
        float s[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) s[c] = value(v[c], ok);
        valid = ok;
        // two at a time: the upper and lower plane side by side
        const float2 r0 = mix2(make_float2(s[0], s[4]), make_float2(s[1], s[5]), ax);
        const float2 r1 = mix2(make_float2(s[2], s[6]), make_float2(s[3], s[7]), ax);
        const float2 r2 = mix2(r0, r1, ay);
        return fmaf(1.0f - az, r2.x, __fmul_rn(az, r2.y));
    }
};

// State of one ray of the march (RayTraceEngine.cu:331-410), in voxel units.
struct RayState {
    float3 r, dir, idir;
    float dist_s, dist_e, sdf;
};

// Ray of pixel (x, y) between the tile's z-range bounds zn..zf; false when the
// tile has no range (the pixel is a miss).  zfine: the nearest visible block
// whose projected box covers the pixel's 4x4 neighbourhood.  The march starts
// at zn as the reference's does; every sample before zfine lies outside every
// visible block, reads "unobserved" and advances one voxel, so those samples
// are taken in one move (two are kept as margin against rounding).
__device__ __forceinline__ bool ray_setup(const Cam &cam, const Rigid32 &T, float vsinv, float zn, float zf,
                                          float zfine, int x, int y, RayState &R) {
    if (zn < FLT_EPSILON || zf < FLT_EPSILON || isnan(zn) || isnan(zf)) return false;
    const float ux = cam.invfx * ((float)x - cam.cx), uy = cam.invfy * ((float)y - cam.cy);
    const float3 pn = make_float3(ux * zn, uy * zn, zn);
    R.dist_s = sqrtf(pn.x * pn.x + pn.y * pn.y + pn.z * pn.z) * vsinv;
    float3 s = rigid_fast(T, pn.x, pn.y, pn.z);
    s = make_float3(s.x * vsinv, s.y * vsinv, s.z * vsinv);
    const float3 pf = make_float3(ux * zf, uy * zf, zf);
    R.dist_e = sqrtf(pf.x * pf.x + pf.y * pf.y + pf.z * pf.z) * vsinv;
    float3 e = rigid_fast(T, pf.x, pf.y, pf.z);
    e = make_float3(e.x * vsinv, e.y * vsinv, e.z * vsinv);
    float3 dir = make_float3(e.x - s.x, e.y - s.y, e.z - s.z);
    const float dn = sqrtf(dir.x * dir.x + dir.y * dir.y + dir.z * dir.z);
    if (dn > 0.0f) dir = make_float3(dir.x / dn, dir.y / dn, dir.z / dn);
    R.r = s;
    R.dir = dir;
    R.idir = make_float3(dir.x != 0.0f ? -1.0f / fabsf(dir.x) : 1.0f, dir.y != 0.0f ? -1.0f / fabsf(dir.y) : 1.0f,
                         dir.z != 0.0f ? -1.0f / fabsf(dir.z) : 1.0f);
    R.sdf = 1.0f;
    if (zfine > zn) {
        const float k = sqrtf(ux * ux + uy * uy + 1.0f) * vsinv;  // voxels of ray per metre of depth
        const float n = floorf(fminf(zfine * k, R.dist_e) - R.dist_s) - 2.0f;
        if (n >= 1.0f) {
            R.r = make_float3(R.r.x + n * dir.x, R.r.y + n * dir.y, R.r.z + n * dir.z);
            R.dist_s += n;
        }
    }
    return true;
}

// Every sample of the march lies within 2^22 voxels of the origin (no NaN).
__device__ __forceinline__ bool ray_near(const RayState &R) {
    return fabsf(R.r.x) < 2097152.0f && fabsf(R.r.y) < 2097152.0f && fabsf(R.r.z) < 2097152.0f &&
           R.dist_e - R.dist_s < 1048576.0f && R.dir.x + R.dir.y + R.dir.z < 4.0f;
}

// R.r n steps on.
__device__ __forceinline__ float3 at_step(const RayState &R, float n) {
    const float2 xy = cfma2(pair(n), make_float2(R.dir.x, R.dir.y), make_float2(R.r.x, R.r.y));
    return make_float3(xy.x, xy.y, fmaf(n, R.dir.z, R.r.z));
}

// One axis of a ray in an unallocated block whose lower face is at x0.  `face`
// is the face that the ray leaves through (1e30 for a ray parallel to the
// axis: none); the result is the steps to the first sample at or past it (the
// upper face is outside the block, the lower one inside): the quotient rounded
// up for a rising ray, the next whole number above it for a falling one.  idir
// is -1 / |dir| (1 for a parallel ray): a rising ray's quotient is negative.
template <bool NEAR>
__device__ __forceinline__ float exit_steps(float x0, float r, float dir, float idir, float &face) {
    const bool falls = dir < 0.0f;
    face = x0 + (falls ? 0.0f : (dir > 0.0f ? 8.0f : 1e30f));
    const float u = (face - r) * idir;
    return fabsf(NEAR ? __fsub_rn(__fadd_rd(u, kFloorShift), kFloorShift) : floorf(u)) + (falls ? 1.0f : 0.0f);
}
// p is outside the block on that axis (it came from inside along dir).
__device__ __forceinline__ bool past(float p, float dir, float face) { return (p >= face) != (dir < 0.0f); }

// Samples to the first one past the unallocated block that holds the sample at
// R.r (its lower corner at x0, y0, z0): every sample until the ray leaves the
// block reads "unobserved" and advances one voxel, so they are taken in one
// move.  k = steps to the first sample outside on the earliest exit axis.  When
// sample k - 1 (computed as the move computes it) is still in the block and
// sample k is not, the move goes straight to sample k; otherwise (k rounded
// the wrong way) it keeps two samples as margin, at least one step.
template <bool NEAR>
__device__ __forceinline__ float empty_steps(const RayState &R, float x0, float y0, float z0) {
    float fx, fy, fz;
    const float kx = exit_steps<NEAR>(x0, R.r.x, R.dir.x, R.idir.x, fx), ky = exit_steps<NEAR>(y0, R.r.y, R.dir.y, R.idir.y, fy);
    const float kz = exit_steps<NEAR>(z0, R.r.z, R.dir.z, R.idir.z, fz);
    const float k = fminf(fminf(kx, ky), kz);
    const float3 p = at_step(R, k - 1.0f), q = at_step(R, k);
    const bool in = !(past(p.x, R.dir.x, fx) || past(p.y, R.dir.y, fy) || past(p.z, R.dir.z, fz));
    const bool out = past(q.x, R.dir.x, fx) || past(q.y, R.dir.y, fy) || past(q.z, R.dir.z, fz);
    const float n = k >= 1.0f && k < 1e29f && in && out ? k : k - 2.0f;
    const float left = R.dist_e - R.dist_s;
    return fmaxf(fminf(n, NEAR ? __fsub_rn(__fadd_ru(left, kFloorShift), kFloorShift) : ceilf(left)), 1.0f);
}

// The march loop, to a sample with sdf <= 0 or the end of the ray's range.
template <int FMT, bool NEAR>
__device__ __forceinline__ void ray_march(const RayReader<FMT> &rd, float rstep, RayState &R) {
    int bx = INT_MIN, by = 0, bz = 0;  // the block of the sample at R.r
    int cptr = -1;                     // its pool index (-1: unallocated)
    bool jumped = false;               // the ray has taken its jump out of that (unallocated) block
    while (R.dist_s < R.dist_e) {
        float n = 1.0f;
        const int vx = ifloor_of<NEAR>(R.r.x), vy = ifloor_of<NEAR>(R.r.y), vz = ifloor_of<NEAR>(R.r.z);
        const int x = vx >> 3, y = vy >> 3, z = vz >> 3;
        if (x != bx || y != by || z != bz) {
            bx = x, by = y, bz = z;
            jumped = false;
            cptr = rd.lookup(x, y, z);
        }
        if (cptr < 0) {
            if (!jumped) n = empty_steps<NEAR>(R, (float)(vx & ~7), (float)(vy & ~7), (float)(vz & ~7));
            jumped = true;
        } else {
            bool valid = true;
            R.sdf = rd.value(rd.at(cptr, vx, vy, vz), valid);
            if (R.sdf <= 0.5f && R.sdf >= -0.5f) R.sdf = rd.template interp<NEAR>(R.r, bx, by, bz, cptr, valid);
            if (R.sdf <= 0.0f) return;
            if (valid) n = fmaxf(R.sdf * rstep, 1.0f);
        }
        R.r = at_step(R, n);
        R.dist_s += n;
    }
}

// Vertex of a finished ray: a hit takes two interpolated correction steps
// and is returned in camera coordinates (w = 1); a miss is NaN with w = -1.
// (Its floors are the general ones: a stored sdf may move the ray anywhere.)
template <int FMT>
__device__ __forceinline__ float4 ray_finish(const RayReader<FMT> &rd, float rstep, float vsinv, const Rigid32 &Ti,
                                             RayState &R) {
    float4 out = make_float4(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff), __int_as_float(0x7fffffff),
                             -1.0f);
    if (R.sdf <= 0.0f) {
        float step = R.sdf * rstep;
        R.r.x += step * R.dir.x;
        R.r.y += step * R.dir.y;
        R.r.z += step * R.dir.z;
        const int x = (int)floorf(R.r.x) >> 3, y = (int)floorf(R.r.y) >> 3, z = (int)floorf(R.r.z) >> 3;
        const int b = rd.lookup(x, y, z);
        bool valid = false;
        R.sdf = b >= 0 ? rd.template interp<false>(R.r, x, y, z, b, valid) : 1.0f;
        step = R.sdf * rstep;
        R.r.x += step * R.dir.x;
        R.r.y += step * R.dir.y;
        R.r.z += step * R.dir.z;
        if (valid) {
            const float3 w = make_float3(R.r.x / vsinv, R.r.y / vsinv, R.r.z / vsinv);
            const float3 c = rigid_fast(Ti, w.x, w.y, w.z);
            out = make_float4(c.x, c.y, c.z, 1.0f);
        }
    }
    return out;
}

// The pixel (x, y) of each lane of a warp (outside the image: none).  `turn` 0:
// only if the warp has a long ray, 1: only if it has none, -1: always.  A ray
// is long when more than kLongBlocks blocks lie between the first visible
// block in front of its pixels and the far bound of its tile.  Each tile is
// launched for both turns, the long ones in the first half of the grid: a warp
// of long rays takes most of the march's time wherever it starts.  16 blocks:
// with the raycast's other kernels, 106 us in a new map at 640x480, 5 mm and 219
// in one of 1000 frames; 24 blocks: 108 and 220, 32: 113 and 240; 8: 240 in the
// latter where 24 took 227.
constexpr float kLongBlocks = 16.0f;
template <int FMT>
__device__ __forceinline__ void march_pixel(const MapDev &m, const Cam &cam, const PosePair *P,
                                            const float *znear, const float *zfar, int zw,
                                            float4 *vmap, int vpitch, bool skipped, const float *fnear,
                                            int fw, const BlockGrid &g, int x, int y, int turn) {
    const float vsinv = 1.0f / m.voxel_size;
    const float rstep = m.trunc / m.voxel_size;
    const bool inside = x < cam.w && y < cam.h;
    RayState R;
    R.sdf = 1.0f;
    float zn = 0.0f, zf = 0.0f, zfine = 0.0f;
    if (inside && !skipped) {
        zn = znear[(y >> 3) * zw + (x >> 3)];
        zf = zfar[(y >> 3) * zw + (x >> 3)];
        zfine = fnear[(y >> kFineShift) * fw + (x >> kFineShift)];
    }
    if (turn >= 0) {
        const bool far = zf - fmaxf(zn, zfine) > kLongBlocks * (float)kBlockSide * m.voxel_size;
        if ((int)!__any_sync(0xffffffffu, far) != turn) return;
    }
    const bool live = inside && !skipped && ray_setup(cam, P->T, vsinv, zn, zf, zfine, x, y, R);
    const RayReader<FMT> rd(m, g);
    if (__all_sync(0xffffffffu, !live || ray_near(R))) {
        if (live) ray_march<FMT, true>(rd, rstep, R);
    } else {
        if (live) ray_march<FMT, false>(rd, rstep, R);
    }
    if (inside) vmap[(size_t)y * vpitch + x] = ray_finish(rd, rstep, vsinv, P->Tinv, R);
}

// Each warp a compact tile of RAYS pixels (32: 8x4, 16: 4x4, 8: 4x2), so its
// rays travel similar depths; a CTA is WX x WY warp tiles.  Warps of fewer rays
// leave lanes idle and run more instructions in all, but each warp less: the
// lanes of a warp that jump, look up and sample take turns.
template <int FMT, int WX, int WY, int RAYS>
__global__ void __launch_bounds__(32 * WX * WY) march_kernel(MapDev m, Cam cam, const PosePair *P,
                                                             const float *znear,
                                                             const float *zfar, int zw, float4 *vmap,
                                                             int vpitch, const int *skip,
                                                             const float *fnear, int fw, BlockGrid g) {
    constexpr int TX = RAYS == 32 ? 8 : 4, TY = RAYS / TX;
    dependent_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int x = lane < RAYS ? (blockIdx.x * WX + warp % WX) * TX + lane % TX : INT_MAX;
    const int y = (blockIdx.y * WY + warp / WX) * TY + lane / TX;
    march_pixel<FMT>(m, cam, P, znear, zfar, zw, vmap, vpitch, skip && *skip, fnear, fw, g, x, y, (int)blockIdx.z);
}

// Persistent march: resident warps take 8x4-pixel tiles from a queue (one
// atomic per tile on rb.queue, tiles row-major), a warp taking the next tile
// once all its rays are done, so no SM idles behind a partial last wave.
// Each ray runs exactly the steps of march_kernel, so the vertex map is the
// same bit for bit.
template <int FMT>
__global__ void __launch_bounds__(128) march_persistent_kernel(MapDev m, Cam cam, const PosePair *P,
                                                               const float *znear,
                                                               const float *zfar, int zw, float4 *vmap,
                                                               int vpitch, const int *skip,
                                                               const float *fnear, int fw,
                                                               BlockGrid g, unsigned *queue,
                                                               unsigned tiles) {
    const int lane = (int)lane_id(), tiles_x = (cam.w + 7) >> 3;
    const bool skipped = skip && *skip;
    for (;;) {
        unsigned t = 0u;
        if (lane == 0) t = atomicAdd(queue, 1u);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= tiles) return;
        const int x = (int)(t % (unsigned)tiles_x) * 8 + (lane & 7), y = (int)(t / (unsigned)tiles_x) * 4 + (lane >> 3);
        march_pixel<FMT>(m, cam, P, znear, zfar, zw, vmap, vpitch, skipped, fnear, fw, g, x, y, -1);
    }
}

static int march_resident_ctas(int fmt) {
    static int cache[4][64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || fmt < 0 || fmt > 3) return kSMs;
    int &c = cache[fmt][dev];
    if (c == 0) {
        int sms = 0, nb = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (fmt == YAS_VOXEL_F32)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, march_persistent_kernel<YAS_VOXEL_F32>, 128, 0);
        else if (fmt == YAS_VOXEL_F16)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, march_persistent_kernel<YAS_VOXEL_F16>, 128, 0);
        else if (fmt == YAS_VOXEL_S16)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, march_persistent_kernel<YAS_VOXEL_S16>, 128, 0);
        else
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, march_persistent_kernel<YAS_VOXEL_S24>, 128, 0);
        cudaGetLastError();
        c = std::max(1, nb) * std::max(1, sms);
    }
    return c;
}

static void launch_march_persistent(const MapDev &m, int fmt, const Cam &cam, const PosePair *P,
                                    const RaycastBuffers &rb, float4 *vmap, int vmap_pitch_elems, const int *skip,
                                    cudaStream_t s) {
    const unsigned tiles = (unsigned)(((cam.w + 7) / 8) * ((cam.h + 3) / 4));
    const int grid = std::min(march_resident_ctas(fmt), (int)((tiles + 3) / 4));
    switch (fmt) {
        case YAS_VOXEL_F32:
            march_persistent_kernel<YAS_VOXEL_F32><<<grid, 128, 0, s>>>(m, cam, P, rb.znear, rb.zfar, rb.zw, vmap,
                                                                        vmap_pitch_elems, skip, rb.fnear, rb.fw, rb.grid, rb.queue, tiles);
            break;
        case YAS_VOXEL_F16:
            march_persistent_kernel<YAS_VOXEL_F16><<<grid, 128, 0, s>>>(m, cam, P, rb.znear, rb.zfar, rb.zw, vmap,
                                                                        vmap_pitch_elems, skip, rb.fnear, rb.fw, rb.grid, rb.queue, tiles);
            break;
        case YAS_VOXEL_S16:
            march_persistent_kernel<YAS_VOXEL_S16><<<grid, 128, 0, s>>>(m, cam, P, rb.znear, rb.zfar, rb.zw, vmap,
                                                                        vmap_pitch_elems, skip, rb.fnear, rb.fw, rb.grid, rb.queue, tiles);
            break;
        default:
            march_persistent_kernel<YAS_VOXEL_S24><<<grid, 128, 0, s>>>(m, cam, P, rb.znear, rb.zfar, rb.zw, vmap,
                                                                        vmap_pitch_elems, skip, rb.fnear, rb.fw, rb.grid, rb.queue, tiles);
            break;
    }
}

template <int WX, int WY, int RAYS>
static void launch_march_rays(const MapDev &m, int fmt, const Cam &cam, const PosePair *P, const RaycastBuffers &rb,
                              float4 *vmap, int vmap_pitch_elems, const int *skip, cudaStream_t s, bool dependent) {
    constexpr int TX = (RAYS == 32 ? 8 : 4) * WX, TY = RAYS / (RAYS == 32 ? 8 : 4) * WY;
    const dim3 grid((cam.w + TX - 1) / TX, (cam.h + TY - 1) / TY, 2);
    const auto launch = [&](auto kernel) {
        launch_kernel(kernel, grid, dim3(32 * WX * WY), s, dependent, m, cam, P, rb.znear, rb.zfar, rb.zw, vmap,
                      vmap_pitch_elems, skip, rb.fnear, rb.fw, rb.grid);
    };
    switch (fmt) {
        case YAS_VOXEL_F32: launch(march_kernel<YAS_VOXEL_F32, WX, WY, RAYS>); break;
        case YAS_VOXEL_F16: launch(march_kernel<YAS_VOXEL_F16, WX, WY, RAYS>); break;
        case YAS_VOXEL_S16: launch(march_kernel<YAS_VOXEL_S16, WX, WY, RAYS>); break;
        default: launch(march_kernel<YAS_VOXEL_S24, WX, WY, RAYS>); break;
    }
}

template <int WX, int WY>
static void launch_march_tile(const MapDev &m, int fmt, const Cam &cam, const PosePair *P, const RaycastBuffers &rb,
                              float4 *vmap, int vmap_pitch_elems, const int *skip, cudaStream_t s,
                              bool dependent = false, bool shared = false) {
    // Rays per warp.  A small image does not fill the GPU with warps of 32 rays,
    // so a march lasts as long as its slowest warp, and that one ends sooner
    // with fewer rays; in larger images instruction issue counts, and full warps
    // take the fewest.  Whole raycasts with 8 / 16 / 32 rays a warp (us, means of
    // three scenes of four frames, the smaller of two runs each):
    //               8 mm F32            5 mm F16
    //   160x120     62 /  67 /  74      75 /  82 /  91
    //   262x196     65 /  69 /  74      73 /  78 /  83
    //   283x212     70 /  70 /  78      75 /  75 /  81
    //   320x240     72 /  70 /  75      78 /  79 /  86
    //   413x310     89 /  80 /  81      97 /  85 /  89
    //   462x346     99 /  81 /  78     109 /  87 /  88
    //   516x387    112 /  88 /  79     124 /  93 /  93
    //   640x480    142 / 103 /  86     164 / 116 /  98
    // The lines lie where neither side is better.  Marches of several sessions fill
    // the GPU beside one another and take full warps.
    const long long px = (long long)cam.w * cam.h;
    if (px <= 60000 && !shared)
        launch_march_rays<WX, WY, 8>(m, fmt, cam, P, rb, vmap, vmap_pitch_elems, skip, s, dependent);
    else if (px <= 160000 && !shared)
        launch_march_rays<WX, WY, 16>(m, fmt, cam, P, rb, vmap, vmap_pitch_elems, skip, s, dependent);
    else
        launch_march_rays<WX, WY, 32>(m, fmt, cam, P, rb, vmap, vmap_pitch_elems, skip, s, dependent);
}

void launch_march(const MapDev &m, int fmt, const Cam &cam, const PosePair *P, const RaycastBuffers &rb,
                  float4 *vmap, int vmap_pitch_elems, const int *skip, cudaStream_t s, int tile, bool shared) {
    switch (tile) {
        case 0: launch_march_persistent(m, fmt, cam, P, rb, vmap, vmap_pitch_elems, skip, s); break;
        case 1: launch_march_tile<1, 4>(m, fmt, cam, P, rb, vmap, vmap_pitch_elems, skip, s, false, shared); break;
        case 4: launch_march_tile<4, 1>(m, fmt, cam, P, rb, vmap, vmap_pitch_elems, skip, s, false, shared); break;
        default: launch_march_tile<2, 2>(m, fmt, cam, P, rb, vmap, vmap_pitch_elems, skip, s, false, shared); break;
    }
}

// Four launches where a pose copy, a memset and four kernels each waited for the
// one before, and a second synchronisation for the count.  A call, before and
// after: 640x480, 5 mm 109 / 89 us, in a map of 1000 frames 218 / 200, 320x240,
// 8 mm 86 / 69.
void launch_raycast(const MapDev &m, int fmt, const Cam &vis_cam, const Cam &cam, const PosePair &pose, PosePair *P,
                    RaycastBuffers &rb, float4 *vmap, int vmap_pitch_elems, unsigned *host_visible, cudaStream_t s) {
    const int n = rb.zw * rb.zh, nf = rb.fw * rb.fh;
    raycast_begin_kernel<<<(std::max({n, nf, kGridSlice}) + 255) / 256, 256, 0, s>>>(m, pose, P, rb.znear, rb.zfar, n, rb.queue,
                                                                       rb.fnear, nf, rb.grid);
    launch_visible(m, vis_cam, P, nullptr, s, true);
    launch_kernel(zrange_fill_kernel, dim3(kSMs * 8), dim3(128), s, true, m, cam, (const PosePair *)P, rb.znear, rb.zfar,
                  rb.zw, rb.zh, (const int *)nullptr, rb.fnear, rb.fw, rb.fh, rb.grid, host_visible);
    launch_march_tile<2, 2>(m, fmt, cam, P, rb, vmap, vmap_pitch_elems, nullptr, s, true);
}

__global__ void vmap_to_depth_kernel(const float4 *vmap, int vpitch, float *depth, int dpitch, int w,
                                     int h) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= w || y >= h) return;
    float4 v = vmap[(size_t)y * vpitch + x];
    depth[(size_t)y * dpitch + x] = v.w > 0.0f ? v.z : 0.0f;
}

void launch_vmap_to_depth(const float4 *vmap, int vpitch, float *depth, int dpitch, int w, int h,
                          cudaStream_t s) {
    dim3 grid((w + 127) / 128, h);
    vmap_to_depth_kernel<<<grid, 128, 0, s>>>(vmap, vpitch, depth, dpitch, w, h);
}

}  // namespace yas
