// mesh.cu — marching-cubes extraction over every allocated block.
//
// Reference semantics (paths relative to the reference project root):
//   RGBDFusion/src/MeshEngine.cu:43-269 (MeshificationFunctor): a cube at voxel
//   p uses corners p + {0,1}^3 in the order 0:(0,0,0) 1:(1,0,0) 2:(1,1,0)
//   3:(0,1,0) 4:(0,0,1) 5:(1,0,1) 6:(1,1,1) 7:(0,1,1); all 8 must be observed
//   (weight != 0); case bit i is set when sdf_i < 0; edge vertices use the
//   reference's interpolation with its 1e-6 guards; positions are voxel
//   coordinates times the voxel size (submap metres) and every triangle carries
//   the face normal normalize((v1-v0) x (v2-v0)).
//
// The triangle table is not the reference's table (RGBDFusion/utils/
// TriangleTable.h): it is generated here from cube topology.  For each case
// the iso-contour is traced on the six faces (each face's crossings paired so
// that inside corners stay separated on ambiguous faces), the directed face
// segments are chained into loops, and each loop is fanned from its
// lowest-numbered edge.  Segment direction keeps the inside (sdf < 0) region
// on the left seen from outside the cube, which makes every triangle's normal
// point toward the inside, the same orientation as the reference table.
//
// GB300 design: one CTA per block reads the 9x9x9 sdf neighbourhood (own block
// with 16-byte loads plus the +x/+y/+z halo from up to 7 neighbour blocks) and
// keeps, per row of 9 voxels, which are observed and which are inside as bits:
// the 8 cubes of a row then take a few logical operations instead of 64 reads.
// Pass 1 counts triangles per block, a scan assigns each block a contiguous
// output range, pass 2 lists the block's triangles in cube order and writes one
// per thread, so the output order (cube order, then table order) is a pure
// function of the map.
#include <algorithm>
#include <cstring>

#include "yas_internal.h"

namespace yas {

// ---------------------------------------------------------------- tables
constexpr int kMcMaxTriIdx = 31;  // up to 10 triangles + terminator

// The table in global memory, a word per case: the edges of its triangles (at
// most 5), 4 bits each, and the number of triangles in bits 60..63 (0 for the
// cases without crossings).  Each CTA copies it into shared memory (a
// constant-memory copy would serialise the lanes' distinct addresses).
constexpr int kMcMaxCaseTris = 5;
__device__ __align__(16) unsigned long long g_mc_table[256];

static const int kCorner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                  {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
static const int kEdge[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                 {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};

static int edge_of(int a, int b) {
    for (int e = 0; e < 12; ++e)
        if ((kEdge[e][0] == a && kEdge[e][1] == b) || (kEdge[e][0] == b && kEdge[e][1] == a)) return e;
    return -1;
}

// Corners of each face in counter-clockwise order about the outward normal.
static void face_ccw(int face, int out[4]) {
    // face: 0 x=0, 1 x=1, 2 y=0, 3 y=1, 4 z=0, 5 z=1
    const int axis = face / 2, side = face % 2;
    int cs[4], n = 0;
    for (int c = 0; c < 8; ++c)
        if (kCorner[c][axis] == side) cs[n++] = c;
    // order the 4 corners cyclically around the face centre
    const int u = (axis + 1) % 3, v = (axis + 2) % 3;
    int order[4] = {-1, -1, -1, -1};
    for (int i = 0; i < 4; ++i) {
        int cu = kCorner[cs[i]][u], cv = kCorner[cs[i]][v];
        int pos = (cu == 0 && cv == 0) ? 0 : (cu == 1 && cv == 0) ? 1 : (cu == 1 && cv == 1) ? 2 : 3;
        order[pos] = cs[i];
    }
    // (u, v, axis) is right-handed, so this order is CCW about +axis.
    if (side == 1) {
        for (int i = 0; i < 4; ++i) out[i] = order[i];
    } else {
        out[0] = order[0];
        out[1] = order[3];
        out[2] = order[2];
        out[3] = order[1];
    }
}

struct McTables {
    unsigned short edge[256];
    signed char tri[256][kMcMaxTriIdx];
    unsigned char count[256];
};

static void build_mc_tables(McTables &t) {
    memset(&t, 0, sizeof(t));
    memset(t.tri, -1, sizeof(t.tri));
    for (int c = 0; c < 256; ++c) {
        unsigned short em = 0;
        for (int e = 0; e < 12; ++e) {
            bool a = (c >> kEdge[e][0]) & 1, b = (c >> kEdge[e][1]) & 1;
            if (a != b) em |= (unsigned short)(1u << e);
        }
        t.edge[c] = em;
        if (em == 0) continue;
        int next[12];
        for (int e = 0; e < 12; ++e) next[e] = -1;
        for (int f = 0; f < 6; ++f) {
            int q[4];
            face_ccw(f, q);
            // crossings in CCW order: edge index and kind (+1 enter inside, -1 exit)
            int ce[4], kind[4], nc = 0;
            for (int i = 0; i < 4; ++i) {
                int a = q[i], b = q[(i + 1) & 3];
                bool ia = (c >> a) & 1, ib = (c >> b) & 1;
                if (ia != ib) {
                    ce[nc] = edge_of(a, b);
                    kind[nc] = ib ? +1 : -1;
                    ++nc;
                }
            }
            if (nc == 2) {
                int ex = kind[0] < 0 ? 0 : 1;
                next[ce[ex]] = ce[1 - ex];
            } else if (nc == 4) {
                // separate inside corners: each exit pairs with the previous enter
                for (int i = 0; i < 4; ++i)
                    if (kind[i] < 0) next[ce[i]] = ce[(i + 3) & 3];
            }
        }
        int ntri = 0, w = 0;
        bool used[12] = {false};
        for (int start = 0; start < 12; ++start) {
            if (!((em >> start) & 1) || used[start]) continue;
            int loop[12], k = 0, e = start;
            while (e >= 0 && !used[e] && k < 12) {
                used[e] = true;
                loop[k++] = e;
                e = next[e];
            }
            // fan from the lowest edge of the loop (start is the lowest unused)
            for (int i = 1; i + 1 < k; ++i) {
                t.tri[c][w++] = (signed char)loop[0];
                t.tri[c][w++] = (signed char)loop[i];
                t.tri[c][w++] = (signed char)loop[i + 1];
                ++ntri;
            }
        }
        t.count[c] = (unsigned char)ntri;
    }
}

void mesh_tables_upload() {
    static McTables tables;
    static bool built = false;
    if (!built) {
        build_mc_tables(tables);
        built = true;
    }
    unsigned long long words[256];
    for (int c = 0; c < 256; ++c) {
        const int n = tables.edge[c] == 0 ? 0 : std::min<int>(tables.count[c], kMcMaxCaseTris);
        words[c] = (unsigned long long)n << 60;
        for (int i = 0; i < 3 * n; ++i) words[c] |= (unsigned long long)tables.tri[c][i] << (4 * i);
    }
    cudaMemcpyToSymbol(g_mc_table, words, sizeof(words));
    // the copy runs on the legacy stream; the engines launch on
    // non-blocking streams, which do not wait for it
    cudaStreamSynchronize(cudaStreamLegacy);
}

// ---------------------------------------------------------------- staging
constexpr int kN = 9;            // staged cells per axis
constexpr int kN3 = kN * kN * kN;

// A block's 9^3 neighbourhood as bits: of row (y, z), index z * 9 + y, bit x is
// set when voxel x is observed, bit 16 + x when its sdf is negative too.
struct BlockRows {
    int nb[8];
    unsigned inner[kN * kN];  // x = 0..7
    unsigned last[kN * kN];   // x = 8
    __device__ __forceinline__ unsigned row(int y, int z) const { return inner[z * kN + y] | last[z * kN + y]; }
};

// Reads block b's neighbourhood into `rows` and, with `s`, its sdf values
// (s[z*81 + y*9 + x], meaningless where unobserved).  Called by all NT threads;
// ends with a barrier.
template <int FMT, int NT>
__device__ __forceinline__ void stage_block(const MapDev &m, int b, int bx, int by, int bz, BlockRows &rows, float *s) {
    typedef VoxelIO<FMT> IO;
    typedef typename IO::T V;
    const V *vox = static_cast<const V *>(m.voxels);
    const int t = (int)threadIdx.x, lane = t & 31;
    // the block's own 512 voxels: 16-byte loads of consecutive words (the pool
    // is 16-byte aligned and a block's words are contiguous, z*64 + y*8 + x),
    // under way while the first warp looks the neighbours up
    constexpr int kPer = 16 / (int)sizeof(V), kOwn = kBlockVoxels / kPer / NT, kLanes = 8 / kPer;
    const int4 *own = reinterpret_cast<const int4 *>(vox + (size_t)b * kBlockVoxels);
    int4 w[kOwn];
#pragma unroll
    for (int k = 0; k < kOwn; ++k) w[k] = __ldg(own + t + k * NT);
    if (t < 8) rows.nb[t] = t == 0 ? b : find_block_xyz(m, bx + (t & 1), by + ((t >> 1) & 1), bz + ((t >> 2) & 1));
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {
        const V *e = reinterpret_cast<const V *>(&w[k]);
        const int i0 = (t + k * NT) * kPer, x = i0 & 7, y = (i0 >> 3) & 7, z = i0 >> 6;
        unsigned bits = 0u;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const float v = IO::sdf(e[j]);
            if (s) s[z * 81 + y * 9 + x + j] = v;
            const bool seen = IO::wt(e[j]) != 0 && !isnan(v);
            bits |= (seen ? 1u << (x + j) : 0u) | (seen && v < 0.0f ? 0x10000u << (x + j) : 0u);
        }
#pragma unroll
        for (int o = 1; o < kLanes; o <<= 1) bits |= __shfl_xor_sync(0xffffffffu, bits, o);
        if (x == 0) rows.inner[z * kN + y] = bits;
    }
    __syncthreads();
    // the halo: 17 rows of 8 voxels (y = 8, then z = 8), then the 81 at x = 8
#pragma unroll
    for (int k = 0; k < (217 + NT - 1) / NT; ++k) {
        const int h = t + k * NT, r = h >> 3, g = h - 136;
        const bool in_row = h < 136;
        const int x = in_row ? h & 7 : 8;
        const int y = in_row ? (r < 9 ? 8 : r - 9) : g % 9, z = in_row ? (r < 9 ? r : 8) : g / 9;
        const int p = h < 217 ? rows.nb[(x >> 3) | ((y >> 3) << 1) | ((z >> 3) << 2)] : -1;
        float v = 0.0f;
        bool seen = false;
        if (p >= 0) {
            const V e = __ldg(vox + (size_t)p * kBlockVoxels + ((z & 7) << 6) + ((y & 7) << 3) + (x & 7));
            v = IO::sdf(e);
            seen = IO::wt(e) != 0 && !isnan(v);
            if (s) s[z * 81 + y * 9 + x] = v;
        }
        const unsigned observed = __ballot_sync(0xffffffffu, seen) >> (lane & 24);
        const unsigned inside = __ballot_sync(0xffffffffu, seen && v < 0.0f) >> (lane & 24);
        if (in_row && x == 0) rows.inner[z * kN + y] = (observed & 255u) | ((inside & 255u) << 16);
        if (!in_row && h < 217) rows.last[z * kN + y] = (seen ? 0x100u : 0u) | (seen && v < 0.0f ? 0x1000000u : 0u);
    }
    __syncthreads();
}

// The 8 cubes of row (y, z): those with all corners observed and a crossing.
struct CubeRow {
    unsigned s00, s10, s01, s11;  // inside bits of the four voxel rows (y, z), (y+1, z), (y, z+1), (y+1, z+1)
    unsigned cubes;
    __device__ __forceinline__ CubeRow(const BlockRows &b, int y, int z) {
        const unsigned a = b.row(y, z), c = b.row(y + 1, z), d = b.row(y, z + 1), e = b.row(y + 1, z + 1);
        const unsigned seen = a & c & d & e;
        s00 = a >> 16;
        s10 = c >> 16;
        s01 = d >> 16;
        s11 = e >> 16;
        const unsigned any = s00 | s10 | s01 | s11, all = s00 & s10 & s01 & s11;
        cubes = seen & (seen >> 1) & (any | (any >> 1)) & ~(all & (all >> 1)) & 255u;
    }
    // Case index: bit c for corner c (kCorner).
    __device__ __forceinline__ unsigned case_of(int x) const {
        const unsigned p = s00 >> x, q = s10 >> x, u = s01 >> x, v = s11 >> x;
        return (p & 3u) | ((q & 2u) << 1) | ((q & 1u) << 3) | ((u & 3u) << 4) | ((v & 2u) << 5) | ((v & 1u) << 7);
    }
};

__device__ __forceinline__ void load_table(unsigned long long *table) {
    for (int i = threadIdx.x; i < 128; i += blockDim.x)
        reinterpret_cast<int4 *>(table)[i] = reinterpret_cast<const int4 *>(g_mc_table)[i];
}

// Small CTAs: a block is a chain of dependent reads (key, neighbours, their
// voxels), so what counts is how many blocks are in flight.  A scene of 1.03 M
// triangles (640x480 frames, 6 mm): 25.4 us with a read per cube corner and 128
// threads, 21.9 here.
constexpr int kCountThreads = 64;

template <int FMT>
__global__ void __launch_bounds__(kCountThreads, 24) mc_count_kernel(MapDev m, unsigned nblocks, unsigned *block_tris) {
    __shared__ BlockRows rows;
    __shared__ unsigned red[kCountThreads / 32];
    __shared__ __align__(16) unsigned long long table[256];
    load_table(table);  // visible after stage_block's barriers
    for (unsigned b = blockIdx.x; b < nblocks; b += gridDim.x) {
        int bx, by, bz;
        unpack_key(m.block_keys[b], bx, by, bz);
        stage_block<FMT, kCountThreads>(m, (int)b, bx, by, bz, rows, nullptr);
        const CubeRow row(rows, threadIdx.x & 7, threadIdx.x >> 3);
        unsigned cnt = 0;
        for (unsigned c = row.cubes; c; c &= c - 1u) cnt += (unsigned)(table[row.case_of(__ffs(c) - 1)] >> 60);
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = cnt;
        __syncthreads();
        if (threadIdx.x == 0) block_tris[b] = red[0] + red[1];
    }
}

// Exclusive scan of per-block counts (single CTA; offsets[n] = total).  Thread
// t owns the contiguous run [t * per, (t + 1) * per), per a multiple of 4 (the
// arrays are 16-byte aligned): it sums its run, the CTA
// scans the 1024 run sums once, and the thread writes its run's prefixes, so
// the CTA synchronises a fixed number of times whatever n is.
__global__ void __launch_bounds__(1024) scan_kernel(const unsigned *in, unsigned *out, unsigned n,
                                                    unsigned *total) {
    __shared__ unsigned warp_sums[32];
    const unsigned per = (n + 4 * blockDim.x - 1) / (4 * blockDim.x) * 4;
    const unsigned lo = min(n, threadIdx.x * per), hi = min(n, lo + per), hi4 = lo + ((hi - lo) & ~3u);
    unsigned sum = 0;
#pragma unroll 4
    for (unsigned i = lo; i < hi4; i += 4) {
        const uint4 v = *reinterpret_cast<const uint4 *>(in + i);
        sum += v.x + v.y + v.z + v.w;
    }
    for (unsigned i = hi4; i < hi; ++i) sum += in[i];
    unsigned x = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) >= (unsigned)o) x += y;
    }
    if ((threadIdx.x & 31) == 31) warp_sums[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned w = warp_sums[threadIdx.x];
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
            if (threadIdx.x >= (unsigned)o) w += y;
        }
        warp_sums[threadIdx.x] = w;
    }
    __syncthreads();
    unsigned run = x - sum + ((threadIdx.x >= 32) ? warp_sums[(threadIdx.x >> 5) - 1] : 0u);
#pragma unroll 4
    for (unsigned i = lo; i < hi4; i += 4) {
        const uint4 v = *reinterpret_cast<const uint4 *>(in + i);
        *reinterpret_cast<uint4 *>(out + i) = make_uint4(run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z);
        run += v.x + v.y + v.z + v.w;
    }
    for (unsigned i = hi4; i < hi; ++i) {
        const unsigned v = in[i];
        out[i] = run;
        run += v;
    }
    if (threadIdx.x == blockDim.x - 1) {
        const unsigned t = warp_sums[31];
        out[n] = t;
        *total = t;
    }
}

__device__ __forceinline__ float mc_interp(float v1, float v2) {
    if (fabsf(0.0f - v1) < 1e-6f) return 0.0f;
    if (fabsf(0.0f - v2) < 1e-6f) return 1.0f;
    if (fabsf(v1 - v2) < 1e-6f) return 0.0f;
    return (0.0f - v1) / (v2 - v1);
}

// Emission: one CTA per block (grid-stride), one thread per triangle.  The
// CTA reads the block's neighbourhood, a thread per row of cubes counts its
// triangles, the rows are scanned in cube order and list (cube, triangle) per
// output slot; a warp then makes 32 consecutive triangles at a time and writes
// them through shared memory, since a triangle's 88 bytes written by its own
// thread touch a sector a word (36-byte stride).  The soup's order is cube
// order, then table order: a pure function of the map.  1.03 M triangles: 89.7
// us with the triangles' own writes, 61.1 with 128 threads, 53.3 here (a block's
// phases, read, list, write, leave the SM idle unless other blocks are in it).
constexpr int kEmitThreads = 64;  // one per row of cubes
constexpr int kMaxBlockTris = kBlockVoxels * kMcMaxCaseTris;  // 2560

// Vertex on edge e of the cube at local (lx,ly,lz), voxel position (px,py,pz),
// in voxel units: the reference's per-edge interpolation from the edge's first
// corner (MeshEngine.cu:151-225), driven by the edge and corner tables instead
// of a switch over the 12 edges, so the lanes of a warp on different edges do
// not diverge.  Along the
// edge's axis the coordinate is p + (a + t (b - a)) for corner coordinates a,
// b in {0, 1}, which is p + t or p + (1 - t) exactly as the per-edge forms.
__device__ __forceinline__ float3 edge_vertex_tab(int e, const float *s, int lx, int ly, int lz, float px, float py,
                                                  float pz) {
    // corners a, b of edge e (kEdge) as nibble e of two constants; corner c's
    // offset (kCorner): dx = bit c of 0x66, dy = bit c of 0xcc, dz = c >> 2
    const int a = (int)((0x321076543210ull >> (4 * e)) & 15ull);
    const int b = (int)((0x765447650321ull >> (4 * e)) & 15ull);
    const int ax = (0x66 >> a) & 1, ay = (0xcc >> a) & 1, az = a >> 2;
    const int bx = (0x66 >> b) & 1, by = (0xcc >> b) & 1, bz = b >> 2;
    const float va = s[(lz + az) * 81 + (ly + ay) * 9 + (lx + ax)];
    const float vb = s[(lz + bz) * 81 + (ly + by) * 9 + (lx + bx)];
    const float t = mc_interp(va, vb);
    const float ox = ax == bx ? (float)ax : (float)ax + t * (float)(bx - ax);
    const float oy = ay == by ? (float)ay : (float)ay + t * (float)(by - ay);
    const float oz = az == bz ? (float)az : (float)az + t * (float)(bz - az);
    return make_float3(px + ox, py + oy, pz + oz);
}

template <int FMT>
__global__ void __launch_bounds__(kEmitThreads) mc_emit_kernel(MapDev m, unsigned nblocks,
                                                               const unsigned *block_offset, int max_tris,
                                                               float *points, float *normals, int *cases,
                                                               int *cube_xyz) {
    __shared__ float s[kN3];
    __shared__ BlockRows rows;
    __shared__ __align__(16) unsigned long long table[256];
    __shared__ unsigned short slot[kMaxBlockTris];  // output slot -> cube << 3 | triangle of the cube
    __shared__ unsigned char ucase[kBlockVoxels];  // case index of each cube with triangles
    __shared__ float out_p[kEmitThreads / 32][32 * 9], out_n[kEmitThreads / 32][32 * 9];
    __shared__ int out_c[kEmitThreads / 32][32 * 3];
    __shared__ unsigned first_half;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    load_table(table);
    const float vs = m.voxel_size;
    for (unsigned b = blockIdx.x; b < nblocks; b += gridDim.x) {
        const unsigned base = block_offset[b];
        const unsigned ntri = block_offset[b + 1] - base;
        if (ntri == 0 || base >= (unsigned)max_tris) continue;  // uniform across the CTA
        int bx, by, bz;
        unpack_key(m.block_keys[b], bx, by, bz);
        stage_block<FMT, kEmitThreads>(m, (int)b, bx, by, bz, rows, s);  // ends with a barrier (also for the table)
        const CubeRow row(rows, threadIdx.x & 7, threadIdx.x >> 3);
        unsigned mine = 0;
        for (unsigned c = row.cubes; c; c &= c - 1u) mine += (unsigned)(table[row.case_of(__ffs(c) - 1)] >> 60);
        unsigned run = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += y;
        }
        if (threadIdx.x == 31) first_half = run;
        __syncthreads();
        run += (warp == 1 ? first_half : 0u) - mine;
        for (unsigned c = row.cubes; c; c &= c - 1u) {
            const int x = __ffs(c) - 1;
            const unsigned k = row.case_of(x), n = (unsigned)(table[k] >> 60), i = threadIdx.x * 8u + (unsigned)x;
            ucase[i] = (unsigned char)k;
            for (unsigned t = 0; t < n; ++t) slot[run + t] = (unsigned short)(i << 3 | t);
            run += n;
        }
        __syncthreads();
        const unsigned nout = min(ntri, (unsigned)max_tris - base);
        for (unsigned j0 = warp * 32; j0 < nout; j0 += kEmitThreads) {
            const int n = (int)min(32u, nout - j0);
            const size_t off = (size_t)base + j0;
            if (lane < n) {
                const unsigned e = slot[j0 + lane];
                const int i = (int)(e >> 3), t = (int)(e & 7u);
                const int lx = i & 7, ly = (i >> 3) & 7, lz = i >> 6;
                const int c = ucase[i];
                const unsigned edges = (unsigned)(table[c] >> (12 * t));
                const int gx = bx * 8 + lx, gy = by * 8 + ly, gz = bz * 8 + lz;
                const float px = (float)gx, py = (float)gy, pz = (float)gz;
                float3 v[3];
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const float3 ev = edge_vertex_tab((int)((edges >> (4 * q)) & 15u), s, lx, ly, lz, px, py, pz);
                    v[q] = make_float3(ev.x * vs, ev.y * vs, ev.z * vs);
                }
                const float ax = v[1].x - v[0].x, ay = v[1].y - v[0].y, az = v[1].z - v[0].z;
                const float cx = v[2].x - v[0].x, cy = v[2].y - v[0].y, cz = v[2].z - v[0].z;
                float nx = ay * cz - az * cy, ny = az * cx - ax * cz, nz = ax * cy - ay * cx;
                const float nn = nx * nx + ny * ny + nz * nz;
                if (nn > 0.0f) {
                    const float inv = 1.0f / sqrtf(nn);
                    nx *= inv;
                    ny *= inv;
                    nz *= inv;
                }
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    out_p[warp][9 * lane + 3 * q] = v[q].x;
                    out_p[warp][9 * lane + 3 * q + 1] = v[q].y;
                    out_p[warp][9 * lane + 3 * q + 2] = v[q].z;
                    out_n[warp][9 * lane + 3 * q] = nx;
                    out_n[warp][9 * lane + 3 * q + 1] = ny;
                    out_n[warp][9 * lane + 3 * q + 2] = nz;
                }
                out_c[warp][3 * lane] = gx;
                out_c[warp][3 * lane + 1] = gy;
                out_c[warp][3 * lane + 2] = gz;
                cases[off + lane] = c;
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const int i = lane + 32 * k;
                if (i < 9 * n) {
                    points[off * 9 + i] = out_p[warp][i];
                    normals[off * 9 + i] = out_n[warp][i];
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int i = lane + 32 * k;
                if (i < 3 * n) cube_xyz[off * 3 + i] = out_c[warp][i];
            }
            __syncwarp();
        }
        __syncthreads();
    }
}

int mesher_ensure_blocks(MeshBuffers &mb, size_t n_blocks) {
    if (mb.cap_blocks >= n_blocks) return YAS_OK;
    cudaFree(mb.block_tris);
    cudaFree(mb.block_offset);
    mb.block_tris = nullptr;
    mb.block_offset = nullptr;
    size_t cap = n_blocks < 1024 ? 1024 : n_blocks;
    if (cudaMalloc(&mb.block_tris, cap * sizeof(unsigned)) != cudaSuccess ||
        cudaMalloc(&mb.block_offset, (cap + 1) * sizeof(unsigned)) != cudaSuccess) {
        cudaGetLastError();
        mb.cap_blocks = 0;
        return YAS_ERR_OOM;
    }
    mb.cap_blocks = cap;
    return YAS_OK;
}

int launch_meshify(const MapDev &m, int fmt, MeshBuffers &mb, unsigned n_blocks, cudaStream_t s) {
    YAS_TRY(mesher_ensure_blocks(mb, n_blocks));
    cudaMemsetAsync(mb.counters, 0, sizeof(unsigned), s);
    if (n_blocks == 0) return YAS_OK;
    const unsigned grid = std::min(n_blocks, (unsigned)kSMs * 32u);
    switch (fmt) {
        case YAS_VOXEL_F32:
            mc_count_kernel<YAS_VOXEL_F32><<<grid, kCountThreads, 0, s>>>(m, n_blocks, mb.block_tris);
            break;
        case YAS_VOXEL_F16:
            mc_count_kernel<YAS_VOXEL_F16><<<grid, kCountThreads, 0, s>>>(m, n_blocks, mb.block_tris);
            break;
        case YAS_VOXEL_S16:
            mc_count_kernel<YAS_VOXEL_S16><<<grid, kCountThreads, 0, s>>>(m, n_blocks, mb.block_tris);
            break;
        default:
            mc_count_kernel<YAS_VOXEL_S24><<<grid, kCountThreads, 0, s>>>(m, n_blocks, mb.block_tris);
            break;
    }
    scan_kernel<<<1, 1024, 0, s>>>(mb.block_tris, mb.block_offset, n_blocks, mb.counters);
    switch (fmt) {
        case YAS_VOXEL_F32:
            mc_emit_kernel<YAS_VOXEL_F32><<<grid, kEmitThreads, 0, s>>>(m, n_blocks, mb.block_offset, mb.max_tris,
                                                               mb.points, mb.normals, mb.cases, mb.cube_xyz);
            break;
        case YAS_VOXEL_F16:
            mc_emit_kernel<YAS_VOXEL_F16><<<grid, kEmitThreads, 0, s>>>(m, n_blocks, mb.block_offset, mb.max_tris,
                                                               mb.points, mb.normals, mb.cases, mb.cube_xyz);
            break;
        case YAS_VOXEL_S16:
            mc_emit_kernel<YAS_VOXEL_S16><<<grid, kEmitThreads, 0, s>>>(m, n_blocks, mb.block_offset, mb.max_tris,
                                                               mb.points, mb.normals, mb.cases, mb.cube_xyz);
            break;
        default:
            mc_emit_kernel<YAS_VOXEL_S24><<<grid, kEmitThreads, 0, s>>>(m, n_blocks, mb.block_offset, mb.max_tris,
                                                               mb.points, mb.normals, mb.cases, mb.cube_xyz);
            break;
    }
    return YAS_OK;
}

}  // namespace yas

// Host-visible table access for tests (same generator as the device tables).
extern "C" YAS_API int yas_mc_tables(unsigned short *edge, signed char *tri, unsigned char *count) {
    yas::McTables t;
    yas::build_mc_tables(t);
    if (edge) memcpy(edge, t.edge, sizeof(t.edge));
    if (tri) memcpy(tri, t.tri, sizeof(t.tri));
    if (count) memcpy(count, t.count, sizeof(t.count));
    return YAS_OK;
}
