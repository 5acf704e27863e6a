// afx_mc.cu -- marching cubes (point-cloud and triangle variants, fused into one pass over
// the volume) with warp-aggregated stream compaction, and the lexicographic sort +
// unique of the canonical point cloud (a merge sort: 2048-element tiles in shared memory,
// then merge-path passes).
//
// Case index, edge interpolation and triangulation follow src/MarchingCubes.cu:294-420
// (corner bit c set when tsdf > iso, cubes skipped when any corner weight is 0, cubes
// x,y,z < dim-2).  The triangulation table is the reference's (packed re-encoding).
#include <cuda.h>

#include <cstring>

#include "afx_host.h"
#include "afx_internal.h"
#include "afx_store.cuh"
#include "afx_tma.h"

namespace afx {

__constant__ uint64_t c_tri_table[256];

static const uint64_t kTriTableHost[256] = {
#include "mc_tables.inc"
};

// The triangle table is constant: uploaded once per device context (before the first marching-cubes launch,
// which is never inside a stream capture: a session's first frame runs eagerly).
static int upload_tables() {
    static ContextOnce once;
    return once_per_context(once, [](int) {
        AFX_CUDA(cudaMemcpyToSymbol(c_tri_table, kTriTableHost, sizeof(kTriTableHost)));
        return (int)AFX_OK;
    });
}

struct McArgs {
    Volume vol;
    float iso;
    float* points;
    unsigned* point_count;
    long point_cap;
    float* verts;
    unsigned* face_count;  // triangles; vertex count = 3 * faces
    unsigned* vert_count;
    long face_cap;
    int* faces;
    int* error;  // TMA path: set on a tile-load timeout
    const unsigned char* occ;  // brick occupancy (8^3 voxels), or null: process every tile
    bool occ_positive;         // it marks values above iso, not weights
    int nbx, nby, nbz;
    unsigned* tile_count;      // persistent grid: occupied tiles listed here (with occ), or null
    unsigned* tile_list;
};


// Corners of edge e: corner offsets (x, y, z) of its two ends, one bit each, 6 bits per edge
// (src/MarchingCubes.cu:338-379; the corner and edge numbers of the tables below), in two registers:
// lanes look up different edges, which constant memory would serve one after the other.
constexpr unsigned corner_bits(int c) {  // c0 (1,1,0) c1 (1,0,0) c2 (0,0,0) c3 (0,1,0), c4..c7 one slice up
    return (unsigned)((c & 3) == 0 || (c & 3) == 1) | (unsigned)((c & 3) == 0 || (c & 3) == 3) << 1 | (unsigned)(c >= 4) << 2;
}
constexpr int kEdge[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6}, {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
constexpr uint64_t edge_ends(int from) {  // of edges from .. from + 5
    uint64_t v = 0;
    for (int e = 0; e < 6; ++e)
        v |= (uint64_t)(corner_bits(kEdge[from + e][0]) | corner_bits(kEdge[from + e][1]) << 3) << (6 * e);
    return v;
}

// Edges that a cube of case ci crosses: those whose ends lie on different sides.
AFX_D unsigned crossed_edges(unsigned ci) {
    const unsigned lo = ci & 15u, hi = ci >> 4;
    const unsigned a = lo ^ (((lo >> 1) | (lo << 3)) & 15u), b = hi ^ (((hi >> 1) | (hi << 3)) & 15u);
    return a | (b << 4) | ((lo ^ hi) << 8);
}

// (float)((double)a + (double)m * (double)d) for 0 <= m <= 1, from binary32 operations: binary64 issues at
// about 1/80 of their rate here.  m d is p + e exactly, a + p is s + f exactly (Knuth's TwoSum), and
// t = f + e has a relative error of at most 2^-24.  So the exact value, and its rounding to binary64,
// lie between s + t (1 - 2^-20) and s + t (1 + 2^-20); where both round to the same binary32 number,
// which is all but about one in 2^18 times, that is the result.  Otherwise, and where e could
// underflow, the binary64 sum is taken.
AFX_D float blend64(float a, float m, float d) {
    const float p = m * d, e = fmaf(m, d, -p);
    const float s = a + p, v = s - a, f = (a - (s - v)) + (p - v);
    const float t = f + e;
    const float lo = s + t * (1.0f - 9.5367431640625e-7f), hi = s + t * (1.0f + 9.5367431640625e-7f);
    if (lo == hi && (fabsf(p) > 1e-25f || p == 0.0f)) return lo;
    return (float)__dadd_rn((double)a, __dmul_rn((double)m, (double)d));
}

// getVertex + interpolate (src/MarchingCubes.cu:294-336) of edge e of cube (x, y, z).  The ends differ in one
// coordinate only; in the others p0 + mu (p1 - p0) is p0 + mu 0 = p0 + 0 for a finite mu.
template <class TT>
AFX_D void edge_vertex(const TT* __restrict__ tsdf, const Volume& vol, int x, int y, int z, int e, float iso,
                       float* o) {
    constexpr uint64_t kLow = edge_ends(0), kHigh = edge_ends(6);
    const unsigned ends = (unsigned)((e < 6 ? kLow >> (6 * e) : kHigh >> (6 * (e - 6))) & 63u);
    const int X = vol.dims[0], Y = vol.dims[1];
    const int x1 = x + (ends & 1), y1 = y + ((ends >> 1) & 1), z1 = z + ((ends >> 2) & 1);
    const int x2 = x + ((ends >> 3) & 1), y2 = y + ((ends >> 4) & 1), z2 = z + (ends >> 5);
    const float t0 = vox_ld_t(tsdf, ((long)z1 * Y + y1) * X + x1);
    const float t1 = vox_ld_t(tsdf, ((long)z2 * Y + y2) * X + x2);
    float p0[3], p1[3];
    voxel_to_world(x1, y1, z1, vol.vs, vol.half, p0);
    voxel_to_world(x2, y2, z2, vol.vs, vol.half, p1);
    o[0] = p0[0];
    o[1] = p0[1];
    o[2] = p0[2];
    // (double)v < 1e-7 is v < 1e-7f for every float v: 1e-7f is the smallest float >= 1e-7
    if (fabsf(iso - t0) < 1e-7f) return;
    if (fabsf(iso - t1) < 1e-7f) {
        o[0] = p1[0];
        o[1] = p1[1];
        o[2] = p1[2];
        return;
    }
    if (fabsf(t0 - t1) < 1e-7f) return;
    float mu = (iso - t0) / (t1 - t0);
    if (mu > 1.0f) mu = 1.0f;
    else if (mu < 0.0f) mu = 0.0f;
    const int axis = (ends ^ (ends >> 3)) & 1 ? 0 : ((ends ^ (ends >> 3)) & 2 ? 1 : 2);
    const float a = axis == 0 ? p0[0] : axis == 1 ? p0[1] : p0[2], b = axis == 0 ? p1[0] : axis == 1 ? p1[1] : p1[2];
    const float v = blend64(a, mu, b - a);
#pragma unroll
    for (int c = 0; c < 3; ++c) o[c] = c == axis ? v : (mu == mu ? p0[c] + 0.0f : v);  // not a number: in all three
}

AFX_D bool vne(const float* a, const float* b) { return a[0] != b[0] || a[1] != b[1] || a[2] != b[2]; }

// Vertices and triangles of up to 32 cubes, one per lane, by the whole warp: the point-cloud vertices
// (marchingCubesMeshKernel) and/or the triangles (marchingCubesFullKernel).  The crossed edges of all
// the cubes are laid out one after the other and interpolated one per lane, so lanes have the same work
// whatever their cubes' cases are, and points and triangles are written in consecutive words.
struct McEdges {                    // of one warp
    int cube[32][3];
    unsigned short edge[32 * 12];   // cube << 4 | edge
};
template <bool kMesh>
struct McScratch : McEdges {
    float vert[32 * 12][3];         // vertices in edge order
    unsigned tri[32 * 5];           // triangles: three indices into vert, 9 bits each
};
template <>
struct McScratch<false> : McEdges {};

template <bool kPoints, bool kMesh, class TT>
AFX_D void mc_emit(const TT* __restrict__ tsdf, const McArgs& a, int x, int y, int z, int ci, bool active,
                   McScratch<kMesh>& S) {
    const int lane = threadIdx.x & 31;
    const unsigned et = active ? crossed_edges((unsigned)ci) : 0u;
    const unsigned ne = __popc(et);
    unsigned incl = ne;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const unsigned total = __shfl_sync(0xffffffffu, incl, 31), first = incl - ne;
    unsigned base = 0;
    if (kPoints && lane == 0 && total) base = atomicAdd(a.point_count, total);
    S.cube[lane][0] = x;
    S.cube[lane][1] = y;
    S.cube[lane][2] = z;
    {
        unsigned k = first;
        for (unsigned rest = et; rest; rest &= rest - 1) S.edge[k++] = (unsigned short)(lane << 4 | (__ffs(rest) - 1));
    }
    if (kPoints) base = __shfl_sync(0xffffffffu, base, 0);
    __syncwarp();
    for (unsigned i = lane; i < total; i += 32) {
        const unsigned item = S.edge[i];
        const int* c = S.cube[item >> 4];
        float v[3];
        edge_vertex(tsdf, a.vol, c[0], c[1], c[2], (int)(item & 15u), a.iso, v);
        if (kPoints && (long)base + i < a.point_cap) {
            float* o = a.points + 3 * ((long)base + i);
            o[0] = v[0];
            o[1] = v[1];
            o[2] = v[2];
        }
        if constexpr (kMesh) {
            S.vert[i][0] = v[0];
            S.vert[i][1] = v[1];
            S.vert[i][2] = v[2];
        }
    }
    __syncwarp();
    if constexpr (kMesh) {
        const uint64_t table = active ? c_tri_table[ci] : 0xFull;
        unsigned tri[5], nt = 0;  // the cube's triangles without two equal corners
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const unsigned e = (unsigned)(table >> (12 * k)) & 0xFFFu;  // three edges
            tri[k] = 0xffffffffu;
            // the table ends a case's list with 0xF; everything after it is not read
            bool on = true;
#pragma unroll
            for (int q = 0; q <= k; ++q) on = on && ((unsigned)(table >> (12 * q)) & 0xFu) != 0xFu;
            if (!on) continue;
            unsigned v[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) v[q] = first + __popc(et & ((1u << ((e >> (4 * q)) & 0xFu)) - 1u));
            if (vne(S.vert[v[0]], S.vert[v[1]]) && vne(S.vert[v[0]], S.vert[v[2]]) && vne(S.vert[v[1]], S.vert[v[2]])) {
                tri[k] = v[0] | v[1] << 9 | v[2] << 18;
                ++nt;
            }
        }
        incl = nt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const unsigned tris = __shfl_sync(0xffffffffu, incl, 31);
        unsigned f = 0;
        if (lane == 0 && tris) f = atomicAdd(a.face_count, tris);
        {
            unsigned k = incl - nt;
#pragma unroll
            for (int q = 0; q < 5; ++q)
                if (tri[q] != 0xffffffffu) S.tri[k++] = tri[q];
        }
        f = __shfl_sync(0xffffffffu, f, 0);
        __syncwarp();
        const long room = max(0L, min((long)tris, a.face_cap - (long)f));
        for (unsigned j = lane; j < 9 * (unsigned)room; j += 32) {
            const unsigned t = j / 9, c = j - 9 * t, q = c / 3;
            a.verts[9 * (long)f + j] = S.vert[(S.tri[t] >> (9 * q)) & 511u][c - 3 * q];
        }
        for (unsigned j = lane; j < 3 * (unsigned)room; j += 32) a.faces[3 * (long)f + j] = (int)(3 * f + j);
        __syncwarp();
    }
}

constexpr int kMcX = 32, kMcY = 8;  // cube columns of a TMA tile

// False when no marked 8^3 brick holds a corner of the cubes [x0, x0+xr) x [y0, y0+yr) x [z0, z0+zr) that
// an active cube has to have: bricks with a weight hold the origin corners (a cube is active only if
// all eight corners have a weight), bricks with a value above iso any corner.  Every thread evaluates
// it (same answer).
AFX_D bool box_occupied(const McArgs& a, int x0, int xr, int y0, int yr, int z0, int zr) {
    if (!a.occ) return true;
    const int last = a.occ_positive ? 0 : 1;
    const int bx1 = min((x0 + xr - last) >> 3, a.nbx - 1), by1 = min((y0 + yr - last) >> 3, a.nby - 1);
    const int bz1 = min((z0 + zr - last) >> 3, a.nbz - 1);
    for (int bz = z0 >> 3; bz <= bz1; ++bz)
        for (int by = y0 >> 3; by <= by1; ++by)
            for (int bx = x0 >> 3; bx <= bx1; ++bx)
                if (__ldg(a.occ + ((long)bz * a.nby + by) * a.nbx + bx)) return true;
    return false;
}

// A TMA tile's box: 32 x 8 cube columns, zr cubes deep.
AFX_D bool tile_occupied(const McArgs& a, int x0, int y0, int z0, int zr) {
    return box_occupied(a, x0, kMcX, y0, kMcY, z0, zr);
}

// Sweep from global memory, for any row length and alignment: a warp marches kSweepZ slices over 32
// columns and kSweepY + 1 rows of voxels (31 x kSweepY cubes a slice), with no barrier anywhere.  A
// lane reads one voxel of each row, coalesced, and keeps two bits of it -- weight not zero, value
// above iso -- so a cube's case comes from its own bits, its right neighbour's by one shuffle and
// those of the slice before; the weights of the next slice are on their way meanwhile, and values
// are read only where the warp's rows hold a weight.  Surface cubes wait in a queue of the warp's own
// until 32 of them are interpolated together.
// Bound: the latency of a slice and, where there is surface, the shared-memory traffic of the emission.
// 257 x 230 x 301 voxels (142 MB) with 0.22 m^2 of surface at 2.5 mm: 60 us, 2.4 TB/s of the volume's bytes (a
// thread per column reading eight corners a cube, and interpolating where it stood, took 400 us; runs of
// 16 slices 111 us, a warp with much surface holding up the rest).
constexpr int kSweepY = 4, kSweepZ = 8, kSweepWarps = 8;

template <class TT, class WT, bool kPoints, bool kMesh>
__global__ void __launch_bounds__(32 * kSweepWarps) mc_sweep_kernel(const TT* __restrict__ tsdf,
                                                                    const WT* __restrict__ weights, McArgs a) {
    __shared__ unsigned queue[kSweepWarps][64];
    extern __shared__ __align__(16) unsigned char sweep_raw[];
    McScratch<kMesh>* scratch = reinterpret_cast<McScratch<kMesh>*>(sweep_raw);  // one per warp
    constexpr int R = kSweepY + 1;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int X = a.vol.dims[0], Y = a.vol.dims[1];
    const int nx = X - 2, ny = Y - 2, nz = a.vol.dims[2] - 2;
    const int x0 = blockIdx.x * 31, y0 = (blockIdx.y * kSweepWarps + w) * kSweepY, z0 = blockIdx.z * kSweepZ;
    const int z1 = min(z0 + kSweepZ, nz);  // the last slice of voxels
    if (y0 >= ny || !box_occupied(a, x0, 31, y0, kSweepY, z0, kSweepZ)) return;  // uniform over the warp
    unsigned* q = queue[w];
    unsigned nq = 0;  // queued cubes (uniform)
    const int x = x0 + lane;
    const long XY = (long)X * Y, base = (long)y0 * X + x;
    const int rows = x < X ? min(R, Y - y0) : 0;
    const unsigned cubes = (lane < 31 && x < nx) ? (1u << min(kSweepY, ny - y0)) - 1u : 0u;  // rows with a cube here
    auto emit = [&](unsigned from, unsigned n) {  // n <= 32 cubes of the queue
        const bool act = (unsigned)lane < n;
        const unsigned e = act ? q[from + lane] : 0u;
        mc_emit<kPoints, kMesh>(tsdf, a, x0 + (int)((e >> 8) & 31u), y0 + (int)((e >> 13) & 7u), z0 + (int)(e >> 16),
                                (int)(e & 255u), act, scratch[w]);
    };
    float wn[R];
    auto load_weights = [&](int z) {
        const WT* p = weights + z * XY + base;
#pragma unroll
        for (int r = 0; r < R; ++r) wn[r] = (r < rows && z <= z1) ? vox_ld_w(p, (long)r * X) : 0.f;
    };
    load_weights(z0);
    // of the slice before, per row of cubes: all four corners weighted, any / every one above iso, and
    // the bits themselves (own column, next column)
    unsigned full0 = 0, any0 = 0, all0 = 0, f0 = 0, g0 = 0;
    for (int z = z0; z <= z1; ++z) {
        unsigned f = 0;  // bit r: weight of row r; bit 8 + r: value above iso
#pragma unroll
        for (int r = 0; r < R; ++r) f |= (wn[r] == 0.0f ? 0u : 1u) << r;
        load_weights(z + 1);
        if (__any_sync(0xffffffffu, f != 0u)) {
            const TT* p = tsdf + z * XY + base;
            float t[R];
#pragma unroll
            for (int r = 0; r < R; ++r) t[r] = (f >> r) & 1u ? vox_ld_t(p, (long)r * X) : 0.f;
#pragma unroll
            for (int r = 0; r < R; ++r) f |= ((f >> r) & 1u && t[r] > a.iso ? 1u : 0u) << (8 + r);
        }
        const unsigned g = __shfl_down_sync(0xffffffffu, f, 1);
        const unsigned both = f & g, either = f | g;
        const unsigned full = both & (both >> 1);                                  // low bits: weights
        const unsigned all = (both & (both >> 1)) >> 8, any = (either | (either >> 1)) >> 8;
        const unsigned act = full & full0 & (any | any0) & ~(all & all0) & cubes;
        if (__any_sync(0xffffffffu, act != 0u)) {
#pragma unroll
            for (int r = 0; r < kSweepY; ++r) {
                const bool on = (act >> r) & 1u;
                const unsigned bal = __ballot_sync(0xffffffffu, on);
                if (bal == 0u) continue;
                if (on) {
                    // corners (src/MarchingCubes.cu:338-379): c0 (1,1,0) c1 (1,0,0) c2 (0,0,0) c3 (0,1,0),
                    // c4..c7 the same one slice up
                    auto bits = [&](unsigned own, unsigned next) {
                        const unsigned o = own >> (8 + r), n = next >> (8 + r);
                        return ((n >> 1) & 1u) | ((n & 1u) << 1) | ((o & 1u) << 2) | (((o >> 1) & 1u) << 3);
                    };
                    const unsigned ci = bits(f0, g0) | (bits(f, g) << 4);
                    q[nq + __popc(bal & ((1u << lane) - 1u))] =
                        ci | ((unsigned)lane << 8) | ((unsigned)r << 13) | ((unsigned)(z - 1 - z0) << 16);
                }
                nq += __popc(bal);
                __syncwarp();
                if (nq >= 32) {
                    emit(nq - 32, 32);
                    nq -= 32;
                    __syncwarp();
                }
            }
        }
        full0 = full;
        any0 = any;
        all0 = all;
        f0 = f;
        g0 = g;
    }
    if (nq) emit(0, nq);
}

// Same cubes again, with the CTA's whole brick of corner values -- 40 x 9 x (ZR + 1)
// elements of TSDF and of weights, x padded to a 16-byte multiple -- brought into shared memory by
// two TMA tile loads on one mbarrier, so the march reads no global memory for inactive cubes.
constexpr int kMcTX = 40;  // box width in elements (>= kMcX + 1; 160 B in FP32, 80 B in FP16)
// each brick starts on a 128-byte boundary (TMA destination alignment), plus slack to align the base
__host__ __device__ constexpr size_t mc_brick_bytes(size_t elem, int zr) {
    return ((size_t)kMcTX * (kMcY + 1) * (zr + 1) * elem + 127) / 128 * 128;
}
__host__ __device__ constexpr size_t mc_tma_smem(size_t elem, int zr) {  // the bricks, or the warps' scratch after them
    const size_t bricks = 2 * mc_brick_bytes(elem, zr), scratch = kMcX * kMcY / 32 * sizeof(McScratch<true>);
    return (bricks > scratch ? bricks : scratch) + 128;
}

AFX_D uint32_t mc_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

AFX_D float smem_t(const float* p, int i) { return p[i]; }
AFX_D float smem_t(const __half* p, int i) { return __half2float(p[i]); }
AFX_D bool smem_w_zero(const float* p, int i) { return p[i] == 0.0f; }
AFX_D bool smem_w_zero(const unsigned short* p, int i) { return p[i] == 0; }

// ZR: cubes per CTA along z (the tile depth the autotuner chooses: 8, 16 or 32)
template <class TT, class WT, bool kPoints, bool kMesh, int ZR>
__global__ void __launch_bounds__(kMcX * kMcY) mc_tma_kernel(const __grid_constant__ CUtensorMap map_t,
                                                            const __grid_constant__ CUtensorMap map_w,
                                                            const TT* __restrict__ tsdf, McArgs a) {
    static_assert(sizeof(TT) == sizeof(WT), "value and weight bricks share one layout");
    static_assert(ZR <= 64, "the queue entry keeps z in 6 bits");
    constexpr size_t kMcBrickBytes = mc_brick_bytes(sizeof(TT), ZR);
    extern __shared__ __align__(128) unsigned char mc_raw[];
    __shared__ alignas(8) unsigned long long mbar;
    __shared__ unsigned q[kMcX * kMcY * ZR];  // surface cubes of this CTA: ci | x << 8 | y << 13 | z << 16
    __shared__ unsigned q_n;
    constexpr int kSlice = kMcTX * (kMcY + 1);
    const uint32_t pad = (128u - (mc_smem_u32(mc_raw) & 127u)) & 127u;
    TT* st = reinterpret_cast<TT*>(mc_raw + pad);
    WT* sw = reinterpret_cast<WT*>(mc_raw + pad + kMcBrickBytes);
    const int tid = threadIdx.y * kMcX + threadIdx.x;
    const int x0 = blockIdx.x * kMcX, y0 = blockIdx.y * kMcY, z0 = blockIdx.z * ZR;
    if (!tile_occupied(a, x0, y0, z0, ZR)) return;  // uniform over the CTA, before any barrier or copy
    if (((mc_smem_u32(st) | mc_smem_u32(sw)) & 127u) != 0u) {  // never expected: refuse rather than fault
        if (tid == 0 && a.error) atomicOr(a.error, ERRF_TMA);
        return;
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mc_smem_u32(&mbar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        q_n = 0;
    }
    __syncthreads();
    if (tid == 0) {
        const unsigned bytes = (unsigned)(kSlice * (ZR + 1) * (sizeof(TT) + sizeof(WT)));
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mc_smem_u32(&mbar)), "r"(bytes)
                     : "memory");
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
            "[%5];" ::"r"(mc_smem_u32(st)),
            "l"(&map_t), "r"(x0), "r"(y0), "r"(z0), "r"(mc_smem_u32(&mbar))
            : "memory");
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
            "[%5];" ::"r"(mc_smem_u32(sw)),
            "l"(&map_w), "r"(x0), "r"(y0), "r"(z0), "r"(mc_smem_u32(&mbar))
            : "memory");
    }
    // bounded wait for the brick (phase 0); the give-up decision is uniform across the CTA
    bool done = false;
    for (int it = 0; it < (1 << 22) && !done; ++it) {
        uint32_t ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(mc_smem_u32(&mbar))
            : "memory");
        done = ok != 0;
    }
    if (__syncthreads_or(!done)) {
        if (tid == 0 && a.error) atomicOr(a.error, ERRF_TMA | ERRF_TIMEOUT);
        // the copies may still land: wait for them (bounded) before the CTA's shared memory goes
        for (int it = 0; it < (1 << 22); ++it) {
            uint32_t ok;
            asm volatile(
                "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
                : "=r"(ok)
                : "r"(mc_smem_u32(&mbar))
                : "memory");
            if (ok) break;
        }
        return;
    }
    const int nx = a.vol.dims[0] - 2, ny = a.vol.dims[1] - 2, nz = a.vol.dims[2] - 2;
    const int x = x0 + threadIdx.x, y = y0 + threadIdx.y;
    const int z1 = min(z0 + ZR, nz);
    const bool col = x < nx && y < ny;
    const int o00 = threadIdx.y * kMcTX + threadIdx.x;  // (x, y) within a slice
    for (int z = z0; z < z1; ++z) {
        const int s0 = (z - z0) * kSlice + o00, s1 = s0 + kSlice;
        int ci = 0;
        if (col) {
            // corners (src/MarchingCubes.cu:338-379): c0 (1,1,0) c1 (1,0,0) c2 (0,0,0) c3 (0,1,0), c4..c7 one slice up
            const int off[8] = {s0 + kMcTX + 1, s0 + 1, s0, s0 + kMcTX, s1 + kMcTX + 1, s1 + 1, s1, s1 + kMcTX};
            bool any_zero = false;
#pragma unroll
            for (int c = 0; c < 8; ++c) any_zero |= smem_w_zero(sw, off[c]);
            if (!any_zero)
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if (smem_t(st, off[c]) > a.iso) ci |= 1 << c;
        }
        const bool active = ci != 0 && ci != 255;
        // queue the surface cubes (warp-aggregated), processed densely below
        const unsigned bal = __ballot_sync(0xffffffffu, active);
        if (bal) {
            const int lane = threadIdx.x & 31;  // blockDim.x == 32: a warp is one row of x
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(&q_n, (unsigned)__popc(bal));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (active)
                q[base + __popc(bal & ((1u << lane) - 1))] =
                    (unsigned)ci | ((unsigned)threadIdx.x << 8) | ((unsigned)threadIdx.y << 13) | ((unsigned)(z - z0) << 16);
        }
    }
    __syncthreads();
    // edge vertices and triangles of the queued cubes, 32 per warp; the warps' scratch takes the place of
    // the bricks, which have been read
    McScratch<kMesh>* scratch = reinterpret_cast<McScratch<kMesh>*>(mc_raw + pad);
    const unsigned nq = q_n;
    for (unsigned r0 = 0; r0 < nq; r0 += kMcX * kMcY) {
        const unsigned qi = r0 + tid;
        const bool act = qi < nq;
        const unsigned e = act ? q[qi] : 0u;
        mc_emit<kPoints, kMesh>(tsdf, a, x0 + (int)((e >> 8) & 31u), y0 + (int)((e >> 13) & 7u),
                                z0 + (int)((e >> 16) & 63u), (int)(e & 255u), act, scratch[tid >> 5]);
    }
}

// The same cubes again, by a persistent grid: a CTA walks the tiles blockIdx.x, + gridDim.x, ...
// with two stages of TMA-loaded bricks.  The load of tile k + 2 is issued as soon as tile k's
// classification has read its stage, so loads overlap the FP64 edge interpolation and the appends
// of the tiles before.  Every wait is bounded; on a timeout the CTA flags the error, waits (bounded)
// for the loads it issued and leaves.
AFX_D bool mc_wait(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < (1 << 22); ++it) {
        uint32_t ok;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return true;
    }
    return false;
}

// The occupied tiles of the volume (those tile_occupied accepts), in no particular order.
__global__ void mc_tile_list_kernel(McArgs a, int tx_n, int ty_n, int tz_n, int zr) {
    const long nt = (long)tx_n * ty_n * tz_n;
    AFX_GRID_STRIDE(t, nt) {
        const int tx = (int)(t % tx_n), ty = (int)((t / tx_n) % ty_n), tz = (int)(t / ((long)tx_n * ty_n));
        if (tile_occupied(a, tx * kMcX, ty * kMcY, tz * zr, zr)) a.tile_list[atomicAdd(a.tile_count, 1u)] = (unsigned)t;
    }
}

// Persistent grid over the tiles -- every tile, or with a.tile_list the listed ones -- with two
// stages of TMA bricks: the next tile's brick loads while this one is classified.
template <class TT, class WT, bool kPoints, bool kMesh, int ZR>
__global__ void __launch_bounds__(kMcX * kMcY) mc_pipe_kernel(const __grid_constant__ CUtensorMap map_t,
                                                             const __grid_constant__ CUtensorMap map_w,
                                                             const TT* __restrict__ tsdf, McArgs a, int tx_n, int ty_n,
                                                             int tz_n) {
    static_assert(sizeof(TT) == sizeof(WT), "value and weight bricks share one layout");
    static_assert(ZR <= 64, "the queue entry keeps z in 6 bits");
    constexpr size_t kBrick = mc_brick_bytes(sizeof(TT), ZR);
    constexpr int kSlice = kMcTX * (kMcY + 1);
    constexpr unsigned kBytes = (unsigned)(kSlice * (ZR + 1) * (sizeof(TT) + sizeof(WT)));
    extern __shared__ __align__(128) unsigned char mc_raw[];
    __shared__ alignas(8) unsigned long long mbar[2];
    __shared__ unsigned q[kMcX * kMcY * ZR];
    __shared__ unsigned q_n;
    McScratch<kMesh>* scratch = reinterpret_cast<McScratch<kMesh>*>(mc_raw);  // the bricks follow
    unsigned char* const mc_bricks = mc_raw + kMcX * kMcY / 32 * sizeof(McScratch<kMesh>);
    const uint32_t pad = (128u - (mc_smem_u32(mc_bricks) & 127u)) & 127u;
    TT* st[2];
    WT* sw[2];
    for (int k = 0; k < 2; ++k) {
        st[k] = reinterpret_cast<TT*>(mc_bricks + pad + (2 * k) * kBrick);
        sw[k] = reinterpret_cast<WT*>(mc_bricks + pad + (2 * k + 1) * kBrick);
    }
    const int tid = threadIdx.y * kMcX + threadIdx.x;
    const long nall = (long)tx_n * ty_n * tz_n;
    const long nt = a.tile_list ? min((long)*a.tile_count, nall) : nall;
    if ((mc_smem_u32(st[0]) & 127u) != 0u) {  // never expected: refuse rather than fault
        if (tid == 0 && a.error) atomicOr(a.error, ERRF_TMA);
        return;
    }
    auto origin = [&](long i, int& x0, int& y0, int& z0) {  // i-th tile of this launch
        const long t = a.tile_list ? (long)a.tile_list[i] : i;
        const int tx = (int)(t % tx_n), ty = (int)((t / tx_n) % ty_n), tz = (int)(t / ((long)tx_n * ty_n));
        x0 = tx * kMcX;
        y0 = ty * kMcY;
        z0 = tz * ZR;
    };
    auto issue = [&](int s, long t) {  // one thread
        int x0, y0, z0;
        origin(t, x0, y0, z0);
        const uint32_t bar = mc_smem_u32(&mbar[s]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kBytes) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
            "[%5];" ::"r"(mc_smem_u32(st[s])),
            "l"(&map_t), "r"(x0), "r"(y0), "r"(z0), "r"(bar)
            : "memory");
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
            "[%5];" ::"r"(mc_smem_u32(sw[s])),
            "l"(&map_w), "r"(x0), "r"(y0), "r"(z0), "r"(bar)
            : "memory");
    };
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mc_smem_u32(&mbar[0])));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mc_smem_u32(&mbar[1])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const long G = gridDim.x;
    if (tid == 0) {
        if ((long)blockIdx.x < nt) issue(0, blockIdx.x);
        if ((long)blockIdx.x + G < nt) issue(1, blockIdx.x + G);
    }
    const int nx = a.vol.dims[0] - 2, ny = a.vol.dims[1] - 2, nz = a.vol.dims[2] - 2;
    const int o00 = threadIdx.y * kMcTX + threadIdx.x;
    int k = 0;
    for (long t = blockIdx.x; t < nt; t += G, ++k) {
        const int s = k & 1;
        const uint32_t parity = (uint32_t)((k >> 1) & 1);
        const bool ok = mc_wait(mc_smem_u32(&mbar[s]), parity);
        if (__syncthreads_or(!ok)) {
            if (tid == 0 && a.error) atomicOr(a.error, ERRF_TMA | ERRF_TIMEOUT);
            // loads issued and not yet waited for: this tile's (stage s, if it timed out) and the next
            mc_wait(mc_smem_u32(&mbar[s]), parity);
            if (t + G < nt) mc_wait(mc_smem_u32(&mbar[s ^ 1]), (uint32_t)(((k + 1) >> 1) & 1));
            return;
        }
        if (tid == 0) q_n = 0;
        __syncthreads();
        int x0, y0, z0;
        origin(t, x0, y0, z0);
        const int x = x0 + threadIdx.x, y = y0 + threadIdx.y;
        const int z1 = min(z0 + ZR, nz);
        const bool col = x < nx && y < ny;
        for (int z = z0; z < z1; ++z) {
            const int s0 = (z - z0) * kSlice + o00, s1 = s0 + kSlice;
            int ci = 0;
            if (col) {
                const int off[8] = {s0 + kMcTX + 1, s0 + 1, s0, s0 + kMcTX, s1 + kMcTX + 1, s1 + 1, s1, s1 + kMcTX};
                bool any_zero = false;
#pragma unroll
                for (int c = 0; c < 8; ++c) any_zero |= smem_w_zero(sw[s], off[c]);
                if (!any_zero)
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        if (smem_t(st[s], off[c]) > a.iso) ci |= 1 << c;
            }
            const bool active = ci != 0 && ci != 255;
            const unsigned bal = __ballot_sync(0xffffffffu, active);
            if (bal) {
                const int lane = threadIdx.x & 31;
                unsigned base = 0;
                if (lane == 0) base = atomicAdd(&q_n, (unsigned)__popc(bal));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (active)
                    q[base + __popc(bal & ((1u << lane) - 1))] = (unsigned)ci | ((unsigned)threadIdx.x << 8) |
                                                                 ((unsigned)threadIdx.y << 13) | ((unsigned)(z - z0) << 16);
            }
        }
        __syncthreads();  // stage s has been read: it can take tile t + 2G
        if (tid == 0 && t + 2 * G < nt) issue(s, t + 2 * G);
        const unsigned nq = q_n;
        for (unsigned r0 = 0; r0 < nq; r0 += kMcX * kMcY) {
            const unsigned qi = r0 + tid;
            const bool act = qi < nq;
            const unsigned e = act ? q[qi] : 0u;
            mc_emit<kPoints, kMesh>(tsdf, a, x0 + (int)((e >> 8) & 31u), y0 + (int)((e >> 13) & 7u),
                                    z0 + (int)((e >> 16) & 63u), (int)(e & 255u), act, scratch[tid >> 5]);
        }
        __syncthreads();  // the queue is reused by the next tile
    }
}

__global__ void mc_vert_count_kernel(const unsigned* face_count, unsigned* vert_count) {
    *vert_count = 3u * *face_count;
}

// 3-D tiled map over one voxel array (element type `type`, `elem` bytes); the box is one CTA's
// brick of corner values.
static bool make_volume_map(CUtensorMap* map, const void* base, const Volume& vol, CUtensorMapDataType type,
                            size_t elem, int zr) {
    if ((vol.dims[0] * elem) % 16 != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0) return false;
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)vol.dims[0], (cuuint64_t)vol.dims[1], (cuuint64_t)vol.dims[2]};
    cuuint64_t strides[2] = {(cuuint64_t)vol.dims[0] * elem, (cuuint64_t)vol.dims[0] * vol.dims[1] * elem};
    cuuint32_t box[3] = {(cuuint32_t)kMcTX, (cuuint32_t)(kMcY + 1), (cuuint32_t)(zr + 1)};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, type, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

template <class TT, class WT, bool kPoints, bool kMesh, int ZR>
static void mc_launch_tma(const TT* tsdf, const McArgs& a, const CUtensorMap* mt, const CUtensorMap* mw,
                          cudaStream_t st) {
    constexpr int smem = (int)mc_tma_smem(sizeof(TT), ZR);
    static ContextOnce once;  // per instantiation: the dynamic shared memory opt-in
    once_per_context(once, [](int) {
        return note_cuda_error(cudaFuncSetAttribute(mc_tma_kernel<TT, WT, kPoints, kMesh, ZR>,
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    });
    const dim3 grid((unsigned)((a.vol.dims[0] - 2 + kMcX - 1) / kMcX), (unsigned)((a.vol.dims[1] - 2 + kMcY - 1) / kMcY),
                    (unsigned)((a.vol.dims[2] - 2 + ZR - 1) / ZR));
    mc_tma_kernel<TT, WT, kPoints, kMesh, ZR><<<grid, dim3(kMcX, kMcY), smem, st>>>(*mt, *mw, tsdf, a);
}

template <class TT, class WT, bool kPoints, bool kMesh, int ZR>
static void mc_launch_pipe(const TT* tsdf, const McArgs& a, const CUtensorMap* mt, const CUtensorMap* mw,
                           cudaStream_t st) {
    constexpr int smem = (int)(4 * mc_brick_bytes(sizeof(TT), ZR) + 128 + kMcX * kMcY / 32 * sizeof(McScratch<kMesh>));
    static ContextOnce once;  // per instantiation: opt-in and resident CTAs per SM, per device
    static int per_sm_dev[kMaxDevices], sms_dev[kMaxDevices];
    once_per_context(once, [](int dev) {
        int per_sm = 0, sms = 0;
        cudaFuncSetAttribute(mc_pipe_kernel<TT, WT, kPoints, kMesh, ZR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mc_pipe_kernel<TT, WT, kPoints, kMesh, ZR>, kMcX * kMcY,
                                                      smem);
        cudaGetLastError();
        per_sm_dev[dev] = per_sm < 1 ? 1 : per_sm;
        sms_dev[dev] = sms < 1 ? 1 : sms;
        return (int)AFX_OK;
    });
    int dev = 0;
    cudaGetDevice(&dev);
    const int per_sm = per_sm_dev[dev] < 1 ? 1 : per_sm_dev[dev], sms = sms_dev[dev] < 1 ? 1 : sms_dev[dev];
    const int tx = (a.vol.dims[0] - 2 + kMcX - 1) / kMcX, ty = (a.vol.dims[1] - 2 + kMcY - 1) / kMcY,
              tz = (a.vol.dims[2] - 2 + ZR - 1) / ZR;
    const long nt = (long)tx * ty * tz;
    const long grid = nt < (long)sms * per_sm ? nt : (long)sms * per_sm;
    McArgs b = a;
    if (a.occ && a.tile_list && a.tile_count) {
        cudaMemsetAsync(a.tile_count, 0, sizeof(unsigned), st);
        mc_tile_list_kernel<<<grid_for(nt, 256), 256, 0, st>>>(a, tx, ty, tz, ZR);
    } else {
        b.tile_list = nullptr;
    }
    mc_pipe_kernel<TT, WT, kPoints, kMesh, ZR><<<(unsigned)grid, dim3(kMcX, kMcY), smem, st>>>(*mt, *mw, tsdf, b, tx,
                                                                                              ty, tz);
}

// Words of the occupied-tile list for a volume (count + one entry per tile of the shallowest depth, 4).
size_t mc_tile_ws_words(const Volume& vol) {
    const long tx = (vol.dims[0] - 2 + kMcX - 1) / kMcX, ty = (vol.dims[1] - 2 + kMcY - 1) / kMcY,
               tz = (vol.dims[2] - 2 + 4 - 1) / 4;
    return (size_t)(1 + (tx > 0 ? tx : 0) * (ty > 0 ? ty : 0) * (tz > 0 ? tz : 0));
}

// tile: kMcTileTma16 (default), kMcTileTma8, kMcTileTma32 (TMA bricks of that many cubes along z),
// kMcTilePipe8 / kMcTilePipe16 / kMcTilePipe4 (persistent grid with two stages of bricks 8, 16 or 4
// cubes deep) or
// kMcTileColumn (sweep from global memory).  mt/mw are the maps encoded for that depth, or null (then the
// sweep runs).
template <class TT, class WT, bool kPoints, bool kMesh>
static void mc_launch(const TT* tsdf, const WT* weights, const McArgs& a, const CUtensorMap* mt, const CUtensorMap* mw,
                      int tile, cudaStream_t st) {
    if (mt && tile == kMcTilePipe8) {
        mc_launch_pipe<TT, WT, kPoints, kMesh, 8>(tsdf, a, mt, mw, st);
    } else if (mt && tile == kMcTilePipe4) {
        mc_launch_pipe<TT, WT, kPoints, kMesh, 4>(tsdf, a, mt, mw, st);
    } else if (mt && tile == kMcTilePipe16) {
        mc_launch_pipe<TT, WT, kPoints, kMesh, 16>(tsdf, a, mt, mw, st);
    } else if (mt && tile == kMcTileTma8) {
        mc_launch_tma<TT, WT, kPoints, kMesh, 8>(tsdf, a, mt, mw, st);
    } else if (mt && tile == kMcTileTma32) {
        mc_launch_tma<TT, WT, kPoints, kMesh, 32>(tsdf, a, mt, mw, st);
    } else if (mt) {
        mc_launch_tma<TT, WT, kPoints, kMesh, 16>(tsdf, a, mt, mw, st);
    } else {
        constexpr int kRows = kSweepY * kSweepWarps;
        const dim3 grid((unsigned)((a.vol.dims[0] - 2 + 30) / 31), (unsigned)((a.vol.dims[1] - 2 + kRows - 1) / kRows),
                        (unsigned)((a.vol.dims[2] - 2 + kSweepZ - 1) / kSweepZ));
        constexpr int smem = kSweepWarps * (int)sizeof(McScratch<kMesh>);
        static ContextOnce once;
        once_per_context(once, [](int) {
            return note_cuda_error(cudaFuncSetAttribute(mc_sweep_kernel<TT, WT, kPoints, kMesh>,
                                                        cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        });
        mc_sweep_kernel<TT, WT, kPoints, kMesh><<<grid, 32 * kSweepWarps, smem, st>>>(tsdf, weights, a);
    }
}

template <class TT, class WT>
static void mc_launch_any(const TT* tsdf, const WT* weights, const McArgs& a, const CUtensorMap* mt,
                          const CUtensorMap* mw, bool P, bool M, int tile, cudaStream_t st) {
    if (P && M) mc_launch<TT, WT, true, true>(tsdf, weights, a, mt, mw, tile, st);
    else if (P) mc_launch<TT, WT, true, false>(tsdf, weights, a, mt, mw, tile, st);
    else mc_launch<TT, WT, false, true>(tsdf, weights, a, mt, mw, tile, st);
}

int mc_fused_impl(const void* tsdf, const void* weights, int fmt, const Volume& vol, float iso, float* points,
                  unsigned* point_count, long point_cap, float* verts, unsigned* vert_count, long vert_cap, int* faces,
                  unsigned* face_count, long face_cap, cudaStream_t st, int* error, int tile,
                  const unsigned char* occ, unsigned* tile_ws, bool occ_positive) {
    int rc = upload_tables();
    if (rc) return rc;
    McArgs a;
    a.vol = vol;
    a.iso = iso;
    a.points = points;
    a.point_count = point_count;
    a.point_cap = point_cap;
    a.verts = verts;
    a.face_count = face_count;
    a.vert_count = vert_count;
    a.face_cap = face_cap < vert_cap / 3 ? face_cap : vert_cap / 3;
    a.faces = faces;
    a.error = error;
    a.occ = occ;
    a.occ_positive = occ_positive;
    a.tile_count = tile_ws;
    a.tile_list = tile_ws ? tile_ws + 1 : nullptr;
    a.nbx = (vol.dims[0] + 7) / 8;
    a.nby = (vol.dims[1] + 7) / 8;
    a.nbz = (vol.dims[2] + 7) / 8;
    const long ncubes = (long)(vol.dims[0] - 2) * (vol.dims[1] - 2) * (vol.dims[2] - 2);
    if (ncubes <= 0) return AFX_OK;
    const bool P = points != nullptr, M = verts != nullptr;
    if (!P && !M) return AFX_OK;
    // TMA bricks where the caller can receive a load-timeout report and the maps encode
    CUtensorMap mt, mw;
    const bool f16 = fmt == kVoxF16;
    const size_t elem = vox_bytes(fmt);
    const int zr = (tile == kMcTileTma8 || tile == kMcTilePipe8) ? 8 : tile == kMcTilePipe4 ? 4 : tile == kMcTileTma32 ? 32 : 16;
    const bool tma = error && tile != kMcTileColumn &&
                     make_volume_map(&mt, tsdf, vol, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 :
                                                           CU_TENSOR_MAP_DATA_TYPE_FLOAT32, elem, zr) &&
                     make_volume_map(&mw, weights, vol, f16 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 :
                                                              CU_TENSOR_MAP_DATA_TYPE_FLOAT32, elem, zr);
    if (f16)
        mc_launch_any(static_cast<const __half*>(tsdf), static_cast<const unsigned short*>(weights), a,
                      tma ? &mt : nullptr, tma ? &mw : nullptr, P, M, tile, st);
    else
        mc_launch_any(static_cast<const float*>(tsdf), static_cast<const float*>(weights), a, tma ? &mt : nullptr,
                      tma ? &mw : nullptr, P, M, tile, st);
    AFX_LAUNCH_CHECK();
    if (M && vert_count) {
        mc_vert_count_kernel<<<1, 1, 0, st>>>(face_count, vert_count);
        AFX_LAUNCH_CHECK();
    }
    return AFX_OK;
}

// ------------------------------------------------------------------------------------
// Lexicographic sort + unique of float triples
// ------------------------------------------------------------------------------------

struct Key3 {
    unsigned k[3];
};

AFX_D unsigned f2key(float f) {
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
AFX_D float key2f(unsigned k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }
AFX_D bool key_less(const Key3& a, const Key3& b) {  // without branches: lanes compare different keys
    const bool l0 = a.k[0] < b.k[0], e0 = a.k[0] == b.k[0], l1 = a.k[1] < b.k[1], e1 = a.k[1] == b.k[1];
    return l0 | (e0 & (l1 | (e1 & (a.k[2] < b.k[2]))));
}
AFX_D Key3 key_pick(bool first, const Key3& a, const Key3& b) {
    return {{first ? a.k[0] : b.k[0], first ? a.k[1] : b.k[1], first ? a.k[2] : b.k[2]}};
}
AFX_D bool key_le(const Key3& a, const Key3& b) { return !key_less(b, a); }

// The points are sorted in tiles of kSortTile (one CTA each), the sorted
// runs merged pairwise in passes over all SMs, then made unique by float equality of consecutive
// points and compacted in order back into the cloud.  The number of points is on the device, so as
// many passes are launched as the capacity can need; those that the live number does not need return
// at once.  The pass a run length belongs to decides which buffer it reads.
// Bound: latency of a pass (a search for the split, one load, a merge of kSortPer keys per thread).
// 450,000 points in room for a million: 102 us (131 with launches that each wait for the one before to be gone; one cluster of
// 16 CTAs doing all of it 1,365); 5,000 points in the same room 50 us (78, 70), none 40 (57, 18).
constexpr int kSortTile = 2048;
constexpr int kSortPer = 8;  // keys per thread
constexpr int kSortThreads = kSortTile / kSortPer;
constexpr int kUniqueThreads = 1024;
constexpr long kSortBlocks = 608;  // four CTAs per SM

// The launches after the first may start while the one before still runs, and wait here for all of it: an empty pass --
// most are, where a cloud is small for its capacity -- costs about 1 us instead of 3.5.  The next launch is
// let in only after that, so a launch waits for all before it.
AFX_D void sort_pass_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Passes that merge runs of kSortTile into one of n.
__host__ __device__ inline int sort_passes(long n) {
    int p = 0;
    for (long L = kSortTile; L < n; L <<= 1) ++p;
    return p;
}

AFX_D Key3 sort_key(const float* p) {
    Key3 k;
    k.k[0] = f2key(p[0]);
    k.k[1] = f2key(p[1]);
    k.k[2] = f2key(p[2]);
    return k;
}

// A tile in shared memory, with a key of padding after every kSortPer: a warp's threads then work on
// kSortPer keys each without meeting in the same banks.
struct SortTile {
    Key3 k[kSortTile + kSortTile / kSortPer];
    AFX_D Key3& operator[](int i) { return k[i + i / kSortPer]; }
};

// Outputs [q0, q0 + kSortPer) of merging the sorted runs s[at, at + la) and s[at + la, at + la + lb), into
// registers.
AFX_D void merge_serial(SortTile& s, int at, int la, int lb, int q0, Key3 (&out)[kSortPer]) {
    int lo = max(0, q0 - lb), hi = min(q0, la);
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (key_le(s[at + mid], s[at + la + q0 - 1 - mid])) lo = mid + 1;
        else hi = mid;
    }
    int ia = lo, ib = q0 - lo;
    const int end = at + la + lb - 1;
    Key3 a = s[min(at + ia, end)], b = s[min(at + la + ib, end)];
#pragma unroll
    for (int q = 0; q < kSortPer; ++q) {
        const bool takeA = (ib >= lb) | ((ia < la) & key_le(a, b));
        out[q] = key_pick(takeA, a, b);
        ia += takeA;
        ib += !takeA;
        const Key3 next = s[min(takeA ? at + ia : at + la + ib, end)];
        a = key_pick(takeA, next, a);
        b = key_pick(takeA, b, next);
    }
}

// Each tile of up to kSortTile points (padding sorts last) sorted into `out`: kSortPer keys per thread by a
// sorting network in registers, then runs merged in shared memory, each thread its kSortPer outputs of
// a merge through registers (a bitonic sort of the tile in shared memory took 50 us for 112 tiles,
// bound by shared-memory accesses).
__global__ void __launch_bounds__(kSortThreads) sort_tiles_kernel(const float* __restrict__ pts, const unsigned* count,
                                                                 long n_max, Key3* out, unsigned* done) {
    __shared__ SortTile s;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long n = min((long)*count, n_max);
    if (blockIdx.x == 0 && threadIdx.x == 0) *done = 0u;
    for (long base = blockIdx.x * (long)kSortTile; base < n; base += gridDim.x * (long)kSortTile) {
        Key3 v[kSortPer];
#pragma unroll
        for (int k = 0; k < kSortPer; ++k) {
            const long j = base + k * kSortThreads + threadIdx.x;
            if (j < n) v[k] = sort_key(pts + 3 * j);
            else v[k].k[0] = v[k].k[1] = v[k].k[2] = 0xffffffffu;
        }
#pragma unroll
        for (int round = 0; round < kSortPer; ++round)  // odd-even transposition
#pragma unroll
            for (int k = round & 1; k + 1 < kSortPer; k += 2) {
                const bool swap = key_less(v[k + 1], v[k]);
                const Key3 t = key_pick(swap, v[k], v[k + 1]);
                v[k] = key_pick(swap, v[k + 1], v[k]);
                v[k + 1] = t;
            }
        const int q0 = threadIdx.x * kSortPer;
#pragma unroll
        for (int k = 0; k < kSortPer; ++k) s[q0 + k] = v[k];
        __syncthreads();
        for (int run = kSortPer; run < kSortTile; run <<= 1) {
            const int pair = q0 / (2 * run) * (2 * run);
            merge_serial(s, pair, run, run, q0 - pair, v);
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kSortPer; ++k) s[q0 + k] = v[k];
            __syncthreads();
        }
        for (int i = threadIdx.x; i < kSortTile; i += kSortThreads)
            if (base + i < n) out[base + i] = s[i];
        __syncthreads();
    }
}

// Merge path: how many of the first d merged keys come from A[0, na), the rest from B[0, nb).  One warp:
// 32 probes per step.
AFX_D long merge_split(const Key3* __restrict__ A, long na, const Key3* __restrict__ B, long nb, long d) {
    const int lane = threadIdx.x & 31;
    long lo = max(0L, d - nb), hi = min(d, na);
    while (lo < hi) {
        const long mid = lo + (hi - lo) * lane / 32;  // lane 0: lo; ascending
        const unsigned yes = __ballot_sync(0xffffffffu, key_le(A[mid], B[d - 1 - mid]));
        const int t = __popc(yes);  // the first t probes are before the split
        const long first_no = __shfl_sync(0xffffffffu, mid, t & 31), last_yes = __shfl_sync(0xffffffffu, mid, (t + 31) & 31);
        if (t < 32) hi = first_no;
        if (t > 0) lo = last_yes + 1;
    }
    return lo;
}

// One pass: runs of length L of `in` merged pairwise into `out`, kSortTile outputs per CTA and step.
__global__ void __launch_bounds__(kSortThreads) merge_pass_kernel(const Key3* __restrict__ in, Key3* __restrict__ out,
                                                                 const unsigned* count, long n_max, long L) {
    __shared__ SortTile s;
    __shared__ long split[2];
    sort_pass_begin();
    const long n = min((long)*count, n_max);
    if (L >= n) return;  // one run already
    for (long o0 = blockIdx.x * (long)kSortTile; o0 < n; o0 += gridDim.x * (long)kSortTile) {
        const long pair = o0 / (2 * L) * (2 * L);
        const Key3 *A = in + pair, *B = in + pair + L;
        const long na = min(L, n - pair), nb = max(0L, min(L, n - pair - L));
        const long d0 = o0 - pair, d1 = min(d0 + kSortTile, na + nb);
        const int w = threadIdx.x >> 5;
        __syncthreads();  // the step before is done with s and split
        if (w < 2) {
            const long i = merge_split(A, na, B, nb, w == 0 ? d0 : d1);
            if ((threadIdx.x & 31) == 0) split[w] = i;
        }
        __syncthreads();
        const long i0 = split[0], j0 = d0 - i0;
        const int la = (int)(split[1] - i0), tot = (int)(d1 - d0), lb = tot - la;
        for (int t = threadIdx.x; t < tot; t += kSortThreads) s[t] = t < la ? A[i0 + t] : B[j0 + (t - la)];
        __syncthreads();
        Key3 v[kSortPer];
        const int q0 = threadIdx.x * kSortPer;
        if (q0 < tot) merge_serial(s, 0, la, lb, q0, v);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSortPer; ++k)
            if (q0 + k < tot) s[q0 + k] = v[k];
        __syncthreads();
        for (int t = threadIdx.x; t < tot; t += kSortThreads) out[o0 + t] = s[t];
    }
}

AFX_D bool key_same_point(const Key3& a, const Key3& b) {
    return key2f(a.k[0]) == key2f(b.k[0]) && key2f(a.k[1]) == key2f(b.k[1]) && key2f(a.k[2]) == key2f(b.k[2]);
}

// Points of each tile that differ from the one before them.
__global__ void __launch_bounds__(kUniqueThreads) unique_count_kernel(const Key3* buf0, const Key3* buf1,
                                                                   const unsigned* count, long n_max, unsigned* tile_cnt) {
    sort_pass_begin();
    const long n = min((long)*count, n_max), tiles = (n + kSortTile - 1) / kSortTile;
    const Key3* src = sort_passes(n) & 1 ? buf1 : buf0;
    for (long t = blockIdx.x; t < tiles; t += gridDim.x) {
        int c = 0;
        for (long i0 = t * kSortTile; i0 < min(n, (t + 1) * kSortTile); i0 += kUniqueThreads) {
            const long i = i0 + threadIdx.x;
            c += __syncthreads_count(i < n && (i == 0 || !key_same_point(src[i - 1], src[i])));
        }
        if (threadIdx.x == 0) tile_cnt[t] = (unsigned)c;
    }
}

// Ordered compaction: a tile starts after the counts of those before it.  The block that finishes last
// writes the new number of points (no block reads the old one any more).
__global__ void __launch_bounds__(kUniqueThreads) unique_compact_kernel(float* pts, const Key3* buf0, const Key3* buf1,
                                                                     unsigned* count, long n_max,
                                                                     const unsigned* __restrict__ tile_cnt, unsigned* done) {
    __shared__ unsigned wsum[kUniqueThreads / 32];
    sort_pass_begin();
    const long n = min((long)*count, n_max), tiles = (n + kSortTile - 1) / kSortTile;
    const Key3* src = sort_passes(n) & 1 ? buf1 : buf0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    auto sum_before = [&](long t) {  // of tile_cnt[0, t), in every thread
        unsigned c = 0;
        for (long k = threadIdx.x; k < t; k += kUniqueThreads) c += tile_cnt[k];
        c = warp_sum(c);
        __syncthreads();
        if (lane == 0) wsum[w] = c;
        __syncthreads();
        return warp_sum(wsum[lane]);
    };
    for (long t = blockIdx.x; t < tiles; t += gridDim.x) {
        unsigned run = sum_before(t);
        // one element per thread per step, in index order
        for (long r0 = t * kSortTile; r0 < min(n, (t + 1) * kSortTile); r0 += kUniqueThreads) {
            const long i = r0 + threadIdx.x;
            const bool keep = i < n && (i == 0 || !key_same_point(src[i - 1], src[i]));
            const unsigned bal = __ballot_sync(0xffffffffu, keep);
            __syncthreads();
            if (lane == 0) wsum[w] = __popc(bal);
            __syncthreads();
            const unsigned c = wsum[lane], before = warp_sum(lane < w ? c : 0u), all = warp_sum(c);
            if (keep) {
                const Key3 k = src[i];
                float* o = pts + 3 * (long)(run + before + __popc(bal & ((1u << lane) - 1)));
                o[0] = key2f(k.k[0]);
                o[1] = key2f(k.k[1]);
                o[2] = key2f(k.k[2]);
            }
            run += all;
        }
    }
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last || n == 0) return;
    const unsigned total = sum_before(tiles);
    if (threadIdx.x == 0) *count = total;
}

static size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

size_t sort_unique_workspace_size(long n_max) {
    if (n_max < 1) n_max = 1;
    return 2 * al(n_max * sizeof(Key3)) + al(((n_max + kSortTile - 1) / kSortTile) * 4) + 256;
}

int sort_unique_impl(float* pts, unsigned* count, long n_max, void* ws, size_t ws_bytes, cudaStream_t st) {
    if (n_max <= 0) return AFX_OK;
    if (!ws || ws_bytes < sort_unique_workspace_size(n_max)) return AFX_ERR_WORKSPACE;
    char* p = static_cast<char*>(ws);
    Key3* buf[2];
    for (Key3*& b : buf) {
        b = reinterpret_cast<Key3*>(p);
        p += al(n_max * sizeof(Key3));
    }
    unsigned* tile_cnt = reinterpret_cast<unsigned*>(p);
    p += al(((n_max + kSortTile - 1) / kSortTile) * 4);
    unsigned* done = reinterpret_cast<unsigned*>(p);
    const long tiles = (n_max + kSortTile - 1) / kSortTile;
    const unsigned grid = (unsigned)(tiles < kSortBlocks ? tiles : kSortBlocks);
    sort_tiles_kernel<<<grid, kSortThreads, 0, st>>>(pts, count, n_max, buf[0], done);
    AFX_LAUNCH_CHECK();
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kSortThreads);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const int passes = sort_passes(n_max);
    for (int k = 0; k < passes; ++k) {
        AFX_CUDA(cudaLaunchKernelEx(&cfg, merge_pass_kernel, (const Key3*)buf[k & 1], buf[(k & 1) ^ 1], (const unsigned*)count, n_max,
                                    (long)kSortTile << k));
        AFX_LAUNCH_CHECK();
    }
    cfg.blockDim = dim3(kUniqueThreads);
    AFX_CUDA(cudaLaunchKernelEx(&cfg, unique_count_kernel, (const Key3*)buf[0], (const Key3*)buf[1], (const unsigned*)count, n_max,
                                tile_cnt));
    AFX_LAUNCH_CHECK();
    AFX_CUDA(cudaLaunchKernelEx(&cfg, unique_compact_kernel, pts, (const Key3*)buf[0], (const Key3*)buf[1], count, n_max,
                                (const unsigned*)tile_cnt, done));
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// ------------------------------------------------------------------------------------
// Column-bucket sort + unique of a marching-cubes point cloud of a known volume.
//
// Every point of the cloud has x in [-half, half] of the volume, and b(x) = trunc((x + half) * inv)
// (clamped) is monotone in x under IEEE rounding, so bucketing by voxel column keeps the
// lexicographic order between buckets and puts equal points (-0 and +0 included) in one bucket.
// Pipeline: count per bucket, scan, scatter (order within a bucket arbitrary), one CTA per bucket
// sorting it in shared memory and counting its unique points, scan of those counts, ordered
// compaction back into the cloud.  A bucket larger than kBucketCap (a surface lying along one x
// column) is sorted by its CTA in runs of kBucketCap in shared memory that are then merged pairwise
// in global memory (merge path, ties from the left run first) between the key buffer and the second
// buffer of the workspace.
// ------------------------------------------------------------------------------------

constexpr int kBucketCap = 8192;  // keys per bucket sorted in shared memory (96 KB)
constexpr int kBucketThreads = 512;

struct BucketArgs {
    float half0, inv0;
    int nb;
};

AFX_D int bucket_of(float x, const BucketArgs& a) {
    const float u = (x + a.half0) * a.inv0;
    const int b = u > 0.f ? f2i(u) : 0;
    return b >= a.nb ? a.nb - 1 : b;
}

struct BucketWs {
    unsigned* cnt;     // [nb] points; cleared together with the next
    unsigned* cursor;  // [nb]
    unsigned* off;     // [nb + 1]
    unsigned* ucnt;    // [nb] distinct points
};

__global__ void bucket_count_kernel(const float* __restrict__ pts, const unsigned* count, long n_max, BucketArgs a,
                                    unsigned* cnt) {
    const long n = min((long)*count, n_max);
    AFX_GRID_STRIDE(i, n) atomicAdd(cnt + bucket_of(pts[3 * i], a), 1u);
}

// The points into their buckets.  Every CTA forms the buckets' offsets for itself (a launch of one CTA for a few
// hundred sums cost more); the first one leaves them for the launches after this.
__global__ void __launch_bounds__(256) bucket_scatter_kernel(const float* __restrict__ pts, const unsigned* count, long n_max,
                                                             BucketArgs a, BucketWs ws, Key3* keys, int* error) {
    extern __shared__ __align__(16) unsigned s_off[];
    __shared__ unsigned s_sum[8];
    const long n = min((long)*count, n_max);
    if ((long)blockIdx.x * blockDim.x >= n && blockIdx.x != 0) return;
    const int per = (a.nb + 255) / 256, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int lo = min(a.nb, (int)threadIdx.x * per), hi = min(a.nb, lo + per);
    unsigned sum = 0;
    for (int i = lo; i < hi; ++i) sum += ws.cnt[i];
    unsigned x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_sum[w] = x;
    __syncthreads();
    unsigned run = x - sum;
    for (int q = 0; q < w; ++q) run += s_sum[q];
    for (int i = lo; i < hi; ++i) {
        s_off[i] = run;
        if (blockIdx.x == 0) ws.off[i] = run;
        run += ws.cnt[i];
    }
    if (blockIdx.x == 0 && threadIdx.x == 255) ws.off[a.nb] = run;
    __syncthreads();
    AFX_GRID_STRIDE(i, n) {
        Key3 k;
        k.k[0] = f2key(pts[3 * i]);
        k.k[1] = f2key(pts[3 * i + 1]);
        k.k[2] = f2key(pts[3 * i + 2]);
        const int b = bucket_of(pts[3 * i], a);
        const unsigned pos = s_off[b] + atomicAdd(ws.cursor + b, 1u);
        if (pos < (unsigned long)n) keys[pos] = k;
        else if (error) atomicOr(error, ERRF_INDEX);
    }
}

// Bitonic sort of m <= kBucketCap keys at g in shared memory (padded to a power of two with keys that
// sort last), written back to g.
AFX_D Key3 key_shfl_xor(Key3 k, int o) {
    return {{__shfl_xor_sync(0xffffffffu, k.k[0], o), __shfl_xor_sync(0xffffffffu, k.k[1], o),
             __shfl_xor_sync(0xffffffffu, k.k[2], o)}};
}

// Bitonic steps of one key per lane: partners `from`, from / 2, .. 1 lanes apart.  Of equal keys each lane keeps its own.
AFX_D Key3 key_lane_merge(Key3 x, int from, bool asc) {
    const int lane = threadIdx.x & 31;
    for (int o = from; o > 0; o >>= 1) {
        const Key3 y = key_shfl_xor(x, o);
        if (((lane & o) == 0) == asc ? key_less(y, x) : key_less(x, y)) x = y;
    }
    return x;
}

// Partners less than 32 apart are lanes of a warp, so only the wider steps need a barrier (10 instead of 45 for 512
// keys).  bucket_sort_kernel in the 256^3 sequence: 12.9 -> 9.0 us, in the 512^3 sequence 42 -> 32 us.
AFX_D void bucket_bitonic(Key3* g, unsigned m, Key3* sk) {
    unsigned P = 32;
    while (P < m) P <<= 1;
    __syncthreads();
    for (unsigned i = threadIdx.x; i < P; i += blockDim.x) {
        Key3 k;
        if (i < m) k = g[i];
        else k.k[0] = k.k[1] = k.k[2] = 0xffffffffu;
        for (unsigned size = 2; size <= 32; size <<= 1) k = key_lane_merge(k, (int)(size >> 1), (i & size) == 0);
        sk[i] = k;
    }
    __syncthreads();
    for (unsigned size = 64; size <= P; size <<= 1) {
        for (unsigned stride = size >> 1; stride >= 32; stride >>= 1) {
            for (unsigned q = threadIdx.x; q < P / 2; q += blockDim.x) {
                const unsigned i = 2 * stride * (q / stride) + (q % stride), j = i + stride;
                const bool asc = (i & size) == 0;
                const Key3 x = sk[i], y = sk[j];
                if (key_less(y, x) == asc) {
                    sk[i] = y;
                    sk[j] = x;
                }
            }
            __syncthreads();
        }
        for (unsigned i = threadIdx.x; i < P; i += blockDim.x) sk[i] = key_lane_merge(sk[i], 16, (i & size) == 0);
        __syncthreads();
    }
    for (unsigned i = threadIdx.x; i < m; i += blockDim.x) g[i] = sk[i];
    __syncthreads();
}

// Stable merge of the sorted runs A[0, la) and B[0, lb) into out by the whole CTA: each thread finds
// where its share of the output starts on the merge path (binary search: the first i with
// B[k - i - 1] < A[i]) and merges its share sequentially.
AFX_D void cta_merge(const Key3* A, unsigned la, const Key3* B, unsigned lb, Key3* out) {
    const unsigned total = la + lb, per = (total + blockDim.x - 1) / blockDim.x;
    const unsigned k0 = min(total, threadIdx.x * per), k1 = min(total, k0 + per);
    if (k0 >= k1) return;
    unsigned lo = k0 > lb ? k0 - lb : 0u, hi = min(k0, la);
    while (lo < hi) {
        const unsigned mid = (lo + hi) >> 1;
        if (key_less(B[k0 - mid - 1], A[mid])) hi = mid;
        else lo = mid + 1;
    }
    unsigned i = lo, j = k0 - lo;
    for (unsigned k = k0; k < k1; ++k) {
        const bool takeA = i < la && (j >= lb || !key_less(B[j], A[i]));
        out[k] = takeA ? A[i++] : B[j++];
    }
}

// One CTA per bucket: sort it in place (in shared memory, or in runs merged through `scratch` when it
// holds more than kBucketCap points) and count its unique points.
__global__ void __launch_bounds__(kBucketThreads) bucket_sort_kernel(Key3* keys, Key3* scratch, const unsigned* off,
                                                                   unsigned* ucnt, long n_max,
                                                                   int* error) {
    extern __shared__ __align__(16) Key3 sk[];
    __shared__ unsigned wsum[kBucketThreads / 32];
    const int b = blockIdx.x;
    const unsigned lo = off[b], n = off[b + 1] - lo;
    if (lo > off[b + 1] || (long)off[b + 1] > n_max) {  // never expected: skip, flag
        if (threadIdx.x == 0) {
            ucnt[b] = 0;
            if (error) atomicOr(error, ERRF_INDEX);
        }
        return;
    }
    if (n == 0) {
        if (threadIdx.x == 0) ucnt[b] = 0;
        return;
    }
    Key3* g = keys + lo;
    if (n <= (unsigned)kBucketCap) {
        bucket_bitonic(g, n, sk);
    } else {
        for (unsigned c0 = 0; c0 < n; c0 += kBucketCap) bucket_bitonic(g + c0, min((unsigned)kBucketCap, n - c0), sk);
        Key3 *src = g, *dst = scratch + lo;
        for (unsigned L = kBucketCap; L < n; L *= 2) {
            for (unsigned s0 = 0; s0 < n; s0 += 2 * L) {
                const unsigned la = min(L, n - s0), lb = min(L, n - s0 - la);
                cta_merge(src + s0, la, src + s0 + la, lb, dst + s0);
            }
            __syncthreads();
            Key3* t = src;
            src = dst;
            dst = t;
        }
        if (src != g) {
            for (unsigned i = threadIdx.x; i < n; i += blockDim.x) g[i] = src[i];
            __syncthreads();
        }
    }
    unsigned c = 0;
    const bool here = n <= (unsigned)kBucketCap;  // still in shared memory
    for (unsigned i = threadIdx.x; i < n; i += blockDim.x)
        c += (i == 0 || !(here ? key_same_point(sk[i - 1], sk[i]) : key_same_point(g[i - 1], g[i]))) ? 1u : 0u;
    c = warp_sum(c);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int w = 0; w < kBucketThreads / 32; ++w) t += wsum[w];
        ucnt[b] = t;
    }
}

// One CTA per bucket: its unique points, in order, at the bucket's place in the output.
__global__ void __launch_bounds__(kBucketThreads) bucket_compact_kernel(const Key3* keys, BucketWs ws,
                                                                      int nb, float* pts, long n_max, int* error,
                                                                      unsigned* count, const float* shift,
                                                                      unsigned* count_copy) {
    __shared__ unsigned wsum[kBucketThreads / 32];
    __shared__ unsigned s_run;
    const int b = blockIdx.x;
    const unsigned* off = ws.off;
    // distinct points of the buckets before this one; the last one's total is the new count
    if (threadIdx.x == 0) s_run = 0u;
    __syncthreads();
    unsigned sum = 0;
    for (int q = threadIdx.x; q < b; q += blockDim.x) sum += ws.ucnt[q];
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&s_run, sum);
    __syncthreads();
    const unsigned first = s_run, after = first + ws.ucnt[b];
    if (b == nb - 1 && threadIdx.x == 0) {
        *count = after;
        if (count_copy) *count_copy = after;
    }
    if (off[b] > off[b + 1] || (long)off[b + 1] > n_max || (long)after > n_max) {
        if (threadIdx.x == 0 && error) atomicOr(error, ERRF_INDEX);
        return;
    }
    const unsigned lo = off[b], n = off[b + 1] - lo;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float t[3] = {shift ? shift[0] : 0.f, shift ? shift[1] : 0.f, shift ? shift[2] : 0.f};
    unsigned run = first;
    for (unsigned r0 = 0; r0 < n; r0 += blockDim.x) {
        const unsigned i = r0 + threadIdx.x;
        const bool keep = i < n && (i == 0 || !key_same_point(keys[lo + i - 1], keys[lo + i]));
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        __syncthreads();
        if (lane == 0) wsum[w] = __popc(bal);
        __syncthreads();
        unsigned before = 0, all = 0;
        for (int k = 0; k < kBucketThreads / 32; ++k) {
            const unsigned v = wsum[k];
            if (k < w) before += v;
            all += v;
        }
        if (keep) {
            const Key3 k = keys[lo + i];
            float* o = pts + 3 * (long)(run + before + __popc(bal & ((1u << lane) - 1)));
#pragma unroll
            for (int c = 0; c < 3; ++c) o[c] = shift ? key2f(k.k[c]) + t[c] : key2f(k.k[c]);
        }
        run += all;
    }
}

size_t sort_unique_volume_workspace_size(long n_max, int nb) {
    return sort_unique_workspace_size(n_max) + al((size_t)(4 * nb + 1) * 4);
}

int sort_unique_volume_impl(float* pts, unsigned* count, long n_max, void* ws, size_t ws_bytes, const Volume& vol,
                            cudaStream_t st, int* error, const float* shift, unsigned* count_copy) {
    if (n_max <= 0) return AFX_OK;
    const int nb = vol.dims[0] + 1;
    if (nb > 8 * 1024) {
        int rc = sort_unique_impl(pts, count, n_max, ws, ws_bytes, st);
        if (!rc && shift) rc = translate_dev_impl(pts, pts, count, n_max, shift, 1.f, st);
        if (!rc && count_copy) AFX_CUDA(cudaMemcpyAsync(count_copy, count, 4, cudaMemcpyDeviceToDevice, st));
        return rc;
    }
    if (!ws || ws_bytes < sort_unique_volume_workspace_size(n_max, nb)) return AFX_ERR_WORKSPACE;
    const size_t base = sort_unique_workspace_size(n_max);
    unsigned* u = reinterpret_cast<unsigned*>(static_cast<char*>(ws) + base);
    BucketWs w{u, u + nb, u + 2 * nb, u + 3 * nb + 1};
    Key3* keys = reinterpret_cast<Key3*>(ws);
    BucketArgs a{vol.half[0], vol.inv[0], nb};
    static ContextOnce once;
    once_per_context(once, [](int) {
        return note_cuda_error(cudaFuncSetAttribute(bucket_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)(kBucketCap * sizeof(Key3))));
    });
    AFX_CUDA(cudaMemsetAsync(w.cnt, 0, 2 * nb * 4, st));
    bucket_count_kernel<<<grid_for(n_max, 256), 256, 0, st>>>(pts, count, n_max, a, w.cnt);
    AFX_LAUNCH_CHECK();
    bucket_scatter_kernel<<<grid_for(n_max, 256), 256, nb * sizeof(unsigned), st>>>(pts, count, n_max, a, w, keys, error);
    AFX_LAUNCH_CHECK();
    Key3* scratch = reinterpret_cast<Key3*>(static_cast<char*>(ws) + al(n_max * sizeof(Key3)));  // the second buffer
    bucket_sort_kernel<<<nb, kBucketThreads, kBucketCap * sizeof(Key3), st>>>(keys, scratch, w.off, w.ucnt, n_max, error);
    AFX_LAUNCH_CHECK();
    bucket_compact_kernel<<<nb, kBucketThreads, 0, st>>>(keys, w, nb, pts, n_max, error, count, shift, count_copy);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

__global__ void translate_kernel(float* pts, const unsigned* count, long n_max, float tx, float ty, float tz) {
    long n = count ? min((long)*count, n_max) : n_max;
    long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    pts[3 * i] = pts[3 * i] + tx;
    pts[3 * i + 1] = pts[3 * i + 1] + ty;
    pts[3 * i + 2] = pts[3 * i + 2] + tz;
}

__global__ void translate_dev_kernel(float* dst, const float* src, const unsigned* count, long n_max, const float* t,
                                     float sign) {
    const long n = count ? min((long)*count, n_max) : n_max;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        for (int c = 0; c < 3; ++c) dst[3 * i + c] = src[3 * i + c] + sign * t[c];
}

int translate_dev_impl(float* dst, const float* src, const unsigned* count, long n_max, const float* t_dev, float sign,
                       cudaStream_t st) {
    if (n_max <= 0) return AFX_OK;
    translate_dev_kernel<<<grid_for(n_max, 256), 256, 0, st>>>(dst, src, count, n_max, t_dev, sign);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int translate_impl(float* pts, const unsigned* count, long n_max, const float* t, cudaStream_t st) {
    if (n_max <= 0) return AFX_OK;
    translate_kernel<<<blocks_for(n_max, 256), 256, 0, st>>>(pts, count, n_max, t[0], t[1], t[2]);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

}  // namespace afx

using namespace afx;

extern "C" {

int afx_marching_cubes_points(float* points, unsigned* count, long capacity, const float* tsdf, const float* weights,
                              const int dims[3], const float voxel_size[3], const float volume_size[3], float iso,
                              void* stream) {
    if (!points || !count || !tsdf || !weights || !dims || capacity < 0) return AFX_ERR_INVALID_ARGUMENT;
    return mc_fused_impl(tsdf, weights, kVoxF32, make_volume(dims, voxel_size, volume_size), iso, points, count, capacity,
                         nullptr, nullptr, 0, nullptr, nullptr, 0, as_stream(stream));
}

int afx_marching_cubes_mesh(float* vertices, unsigned* vertex_count, long vertex_capacity, int* faces,
                            unsigned* face_count, long face_capacity, const float* tsdf, const float* weights,
                            const int dims[3], const float voxel_size[3], const float volume_size[3], float iso,
                            void* stream) {
    if (!vertices || !vertex_count || !faces || !face_count || !tsdf || !weights || !dims)
        return AFX_ERR_INVALID_ARGUMENT;
    return mc_fused_impl(tsdf, weights, kVoxF32, make_volume(dims, voxel_size, volume_size), iso, nullptr, nullptr, 0, vertices,
                         vertex_count, vertex_capacity, faces, face_count, face_capacity, as_stream(stream));
}

size_t afx_sort_unique_points_workspace_size(long n_max) { return sort_unique_workspace_size(n_max); }

int afx_sort_unique_points(float* points, unsigned* count, long n_max, void* workspace, size_t workspace_bytes,
                           void* stream) {
    if (!points || !count || n_max < 0) return AFX_ERR_INVALID_ARGUMENT;
    return sort_unique_impl(points, count, n_max, workspace, workspace_bytes, as_stream(stream));
}

size_t afx_sort_unique_volume_points_workspace_size(long n_max, const int dims[3]) {
    if (!dims || dims[0] < 1) return 0;
    return sort_unique_volume_workspace_size(n_max < 1 ? 1 : n_max, dims[0] + 1);
}

int afx_sort_unique_volume_points(float* points, unsigned* count, long n_max, const int dims[3],
                                  const float voxel_size[3], const float volume_size[3], void* workspace,
                                  size_t workspace_bytes, void* stream) {
    if (!points || !count || n_max < 0 || !dims || !voxel_size || !volume_size || dims[0] < 1)
        return AFX_ERR_INVALID_ARGUMENT;
    return sort_unique_volume_impl(points, count, n_max, workspace, workspace_bytes,
                                   make_volume(dims, voxel_size, volume_size), as_stream(stream), nullptr);
}

int afx_extract_point_cloud(float* points, unsigned* count, long capacity, const float* tsdf, const float* weights,
                            const int dims[3], const float voxel_size[3], const float volume_size[3], float iso,
                            void* workspace, size_t workspace_bytes, void* stream) {
    if (!points || !count || !tsdf || !weights || !dims) return AFX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    AFX_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned), st));
    int rc = mc_fused_impl(tsdf, weights, kVoxF32, make_volume(dims, voxel_size, volume_size), iso, points, count, capacity,
                           nullptr, nullptr, 0, nullptr, nullptr, 0, st);
    if (rc) return rc;
    return sort_unique_impl(points, count, capacity, workspace, workspace_bytes, st);
}

int afx_translate(float* points, const unsigned* count, long n_max, const float t[3], void* stream) {
    if (!points || !t || n_max < 0) return AFX_ERR_INVALID_ARGUMENT;
    return translate_impl(points, count, n_max, t, as_stream(stream));
}

}  // extern "C"
