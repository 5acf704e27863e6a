// afx_integrate.cu -- TSDF integration: rigid projective integration and the non-rigid
// path (voxel -> node support, skinning weights, voxel warp, collision count, warped
// integration).
//
// The reference materialises per-voxel KNN index/distance/weight arrays and warped
// centres for the whole grid (~1.5 GB at 256^3, src/VolumeFusion.cu:252-260) and fills
// the KNN slots with atomics (first K to arrive, src/TSDFWarp.cu:61-67).  Here the
// active region is gathered brick by brick (8^3 voxels): each node lists the bricks
// its support cube touches, and one CTA per active brick selects, for each of its
// voxels, the K nearest supporting nodes (ties by node index), blends them, warps the
// voxel centre and counts collisions; a second pass integrates.  Only active voxels
// are touched.
#include <cstring>
#include <type_traits>

#include "afx_dqb.cuh"
#include "afx_store.cuh"
#include "afx_voxel.h"

namespace afx {

Volume make_volume(const int dims[3], const float voxel_size[3], const float volume_size[3]) {
    Volume v;
    for (int c = 0; c < 3; ++c) {
        v.dims[c] = dims[c];
        v.vs[c] = voxel_size[c];
        v.half[c] = volume_size[c] * 0.5f;
        v.inv[c] = (float)(1.0 / (double)voxel_size[c]);
    }
    return v;
}

// ------------------------------------------------------------------------------------
// Rigid integration (integrateTSDFFromFrameKernel, src/TSDFIntegration.cu:69-96)
//
// The volume is taken in blocks of 32 x 16 x 16 voxels (thinner ones in smaller volumes).  The pixels that a block projects to are bounded
// by its eight corner voxels (the projection of a box in front of the camera lies within theirs) and
// compared by the largest depth among them: a block that lies outside the image, sees no valid depth,
// or lies more than the truncation distance behind every one of them has no voxel to update, and most
// blocks are such.  The bounds have margins far above the rounding of a voxel's own projection, and
// every voxel of the other blocks is evaluated as before, so the volume is the same bit for bit.
// Threads own four consecutive voxels along x where rows allow it (one 16-byte access per array in
// FP32), else single ones, and touch the volume only where a voxel is updated.
// The fresh form (DeviceTsdf::initDefault followed by the integration, one pass that only writes): a
// freshly initialised voxel (-1, weight 0) that is updated becomes ((-1 * 0) + t * 1) / (0 + 1) = t
// with weight min(0 + 1, 15) = 1 -- exactly, since -0 + t = t and t / 1 = t -- and every other voxel
// stays (-1, 0).  8 B per voxel written instead of 8 written + 16 read and written.
// Bound: the latency of looking at a block (two divisions, a load of its pixels, one barrier), or HBM writes
// (fresh).  One 640 x 576 frame of an object: 512^3 FP32, 1,054 of 16,384 blocks evaluated, 69 us (a thread
// for every four voxels: 290 us; looking at 2 x 2 x 2 blocks first, and then integrating those that
// remain one after the other: 134 us); fresh 400^3 83 us, 6.2 TB/s written (164 us).
// ------------------------------------------------------------------------------------

struct RigidArgs {
    Volume vol;
    float R[9];
    float t[3];
    const float* t_dev;  // when set, the translation is read from device memory
    Intrinsics K;
    float delta;
    int W, H;
    unsigned char* occ;  // brick occupancy, or null
    int nbx, nby;        // bricks per axis (x, y)
};

// Marks the 8^3 brick of voxel (x, y, z) as holding a voxel with a weight (many threads may store 1).
AFX_D void mark_brick(unsigned char* occ, int nbx, int nby, int x, int y, int z) {
    if (occ) occ[((long)(z >> 3) * nby + (y >> 3)) * nbx + (x >> 3)] = 1;
}

// Blocks of kBlkZ slices.  Below kMidVoxels half as deep, since there are few for the SMs (256^3: an object 29 -> 27.5 us,
// every voxel updated 70 -> 64.5; rows of 255 voxels 84 -> 71; at 320^3 the looking costs more than that saves, an
// object 37 -> 41.5).  Below kThinVoxels a quarter as deep and without looking, for which there is little to leave
// out (an object and every voxel updated, from kBlkZ slices to these: 64^3 21 -> 11 us both, 128^3 21 -> 11 and 23 -> 13,
// 192^3 23 -> 21 and 31 -> 29; at 256^3 29 -> 42 and 70 -> 62).
constexpr int kBlkX = 32, kBlkY = 16, kBlkZ = 16, kMidZ = 8, kThinZ = 4;  // whole 8^3 bricks, but for kThinZ
constexpr long kThinVoxels = 10000000, kMidVoxels = 20000000;
constexpr int kBlkThreads = 256;
// CTAs per SM that the registers of each form are held to.
__host__ __device__ constexpr int blk_ctas(bool vec, int depth) { return depth == kBlkZ ? 5 : depth == kThinZ && !vec ? 8 : 6; }
constexpr int kBlkPixels = 4096;        // a block that spans more pixels is evaluated without looking at them

AFX_D void rigid_point(const RigidArgs& a, float t0, float t1, float t2, int x, int y, int z, float* q) {
    float p[3];
    voxel_to_world(x, y, z, a.vol.vs, a.vol.half, p);
    mat3_vec3(a.R, p, q);
    q[0] = q[0] + t0;
    q[1] = q[1] + t1;
    q[2] = q[2] + t2;
}

AFX_D float warp_min8(float v) {  // over lanes 8k .. 8k + 7
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// What the corners of a block say: nothing in it can be updated, nothing is known, or it depends on
// the depths in a box of pixels.  Evaluated by whole warps, the same answer in every lane.
struct BoxView {
    int state;  // 0: nothing to update, 1: not known, 2: look at the pixels
    int px0, py0, w, h;
    float behind;  // a box whose pixels' largest valid depth is below this has nothing to update
};

template <int kZ>
AFX_D BoxView box_view(const RigidArgs& a, float t0, float t1, float t2, int x0, int y0, int z0) {
    const int lane = threadIdx.x & 31;
    const int* D = a.vol.dims;
    float q[3];
    rigid_point(a, t0, t1, t2, (lane & 1) ? min(x0 + kBlkX, D[0]) - 1 : x0, (lane & 2) ? min(y0 + kBlkY, D[1]) - 1 : y0,
                (lane & 4) ? min(z0 + kZ, D[2]) - 1 : z0, q);
    const float zmin = warp_min8(q[2]), zmax = -warp_min8(-q[2]);
    const float u = a.K.fx * q[0] / q[2] + a.K.cx, v = a.K.fy * q[1] / q[2] + a.K.cy;
    const float umin = warp_min8(u), umax = -warp_min8(-u), vmin = warp_min8(v), vmax = -warp_min8(-v);
    const float zm = 1e-5f * (fabsf(zmin) + fabsf(zmax)) + 1e-6f;  // margin
    BoxView b{1, 0, 0, 0, 0, 0.f};
    if (!__all_sync(0xffffffffu, fabsf(q[0]) < 1e30f && fabsf(q[1]) < 1e30f && fabsf(q[2]) < 1e30f)) return b;
    if (zmax < 1e-4f - zm) {  // behind the camera
        b.state = 0;
        return b;
    }
    if (!(zmin > 1e-3f + zm)) return b;  // around the camera plane: no bound
    const float um = 2.f + 1e-4f * fmaxf(fabsf(umin), fabsf(umax)), vm = 2.f + 1e-4f * fmaxf(fabsf(vmin), fabsf(vmax));
    if (!(fabsf(umin) < 1e9f && fabsf(umax) < 1e9f && fabsf(vmin) < 1e9f && fabsf(vmax) < 1e9f)) return b;
    b.px0 = max(0, (int)floorf(umin - um));
    b.py0 = max(0, (int)floorf(vmin - vm));
    b.w = min(a.W - 1, (int)ceilf(umax + um)) - b.px0 + 1;
    b.h = min(a.H - 1, (int)ceilf(vmax + vm)) - b.py0 + 1;
    if (b.w <= 0 || b.h <= 0) {
        b.state = 0;
        return b;
    }
    if ((long)b.w * b.h > kBlkPixels) return b;
    b.state = 2;
    // sdf = z - depth > delta for every voxel, with a margin for the roundings: below even for a depth that
    // fills the left side's margin
    b.behind = (zmin - (zm + a.delta)) / (1.f + 2e-5f) - 1e-5f * fabsf(a.delta);
    return b;
}

// A valid depth as bits: positive floats compare as integers; 0: none; not a number counts as infinitely far, since it
// updates.
AFX_D unsigned depth_key(float d) { return d != d ? 0x7f800000u : (isinf(d) || d < 1.e-4f) ? 0u : __float_as_uint(d); }

// Largest of the box's pixels over this thread's share of them.
AFX_D unsigned box_depth(const BoxView& b, const float* __restrict__ depth, int W, int first, int step) {
    const int n = b.w * b.h;
    const float inv = 1.0f / (float)b.w;  // (i + 1/2) / w is at least 1/2w from an integer: exact for these n
    unsigned best = 0u;
#pragma unroll 8
    for (int i = first; i < n; i += step) {
        const int row = (int)(((float)i + 0.5f) * inv);
        const float d = __ldg(depth + (long)(b.py0 + row) * W + b.px0 + (i - row * b.w));
        best = max(best, depth_key(d));
    }
    return __reduce_max_sync(0xffffffffu, best);
}

// No valid pixel, or all of them in front by more than the truncation distance (a comparison with not a
// number says no).
AFX_D bool box_empty(const BoxView& b, unsigned best) { return best == 0u || __uint_as_float(best) < b.behind; }

// The voxels of the block at (x0, y0, z0), by the whole CTA.  kVec: rows of a multiple of four voxels,
// 16-byte (FP16: 8-byte) aligned.  kFresh: every voxel is written; `seen`: whether any can be updated.
// Returns the bricks of the block in which this thread left a positive value (kFresh), a bit each.  kZ: depth of the block.
template <class TT, class WT, bool kVec, bool kFresh, int kZ>
AFX_D unsigned integrate_block(TT* __restrict__ tsdf, WT* __restrict__ weights, const float* __restrict__ depth,
                               const RigidArgs& a, float t0, float t1, float t2, int x0, int y0, int z0, bool seen) {
    constexpr int N = kVec ? 4 : 1;                           // voxels per access
    constexpr int kTx = kBlkX / N, kTy = kVec ? kBlkY : 8;    // threads along x and y
    constexpr int kTz = kBlkThreads / (kTx * kTy);
    const int X = a.vol.dims[0], Y = a.vol.dims[1], Z = a.vol.dims[2];
    const int tx = threadIdx.x % kTx, ty = (threadIdx.x / kTx) % kTy, tz = threadIdx.x / (kTx * kTy);
    const int x = x0 + tx * N;
    unsigned mine = 0u;
    if (x >= X) return mine;
    for (int y = y0 + ty; y < min(y0 + kBlkY, Y); y += kTy)
        for (int z = z0 + tz; z < min(z0 + kZ, Z); z += kTz) {
            float tn[N];
            unsigned upd = 0;
            if (!kFresh || seen) {
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    float q[3];
                    rigid_point(a, t0, t1, t2, x + i, y, z, q);
                    if (tsdf_update_value(q, depth, a.W, a.H, a.delta, a.K, &tn[i])) upd |= 1u << i;
                }
            }
            const long base = ((long)z * Y + y) * X + x;
            float tv[N], wv[N];
            if (kFresh) {
                // (the blend written out as its result: the division by 0 + 1 and the products by 0 and 1
                // change nothing)
                bool positive = false;
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    positive |= ((upd >> i) & 1u) && tn[i] > 0.f;
                    tv[i] = (upd >> i) & 1u ? tn[i] : -1.f;
                    wv[i] = (upd >> i) & 1u ? 1.f : 0.f;
                }
                if (positive) mine |= 1u << (((x - x0) >> 3) + 4 * ((y - y0) >> 3) + 8 * ((z - z0) >> 3));
            } else {
                if (!upd) continue;
                mark_brick(a.occ, a.nbx, a.nby, x, y, z);  // the four voxels share a brick
                if constexpr (kVec) {
                    vox_get4(tsdf, weights, base, tv, wv);
                } else {
                    tv[0] = vox_get_t(tsdf, base);
                    wv[0] = vox_get_w(weights, base);
                }
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if (upd & (1u << i)) tsdf_blend(tv[i], wv[i], tn[i]);
            }
            if constexpr (kVec) vox_put4(tsdf, weights, base, tv, wv);
            else vox_put(tsdf, weights, base, tv[0], wv[0]);
        }
    return mine;
}

// Whether any voxel of the CTA's block can be updated (the same answer in every thread).
template <int kZ>
AFX_D bool block_seen(const RigidArgs& a, const float* __restrict__ depth, float t0, float t1, float t2, int x0, int y0,
                      int z0) {
    __shared__ unsigned wmax[kBlkThreads / 32];
    const int lane = threadIdx.x & 31;
    const BoxView b = box_view<kZ>(a, t0, t1, t2, x0, y0, z0);
    if (b.state != 2) return b.state != 0;
    const int n = b.w * b.h;
    if (kZ == kMidZ && n > 4 * kBlkThreads) {  // one pixel a thread first: a block that is seen mostly is by one of these
        const int i = (int)((unsigned)threadIdx.x * (unsigned)n / kBlkThreads), row = i / b.w;
        const float d = __ldg(depth + (long)(b.py0 + row) * a.W + b.px0 + (i - row * b.w));
        if (__syncthreads_or(!box_empty(b, depth_key(d)))) return true;
    }
    const unsigned m = box_depth(b, depth, a.W, threadIdx.x, kBlkThreads);
    if (lane == 0) wmax[threadIdx.x >> 5] = m;
    __syncthreads();
    return !box_empty(b, __reduce_max_sync(0xffffffffu, lane < kBlkThreads / 32 ? wmax[lane] : 0u));
}

// kZ: depth of the blocks; kLook: leave out those without a voxel to update.
template <class TT, class WT, bool kVec, int kZ, bool kLook>
__global__ void __launch_bounds__(kBlkThreads, blk_ctas(kVec, kZ)) integrate_rigid_kernel(TT* __restrict__ tsdf,
                                                                                         WT* __restrict__ weights,
                                                                                         const float* __restrict__ depth,
                                                                                         RigidArgs a) {
    const int x0 = blockIdx.x * kBlkX, y0 = blockIdx.y * kBlkY, z0 = blockIdx.z * kZ;
    const float t0 = a.t_dev ? a.t_dev[0] : a.t[0], t1 = a.t_dev ? a.t_dev[1] : a.t[1],
                t2 = a.t_dev ? a.t_dev[2] : a.t[2];
    if (kLook && !block_seen<kZ>(a, depth, t0, t1, t2, x0, y0, z0)) return;
    integrate_block<TT, WT, kVec, false, kZ>(tsdf, weights, depth, a, t0, t1, t2, x0, y0, z0, true);
}

// a.occ (optional; blocks of whole bricks): every byte of it is written, whether the brick has a weighted voxel with a
// positive value.
template <bool kVec, int kZ, bool kLook>
__global__ void __launch_bounds__(kBlkThreads, blk_ctas(kVec, kZ)) integrate_fresh_kernel(float* __restrict__ tsdf,
                                                                                         float* __restrict__ weights,
                                                                                         const float* __restrict__ depth,
                                                                                         RigidArgs a) {
    __shared__ unsigned bricks;  // bit per 8^3 brick of the block with a positive value
    const int X = a.vol.dims[0], Y = a.vol.dims[1], Z = a.vol.dims[2];
    const int x0 = blockIdx.x * kBlkX, y0 = blockIdx.y * kBlkY, z0 = blockIdx.z * kZ;
    const bool seen = !kLook || block_seen<kZ>(a, depth, a.t[0], a.t[1], a.t[2], x0, y0, z0);
    const unsigned mine = __reduce_or_sync(0xffffffffu, integrate_block<float, float, kVec, true, kZ>(
                                                            tsdf, weights, depth, a, a.t[0], a.t[1], a.t[2], x0, y0, z0, seen));
    if (kZ % 8 != 0 || !a.occ) return;
    if (threadIdx.x == 0) bricks = 0u;
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && mine) atomicOr(&bricks, mine);
    __syncthreads();
    const int k = threadIdx.x, bx = (x0 >> 3) + (k & 3), by = (y0 >> 3) + ((k >> 2) & 1), bz = (z0 >> 3) + (k >> 3);
    if (k < kZ && bx * 8 < X && by * 8 < Y && bz * 8 < Z)  // 4 x 2 x kZ / 8 of them
        a.occ[((long)bz * a.nby + by) * a.nbx + bx] = (unsigned char)((bricks >> k) & 1u);
}

static RigidArgs rigid_args(const Volume& vol, const float* R, const float* t, const float* t_dev, const float* K,
                            float delta, int W, int H, unsigned char* occ) {
    RigidArgs a;
    a.vol = vol;
    a.occ = occ;
    const BrickGrid bg = make_bricks(vol);
    a.nbx = bg.nb[0];
    a.nby = bg.nb[1];
    for (int i = 0; i < 9; ++i) a.R[i] = R[i];
    for (int i = 0; i < 3; ++i) a.t[i] = t ? t[i] : 0.f;
    a.t_dev = t_dev;
    a.K = make_intrinsics(K);
    a.delta = delta;
    a.W = W;
    a.H = H;
    return a;
}

static dim3 rigid_grid(const Volume& vol, int depth) {
    return dim3((unsigned)((vol.dims[0] + kBlkX - 1) / kBlkX), (unsigned)((vol.dims[1] + kBlkY - 1) / kBlkY),
                (unsigned)((vol.dims[2] + depth - 1) / depth));
}

static long voxels_of(const Volume& vol) { return (long)vol.dims[0] * vol.dims[1] * vol.dims[2]; }

// Whether rows of four voxels are aligned vectors (`elem` bytes per voxel and array).
static bool rows_vectorize(const void* tsdf, const void* weights, const Volume& vol, size_t elem) {
    return vol.dims[0] % 4 == 0 &&
           ((reinterpret_cast<uintptr_t>(tsdf) | reinterpret_cast<uintptr_t>(weights)) & (4 * elem - 1)) == 0;
}

int integrate_fresh_impl(float* tsdf, float* weights, const float* depth, int W, int H, float delta, const Volume& vol,
                         const float* R, const float* t, const float* K, cudaStream_t st, unsigned char* occ) {
    const RigidArgs a = rigid_args(vol, R, t, nullptr, K, delta, W, H, occ);
    const bool vec = rows_vectorize(tsdf, weights, vol, sizeof(float));
    auto launch = [&](auto depth_of, auto look_of) {
        constexpr int kZ = decltype(depth_of)::value;
        constexpr bool kLook = decltype(look_of)::value;
        if (vec) integrate_fresh_kernel<true, kZ, kLook><<<rigid_grid(vol, kZ), kBlkThreads, 0, st>>>(tsdf, weights, depth, a);
        else integrate_fresh_kernel<false, kZ, kLook><<<rigid_grid(vol, kZ), kBlkThreads, 0, st>>>(tsdf, weights, depth, a);
    };
    // (every voxel is written, so only the thin blocks pay here; whole bricks where their marks are asked for)
    if (voxels_of(vol) >= kThinVoxels) launch(std::integral_constant<int, kBlkZ>(), std::true_type());
    else if (occ) launch(std::integral_constant<int, kMidZ>(), std::false_type());
    else launch(std::integral_constant<int, kThinZ>(), std::false_type());
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int integrate_rigid_impl(void* tsdf, void* weights, int fmt, const float* depth, int W, int H, float delta,
                         const Volume& vol, const float* R, const float* t, const float* K, cudaStream_t st,
                         const float* t_dev, unsigned char* occ) {
    const RigidArgs a = rigid_args(vol, R, t, t_dev, K, delta, W, H, occ);
    const bool vec = rows_vectorize(tsdf, weights, vol, vox_bytes(fmt));
    vox_dispatch(fmt, tsdf, weights, [&](auto* tp, auto* wp) {
        using TT = std::remove_pointer_t<decltype(tp)>;
        using WT = std::remove_pointer_t<decltype(wp)>;
        auto launch = [&](auto depth_of, auto look_of) {
            constexpr int kZ = decltype(depth_of)::value;
            constexpr bool kLook = decltype(look_of)::value;
            const dim3 grid = rigid_grid(vol, kZ);
            if (vec) integrate_rigid_kernel<TT, WT, true, kZ, kLook><<<grid, kBlkThreads, 0, st>>>(tp, wp, depth, a);
            else integrate_rigid_kernel<TT, WT, false, kZ, kLook><<<grid, kBlkThreads, 0, st>>>(tp, wp, depth, a);
        };
        if (voxels_of(vol) >= kMidVoxels) launch(std::integral_constant<int, kBlkZ>(), std::true_type());
        else if (voxels_of(vol) >= kThinVoxels) launch(std::integral_constant<int, kMidZ>(), std::true_type());
        else launch(std::integral_constant<int, kThinZ>(), std::false_type());
        return 0;
    });
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// ------------------------------------------------------------------------------------
// Brick-sparse voxel support (replaces tsdfKNNGraph, src/TSDFWarp.cu:23-68)
// ------------------------------------------------------------------------------------

// Node support cube: node voxel (worldToVoxel of the translated node), minus (per-1)/2,
// plus [0, per) per axis (src/TSDFWarp.cu:40-50), clipped to the volume.
AFX_D bool node_cube(const float* node_t, const Volume& vol, const int* per, NodeCube* c) {
    int nv[3];
    world_to_voxel(node_t, vol.inv, vol.half, nv);
    bool empty = false;
    for (int a = 0; a < 3; ++a) {
        int lo = nv[a] - (per[a] - 1) / 2;
        int hi = lo + per[a] - 1;
        c->lo[a] = max(lo, 0);
        c->hi[a] = min(hi, vol.dims[a] - 1);
        if (c->lo[a] > c->hi[a]) empty = true;
    }
    return !empty;
}

__global__ void brick_count_kernel(SupportArgs a) {
    const int n = min(*a.n_nodes, a.n_max);
    AFX_GRID_STRIDE(j, n) {
    NodeCube c;
    if (!node_cube(a.nodes + 3 * j, a.vol, a.per, &c)) continue;
    for (int bz = c.lo[2] / kBrick; bz <= c.hi[2] / kBrick; ++bz)
        for (int by = c.lo[1] / kBrick; by <= c.hi[1] / kBrick; ++by)
            for (int bx = c.lo[0] / kBrick; bx <= c.hi[0] / kBrick; ++bx)
                atomicAdd(a.brick_count + ((long)bz * a.bg.nb[1] + by) * a.bg.nb[0] + bx, 1u);
    }
}

__global__ void brick_fill_kernel(SupportArgs a) {
    const int n = min(*a.n_nodes, a.n_max);
    AFX_GRID_STRIDE(j, n) {
    NodeCube c;
    if (!node_cube(a.nodes + 3 * j, a.vol, a.per, &c)) continue;
    for (int bz = c.lo[2] / kBrick; bz <= c.hi[2] / kBrick; ++bz)
        for (int by = c.lo[1] / kBrick; by <= c.hi[1] / kBrick; ++by)
            for (int bx = c.lo[0] / kBrick; bx <= c.hi[0] / kBrick; ++bx) {
                long b = ((long)bz * a.bg.nb[1] + by) * a.bg.nb[0] + bx;
                unsigned pos = a.brick_offset[b] + atomicAdd(a.brick_cursor + b, 1u);
                if (pos < a.pair_capacity) a.brick_nodes[pos] = (unsigned)j;
                else atomicOr(a.error, ERRF_CAPACITY);
            }
    }
}

__global__ void brick_active_kernel(const unsigned* brick_count, long nb, unsigned* active, unsigned* n_active) {
    const long b = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const bool on = b < nb && brick_count[b] > 0;  // every lane takes part in the ballot
    unsigned m = __ballot_sync(0xffffffffu, on);
    unsigned base = 0;
    int lane = threadIdx.x & 31;
    if (lane == 0 && m) base = atomicAdd(n_active, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (on) active[base + __popc(m & ((1u << lane) - 1))] = (unsigned)b;
}

template <class Id>
AFX_D void topk_insert(float* kd, Id* ki, int& cnt, int cap, float d, Id idx) {
    if (cnt == cap && !(d < kd[cap - 1] || (d == kd[cap - 1] && idx < ki[cap - 1]))) return;
    int i = (cnt < cap) ? cnt++ : cap - 1;
    while (i > 0 && (d < kd[i - 1] || (d == kd[i - 1] && idx < ki[i - 1]))) {
        kd[i] = kd[i - 1];
        ki[i] = ki[i - 1];
        --i;
    }
    kd[i] = d;
    ki[i] = idx;
}

AFX_D void coll_add(unsigned* w, unsigned epoch) {
    unsigned old = *w, assumed;
    do {
        assumed = old;
        unsigned nw = ((assumed >> 8) == epoch) ? (((assumed & 255u) < 255u) ? assumed + 1u : assumed) : ((epoch << 8) | 1u);
        old = atomicCAS(w, assumed, nw);
    } while (old != assumed);
}

AFX_D int coll_get(const unsigned* w, unsigned epoch) {
    unsigned v = *w;
    return ((v >> 8) == epoch) ? (int)(v & 255u) : 0;
}

// The K nearest supporters of every voxel of the active bricks, their weights, and the voxel's centre moved by
// them.  The brick's candidate nodes are staged in shared memory with their transforms, so that what a voxel does
// after its search waits for no further gather, and a voxel is inside a node's cube where three bits of the
// candidate's word say so.  The list is kept sorted in registers (indexed ones went to local memory).
// Bound: the chain active brick -> candidates -> nodes in front of each brick.  200^3 voxels, 600 nodes, dense lists: 24.4 ->
// 14.6 us; a frame of the 256^3 sequence 23 -> 17 us, of the 512^3 sequence 57 -> 40 us.
// Id: a node and its place in the brick's list in one number, 64 bits for graphs whose nodes do not fit in 24.
template <int K, class Id>
__global__ void __launch_bounds__(kBrickVox) brick_warp_kernel(WarpArgs a) {
    __shared__ float4 s_node[kMaxBrickNodes];      // position, radius
    __shared__ float4 s_T[kMaxBrickNodes * 4];     // columns of the transform
    __shared__ unsigned s_cube[kMaxBrickNodes];    // x, y, z of the brick inside the node's cube, eight bits each
    __shared__ Id s_id[kMaxBrickNodes];            // node << 8 | place here
    static_assert(kMaxBrickNodes <= 256, "a place fits in eight bits");
    const unsigned n_active = *a.n_active;
    const int lx = threadIdx.x % kBrick, ly = (threadIdx.x / kBrick) % kBrick, lz = threadIdx.x / (kBrick * kBrick);
    const unsigned here = 1u << lx | 1u << (8 + ly) | 1u << (16 + lz);
    for (unsigned slot = blockIdx.x; slot < n_active; slot += gridDim.x) {
    const unsigned b = a.active[slot];
    const unsigned off = a.brick_offset[b];
    const int nc = min((int)a.brick_count[b], kMaxBrickNodes);
    const int bx = b % a.bg.nb[0], by = (b / a.bg.nb[0]) % a.bg.nb[1], bz = b / ((unsigned)a.bg.nb[0] * a.bg.nb[1]);
    __syncthreads();  // the previous brick's staged nodes are no longer read
    if (threadIdx.x == 0 && a.brick_count[b] > kMaxBrickNodes) atomicOr(a.error, ERRF_CAPACITY);
    bool odd = false;  // a position that is not a number
    for (int i = threadIdx.x; i < nc; i += blockDim.x) {
        const unsigned j = a.brick_nodes[off + i];
        const float p[3] = {a.nodes_t[3 * (long)j], a.nodes_t[3 * (long)j + 1], a.nodes_t[3 * (long)j + 2]};
        s_id[i] = (Id)j << 8 | (unsigned)i;
        s_node[i] = make_float4(p[0], p[1], p[2], a.radii[j]);
        odd |= p[0] != p[0] || p[1] != p[1] || p[2] != p[2];
        NodeCube c;
        node_cube(p, a.vol, a.per, &c);
        const int base[3] = {bx * kBrick, by * kBrick, bz * kBrick};
        unsigned cube = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int lo = max(c.lo[q] - base[q], 0), hi = min(c.hi[q] - base[q], kBrick - 1);
            if (lo <= hi) cube |= ((2u << hi) - (1u << lo)) << (8 * q);
        }
        s_cube[i] = cube;
    }
    if (a.out)
        for (int t = threadIdx.x; t < nc * 4; t += blockDim.x)
            s_T[t] = reinterpret_cast<const float4*>(a.transforms)[4 * (long)a.brick_nodes[off + (t >> 2)] + (t & 3)];
    odd = __syncthreads_or(odd);
    [&] {
    const int x = bx * kBrick + lx, y = by * kBrick + ly, z = bz * kBrick + lz;
    const long local = (long)slot * kBrickVox + threadIdx.x;
    const int X = a.vol.dims[0], Y = a.vol.dims[1], Z = a.vol.dims[2];
    const bool inside = x < X && y < Y && z < Z;
    constexpr Id kEmpty = ~(Id)0;
    float kd[K];
    Id ki[K];  // as s_id: in node order
#pragma unroll
    for (int s = 0; s < K; ++s) {
        kd[s] = INFINITY;
        ki[s] = kEmpty;
    }
    float p[3];
    voxel_to_world(x, y, z, a.vol.vs, a.vol.half, p);
    if (inside && !odd) {
        for (int i = 0; i < nc; ++i) {
            if ((s_cube[i] & here) != here) continue;
            const float4 v = s_node[i];
            const float d3[3] = {p[0] - v.x, p[1] - v.y, p[2] - v.z};
            const float d = norm3(d3);
            if (d > v.w * 2.0f) continue;
            const Id id = s_id[i];
            if (!(d < kd[K - 1] || (d == kd[K - 1] && id < ki[K - 1]))) continue;
            kd[K - 1] = d;
            ki[K - 1] = id;
#pragma unroll
            for (int s = K - 1; s > 0; --s) {
                const bool up = kd[s] < kd[s - 1] || (kd[s] == kd[s - 1] && ki[s] < ki[s - 1]);
                const float ds = kd[s], dt = kd[s - 1];
                const Id is = ki[s], it = ki[s - 1];
                kd[s] = up ? dt : ds;
                kd[s - 1] = up ? ds : dt;
                ki[s] = up ? it : is;
                ki[s - 1] = up ? is : it;
            }
        }
    } else if (inside) {  // distances that are not numbers keep the place they were put at
        float ld[K];
        Id li[K];
        int n = 0;
        for (int i = 0; i < nc; ++i) {
            if ((s_cube[i] & here) != here) continue;
            const float4 v = s_node[i];
            const float d3[3] = {p[0] - v.x, p[1] - v.y, p[2] - v.z};
            const float d = norm3(d3);
            if (d > v.w * 2.0f) continue;
            topk_insert(ld, li, n, K < a.k ? K : a.k, d, s_id[i]);
        }
        for (int s = 0; s < n; ++s) {
            kd[s] = ld[s];
            ki[s] = li[s];
        }
    }
    int cnt = 0;
#pragma unroll
    for (int s = 0; s < K; ++s) cnt += s < a.k && ki[s] != kEmpty;
    if (a.dense_count && inside) {
        const long v = ((long)z * Y + y) * X + x;
        a.dense_count[v] = cnt;
#pragma unroll
        for (int s = 0; s < K; ++s) {
            if (s >= a.k) break;
            a.dense_idx[v * a.k + s] = s < cnt ? (uint32_t)(ki[s] >> 8) : AFX_INVALID_INDEX;
            a.dense_dist[v * a.k + s] = s < cnt ? kd[s] : 3.402823466e+38f;
        }
    }
    if (!a.out) return;
    a.out_count[local] = (unsigned char)cnt;
    if (cnt == 0) return;
    // weights (computeTsdfWarpWeightsKernel, src/TSDFWarp.cu:88-116: no cut-off)
    float w[K];
    float sum = 0.f;
#pragma unroll
    for (int s = 0; s < K; ++s) {
        w[s] = 0.f;
        if (s >= cnt) continue;
        const float r = s_node[(unsigned)ki[s] & 0xffu].w, d = kd[s];
        w[s] = afx_expf(-(d * d) / (2.0f * (r * r)));
        sum = sum + w[s];
    }
    bool zero = true;
#pragma unroll
    for (int s = 0; s < K; ++s) {
        if (s >= cnt) continue;
        if (sum != 0.f) w[s] = w[s] / sum;
        if (!(fabsf(w[s]) <= 1e-5f)) zero = false;
    }
    // voxel centre in camera space (generateTsdfVertices + translate, src/VolumeFusion.cu:718-723)
    const float cen[3] = {a.centroid_dev[0], a.centroid_dev[1], a.centroid_dev[2]};
    float c[3] = {p[0] + cen[0], p[1] + cen[1], p[2] + cen[2]};
    float q[3] = {c[0], c[1], c[2]};
    if (!zero && a.blend == AFX_BLEND_DQB) {  // dual-quaternion blend (afx_dqb.cuh)
        uint32_t kidx[K];
        for (int s = 0; s < cnt; ++s) kidx[s] = (uint32_t)(ki[s] >> 8);
        dq_blend_point(a.transforms, kidx, w, cnt, AFX_INVALID_INDEX, c, q);
    } else if (!zero) {  // warpTsdfKernel (src/TSDFWarp.cu:158-190)
        q[0] = q[1] = q[2] = 0.f;
#pragma unroll
        for (int s = 0; s < K; ++s) {
            if (s >= cnt) continue;
            const float4* T = s_T + 4 * ((unsigned)ki[s] & 0xffu);
            const float4 t0 = T[0], t1 = T[1], t2 = T[2], t3 = T[3];
            const float M[16] = {t0.x, t0.y, t0.z, 0.f, t1.x, t1.y, t1.z, 0.f, t2.x, t2.y, t2.z, 0.f, t3.x, t3.y, t3.z, 0.f};
            float o[3];
            mat4_point(M, c, o);
            q[0] = q[0] + w[s] * o[0];
            q[1] = q[1] + w[s] * o[1];
            q[2] = q[2] + w[s] * o[2];
        }
    }
    // target voxel (countCollisionsPerVoxelKernel, src/TSDFIntegration.cu:272-282)
    float dq[3] = {q[0] - cen[0], q[1] - cen[1], q[2] - cen[2]};
    float o[3];
    mat3_vec3(a.Rinv, dq, o);
    int tv[3];
    world_to_voxel(o, a.vol.inv, a.vol.half, tv);
    int target = -1;
    if (tv[0] >= 0 && tv[1] >= 0 && tv[2] >= 0 && tv[0] < X && tv[1] < Y && tv[2] < Z) {
        target = (int)(((long)tv[2] * Y + tv[1]) * X + tv[0]);
        coll_add(a.coll + target, *a.epoch_dev);
    }
    WarpedVoxel wv;
    wv.p[0] = q[0];
    wv.p[1] = q[1];
    wv.p[2] = q[2];
    wv.target = target;
    a.out[local] = wv;
    }();
    }
}

// integrateWarpedTSDFFromFrameKernel (src/TSDFIntegration.cu:173-226) over the active bricks
template <class TT, class WT>
__global__ void __launch_bounds__(kBrickVox) brick_integrate_kernel(WarpedIntegrateArgs a) {
    TT* __restrict__ tsdf = static_cast<TT*>(a.tsdf);
    WT* __restrict__ weights = static_cast<WT*>(a.weights);
    const unsigned n_active = *a.n_active;
    for (unsigned slot = blockIdx.x; slot < n_active; slot += gridDim.x) [&] {
    const long local = (long)slot * kBrickVox + threadIdx.x;
    if (a.in_count[local] == 0) return;
    const WarpedVoxel wv = a.in[local];
    if (wv.target < 0) return;
    if (coll_get(a.coll + wv.target, *a.epoch_dev) > 1) return;
    float tn;
    if (!tsdf_update_value(wv.p, a.depth, a.W, a.H, a.delta, a.K, &tn)) return;
    const unsigned b = a.active[slot];
    const int bx = b % a.bg.nb[0], by = (b / a.bg.nb[0]) % a.bg.nb[1], bz = b / ((unsigned)a.bg.nb[0] * a.bg.nb[1]);
    const int x = bx * kBrick + threadIdx.x % kBrick, y = by * kBrick + (threadIdx.x / kBrick) % kBrick,
              z = bz * kBrick + threadIdx.x / (kBrick * kBrick);
    const long v = ((long)z * a.vol.dims[1] + y) * a.vol.dims[0] + x;
    float t = vox_get_t(tsdf, v), w = vox_get_w(weights, v);
    tsdf_blend(t, w, tn);
    vox_put(tsdf, weights, v, t, w);
    if (a.occ) a.occ[b] = 1;
    }();
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Bricks a node's support cube can touch: per axis at most ceil((per - 1) / 8) + 1.
static long pairs_per_node(const int* per) {
    long p = 1;
    for (int c = 0; c < 3; ++c) p *= (per[c] - 1 + kBrick - 1) / kBrick + 1;
    return p;
}

size_t support_workspace_size(const Volume& vol, int n_nodes_max, const int* per) {
    BrickGrid bg = make_bricks(vol);
    size_t scan = scan_workspace_size(bg.n);
    long pairs = (long)n_nodes_max * pairs_per_node(per) + 1024;
    return align256(bg.n * 4) * 3 + align256((bg.n + 1) * 4) + align256(pairs * 4) + align256(bg.n * 4) + 256 +
           align256(scan) + 1024;
}

bool carve_support(void* ws, size_t bytes, const Volume& vol, int n_nodes_max, const int* per, SupportWorkspace* s) {
    if (bytes < support_workspace_size(vol, n_nodes_max, per) || !ws) return false;
    BrickGrid bg = make_bricks(vol);
    char* p = static_cast<char*>(ws);
    auto take = [&](size_t n) {
        char* r = p;
        p += align256(n);
        return r;
    };
    s->brick_count = (unsigned*)take(bg.n * 4);
    s->brick_cursor = (unsigned*)take(bg.n * 4);
    s->brick_offset = (unsigned*)take((bg.n + 1) * 4);
    s->pair_capacity = (long)n_nodes_max * pairs_per_node(per) + 1024;
    s->brick_nodes = (unsigned*)take(s->pair_capacity * 4);
    s->active = (unsigned*)take(bg.n * 4);
    s->n_active = (unsigned*)take(256);
    size_t scan = scan_workspace_size(bg.n);
    s->scan_tmp_bytes = scan;
    s->scan_tmp = take(scan);
    return true;
}

// Builds the brick -> node candidate lists and the active brick list.
int build_support(const SupportWorkspace& s, const Volume& vol, const int* per, const float* nodes_t,
                  const float* radii, const int* n_nodes, int n_max, int* error, cudaStream_t st) {
    BrickGrid bg = make_bricks(vol);
    AFX_CUDA(cudaMemsetAsync(s.brick_count, 0, bg.n * 4, st));
    AFX_CUDA(cudaMemsetAsync(s.brick_cursor, 0, bg.n * 4, st));
    AFX_CUDA(cudaMemsetAsync(s.n_active, 0, 4, st));
    SupportArgs a;
    a.vol = vol;
    a.bg = bg;
    for (int c = 0; c < 3; ++c) a.per[c] = per[c];
    a.nodes = nodes_t;
    a.radii = radii;
    a.n_nodes = n_nodes;
    a.n_max = n_max;
    a.brick_count = s.brick_count;
    a.brick_offset = s.brick_offset;
    a.brick_cursor = s.brick_cursor;
    a.brick_nodes = s.brick_nodes;
    a.pair_capacity = s.pair_capacity;
    a.error = error;
    if (n_max > 0) {
        brick_count_kernel<<<grid_for(n_max, 128), 128, 0, st>>>(a);
        AFX_LAUNCH_CHECK();
    }
    int rc = scan_exclusive(s.brick_count, s.brick_offset, bg.n, nullptr, s.scan_tmp, st);
    if (rc) return rc;
    if (n_max > 0) {
        brick_fill_kernel<<<grid_for(n_max, 128), 128, 0, st>>>(a);
        AFX_LAUNCH_CHECK();
    }
    brick_active_kernel<<<blocks_for(bg.n, 256), 256, 0, st>>>(s.brick_count, bg.n, s.active, s.n_active);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// Block-stride grid over the active bricks (their number is on the device).
static unsigned brick_grid(long max_active) { return (unsigned)(max_active < 608 ? max_active : 608); }

int launch_brick_warp(const WarpArgs& a, long max_active, cudaStream_t st) {
    if (max_active <= 0) return AFX_OK;
    const unsigned grid = brick_grid(max_active);
    if (a.n_max > 1 << 24) {  // node numbers past 24 bits
        if (a.k <= 4) brick_warp_kernel<4, unsigned long long><<<grid, kBrickVox, 0, st>>>(a);
        else brick_warp_kernel<8, unsigned long long><<<grid, kBrickVox, 0, st>>>(a);
    } else {
        if (a.k <= 4) brick_warp_kernel<4, unsigned><<<grid, kBrickVox, 0, st>>>(a);
        else brick_warp_kernel<8, unsigned><<<grid, kBrickVox, 0, st>>>(a);
    }
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int launch_brick_integrate(const WarpedIntegrateArgs& a, long max_active, cudaStream_t st) {
    if (max_active <= 0) return AFX_OK;
    if (a.fmt == kVoxF16) brick_integrate_kernel<__half, unsigned short><<<brick_grid(max_active), kBrickVox, 0, st>>>(a);
    else brick_integrate_kernel<float, float><<<brick_grid(max_active), kBrickVox, 0, st>>>(a);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

long brick_count_total(const Volume& vol) { return make_bricks(vol).n; }

// ------------------------------------------------------------------------------------
// Dense per-voxel stage kernels (the reference's layouts)
// ------------------------------------------------------------------------------------

// Calls f(i, count) for the voxels that have neighbours.  They are few and lie together along x, so what these
// kernels spend their time on is the others' counts: a thread looks at four, 32 apart, whose loads are in
// flight together, and a warp's idle groups are skipped.  200^3 voxels, a sixth of them supported: collisions 17.7 ->
// 6.9 us, integration 17.8 -> 11.5 us, weights 18.6 -> 15.2 us (the warp, which is bound by its gathers, gained nothing).
// In small volumes the weights of the supported voxels bound their kernel, not the counts, and four to a thread leave too few
// threads to hide them: an eighth of the voxels supported, k = 8, 64^3 8.2 us (14.5 with four), 128^3 17 (21), 160^3 25
// (26), 200^3 43 (45; a sixth in a block at k = 4, as in a sequence, 35 and 25).
constexpr int kVoxPerThread = 4;
constexpr long kFewVoxels = 3000000;

template <int kVox, class F>
AFX_D void each_supported(const int* __restrict__ kcount, long S, F&& f) {
    const int lane = threadIdx.x & 31;
    const long base = ((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5) * (32 * kVox) + lane;
    int c[kVox];
#pragma unroll
    for (int q = 0; q < kVox; ++q) c[q] = base + 32 * q < S ? kcount[base + 32 * q] : 0;
#pragma unroll
    for (int q = 0; q < kVox; ++q)
        if (c[q]) f(base + 32 * q, c[q]);
}

template <int kVox>
__global__ void tsdf_weights_kernel(float* kw, const float* radii, const uint32_t* kidx, const float* kdist,
                                    const int* kcount, long S, int k) {
    // as the reference: empty voxels keep whatever the array held
    each_supported<kVox>(kcount, S, [&](long i, int cnt) {
        float w[kMaxK];
        float sum = 0.f;
        for (int s = 0; s < k; ++s) w[s] = 0.f;
        for (int s = 0; s < cnt && s < k; ++s) {
            float r = radii[kidx[i * k + s]], d = kdist[i * k + s];
            w[s] = afx_expf(-(d * d) / (2.0f * (r * r)));
            sum = sum + w[s];
        }
        if (sum != 0.f)
            for (int s = 0; s < k; ++s) w[s] = w[s] / sum;
        for (int s = 0; s < k; ++s) kw[i * k + s] = w[s];
    });
}

__global__ void tsdf_vertices_kernel(float* v, Volume vol) {
    long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long S = (long)vol.dims[0] * vol.dims[1] * vol.dims[2];
    if (i >= S) return;
    int x = i % vol.dims[0], y = (i / vol.dims[0]) % vol.dims[1], z = i / ((long)vol.dims[0] * vol.dims[1]);
    voxel_to_world(x, y, z, vol.vs, vol.half, v + 3 * i);
}

// The same where rows start on 16 bytes (dims[0] a multiple of four): a warp per row writes four coordinates a lane,
// and only x changes along it.  With a thread per voxel, two divisions for 12 bytes in three stores set the time:
// 200^3 took 31 us, now 16.
__global__ void __launch_bounds__(256) tsdf_vertices_rows_kernel(float4* v, Volume vol) {
    const long row = blockIdx.x * 8L + (threadIdx.x >> 5), rows = (long)vol.dims[1] * vol.dims[2];
    if (row >= rows) return;
    const int z = (int)(row / vol.dims[1]), y = (int)(row - (long)z * vol.dims[1]), n = vol.dims[0] / 4 * 3;
    v += row * n;
    for (int f = threadIdx.x & 31; f < n; f += 32) {
        const int x = 4 * f / 3, c = 4 * f - 3 * x;
        float a[3], b[3];
        voxel_to_world(x, y, z, vol.vs, vol.half, a);
        voxel_to_world(x + 1, y, z, vol.vs, vol.half, b);
        v[f] = c == 0 ? make_float4(a[0], a[1], a[2], b[0]) : c == 1 ? make_float4(a[1], a[2], b[0], b[1]) : make_float4(a[2], b[0], b[1], b[2]);
    }
}

__global__ void warp_tsdf_kernel(float* verts, const float* T, const uint32_t* kidx, const float* kw,
                                 const int* kcount, long S, int k) {
    long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= S) return;
    int cnt = kcount[i];
    if (!cnt) return;
    bool zero = true;
    for (int s = 0; s < k; ++s)
        if (!(fabsf(kw[i * k + s]) <= 1e-5f)) zero = false;
    if (zero) return;
    float p[3] = {verts[3 * i], verts[3 * i + 1], verts[3 * i + 2]};
    float q[3] = {0.f, 0.f, 0.f};
    for (int s = 0; s < cnt; ++s) {
        float o[3];
        mat4_point(T + 16 * (long)kidx[i * k + s], p, o);
        float w = kw[i * k + s];
        q[0] = q[0] + w * o[0];
        q[1] = q[1] + w * o[1];
        q[2] = q[2] + w * o[2];
    }
    verts[3 * i] = q[0];
    verts[3 * i + 1] = q[1];
    verts[3 * i + 2] = q[2];
}

AFX_D long warped_target(const float* wp, const Volume& vol, const float* Rinv, const float* t) {
    float d[3] = {wp[0] - t[0], wp[1] - t[1], wp[2] - t[2]};
    float o[3];
    mat3_vec3(Rinv, d, o);
    int v[3];
    world_to_voxel(o, vol.inv, vol.half, v);
    if (v[0] < 0 || v[1] < 0 || v[2] < 0 || v[0] >= vol.dims[0] || v[1] >= vol.dims[1] || v[2] >= vol.dims[2])
        return -1;
    return ((long)v[2] * vol.dims[1] + v[1]) * vol.dims[0] + v[0];
}

struct DenseWarpArgs {
    Volume vol;
    float Rinv[9];
    float t[3];
};

__global__ void count_collisions_kernel(int* counts, const float* verts, const int* kcount, DenseWarpArgs a) {
    each_supported<kVoxPerThread>(kcount, (long)a.vol.dims[0] * a.vol.dims[1] * a.vol.dims[2], [&](long i, int) {
        const long tg = warped_target(verts + 3 * i, a.vol, a.Rinv, a.t);
        if (tg >= 0) atomicAdd(counts + tg, 1);
    });
}

__global__ void integrate_warped_kernel(float* tsdf, float* weights, const float* verts, const int* coll,
                                        const int* kcount, const float* depth, int W, int H, float delta,
                                        Intrinsics K, DenseWarpArgs a) {
    each_supported<kVoxPerThread>(kcount, (long)a.vol.dims[0] * a.vol.dims[1] * a.vol.dims[2], [&](long i, int) {
        const long tg = warped_target(verts + 3 * i, a.vol, a.Rinv, a.t);
        if (tg < 0 || coll[tg] > 1) return;
        float tn;
        if (!tsdf_update_value(verts + 3 * i, depth, W, H, delta, K, &tn)) return;
        float t = tsdf[i], w = weights[i];
        tsdf_blend(t, w, tn);
        tsdf[i] = t;
        weights[i] = w;
    });
}

static void inverse3(const float* R, float* Rinv) {
    // Mat3f::inverse() for the rotations the pipeline passes; identity stays exact
    double a[9];
    for (int i = 0; i < 9; ++i) a[i] = R[i];
    // column-major: a[c*3 + r]
    auto m = [&](int r, int c) { return a[c * 3 + r]; };
    double det = m(0, 0) * (m(1, 1) * m(2, 2) - m(1, 2) * m(2, 1)) - m(0, 1) * (m(1, 0) * m(2, 2) - m(1, 2) * m(2, 0)) +
                 m(0, 2) * (m(1, 0) * m(2, 1) - m(1, 1) * m(2, 0));
    double inv[3][3];
    inv[0][0] = (m(1, 1) * m(2, 2) - m(1, 2) * m(2, 1)) / det;
    inv[0][1] = (m(0, 2) * m(2, 1) - m(0, 1) * m(2, 2)) / det;
    inv[0][2] = (m(0, 1) * m(1, 2) - m(0, 2) * m(1, 1)) / det;
    inv[1][0] = (m(1, 2) * m(2, 0) - m(1, 0) * m(2, 2)) / det;
    inv[1][1] = (m(0, 0) * m(2, 2) - m(0, 2) * m(2, 0)) / det;
    inv[1][2] = (m(0, 2) * m(1, 0) - m(0, 0) * m(1, 2)) / det;
    inv[2][0] = (m(1, 0) * m(2, 1) - m(1, 1) * m(2, 0)) / det;
    inv[2][1] = (m(0, 1) * m(2, 0) - m(0, 0) * m(2, 1)) / det;
    inv[2][2] = (m(0, 0) * m(1, 1) - m(0, 1) * m(1, 0)) / det;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) Rinv[c * 3 + r] = (float)inv[r][c];
}

void rotation_inverse(const float* R, float* Rinv) { inverse3(R, Rinv); }

}  // namespace afx

using namespace afx;

extern "C" {

int afx_integrate_tsdf(float* tsdf, float* weights, const float* depth, int width, int height, float delta,
                       const int dims[3], const float voxel_size[3], const float volume_size[3], const float rotate[9],
                       const float translate[3], const float K[9], void* stream) {
    if (!tsdf || !weights || !depth || !dims || !voxel_size || !volume_size || !rotate || !translate || !K)
        return AFX_ERR_INVALID_ARGUMENT;
    if (width <= 0 || height <= 0 || dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0) return AFX_ERR_INVALID_ARGUMENT;
    return integrate_rigid_impl(tsdf, weights, kVoxF32, depth, width, height, delta,
                                make_volume(dims, voxel_size, volume_size),
                                rotate, translate, K, as_stream(stream));
}

int afx_integrate_tsdf_fresh(float* tsdf, float* weights, const float* depth, int width, int height, float delta,
                             const int dims[3], const float voxel_size[3], const float volume_size[3],
                             const float rotate[9], const float translate[3], const float K[9], void* stream) {
    if (!tsdf || !weights || !depth || !dims || !voxel_size || !volume_size || !rotate || !translate || !K)
        return AFX_ERR_INVALID_ARGUMENT;
    if (width <= 0 || height <= 0 || dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0) return AFX_ERR_INVALID_ARGUMENT;
    const Volume vol = make_volume(dims, voxel_size, volume_size);
    if (!rows_vectorize(tsdf, weights, vol, sizeof(float))) return AFX_ERR_UNSUPPORTED;
    return integrate_fresh_impl(tsdf, weights, depth, width, height, delta, vol, rotate, translate, K, as_stream(stream));
}

size_t afx_tsdf_knn_workspace_size(const int dims[3], int n_nodes, const int voxels_per_node[3]) {
    float one[3] = {1, 1, 1};
    if (!dims || !voxels_per_node) return 0;
    return support_workspace_size(make_volume(dims, one, one), n_nodes, voxels_per_node);
}

int afx_tsdf_knn(uint32_t* knn_idx, float* knn_dist, int* knn_counts, const float* nodes, const float* radii,
                 int n_nodes, const float voxel_size[3], const float volume_size[3], const int dims[3],
                 const int voxels_per_node[3], int k, void* workspace, size_t workspace_bytes, void* stream) {
    if (!knn_idx || !knn_dist || !knn_counts || (!nodes && n_nodes) || !dims || k < 1 || k > kMaxK || n_nodes < 0)
        return AFX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    Volume vol = make_volume(dims, voxel_size, volume_size);
    SupportWorkspace s;
    if (!carve_support(workspace, workspace_bytes, vol, n_nodes, voxels_per_node, &s)) return AFX_ERR_WORKSPACE;
    const long S = (long)dims[0] * dims[1] * dims[2];
    AFX_CUDA(cudaMemsetAsync(knn_counts, 0, S * sizeof(int), st));
    int* d_n = reinterpret_cast<int*>(s.n_active) + 1;  // spare word in the n_active slot
    int* d_err = reinterpret_cast<int*>(s.n_active) + 2;
    AFX_CUDA(cudaMemcpyAsync(d_n, &n_nodes, sizeof(int), cudaMemcpyHostToDevice, st));
    AFX_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int), st));
    int st_ = build_support(s, vol, voxels_per_node, nodes, radii, d_n, n_nodes, d_err, st);
    if (st_) return st_;
    WarpArgs a;
    std::memset(&a, 0, sizeof(a));
    a.vol = vol;
    a.bg = make_bricks(vol);
    a.k = k;
    a.n_max = n_nodes;
    a.nodes_t = nodes;
    a.radii = radii;
    a.brick_offset = s.brick_offset;
    a.brick_count = s.brick_count;
    a.brick_nodes = s.brick_nodes;
    a.active = s.active;
    a.n_active = s.n_active;
    for (int c = 0; c < 3; ++c) a.per[c] = voxels_per_node[c];
    a.dense_idx = knn_idx;
    a.dense_dist = knn_dist;
    a.dense_count = knn_counts;
    a.error = d_err;
    int rc = launch_brick_warp(a, a.bg.n, st);
    if (rc) return rc;
    int err = 0;
    AFX_CUDA(cudaMemcpyAsync(&err, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    AFX_CUDA(cudaStreamSynchronize(st));
    return err ? AFX_ERR_CAPACITY : AFX_OK;
}

int afx_tsdf_warp_weights(float* knn_weights, const float* radii, const uint32_t* knn_idx, const float* knn_dist,
                          const int* knn_counts, long n_voxels, int k, void* stream) {
    if (!knn_weights || !radii || !knn_idx || !knn_dist || !knn_counts || k < 1 || k > kMaxK)
        return AFX_ERR_INVALID_ARGUMENT;
    if (n_voxels <= 0) return AFX_OK;
    const int per = n_voxels < kFewVoxels ? 1 : kVoxPerThread;
    const auto kernel = per == 1 ? tsdf_weights_kernel<1> : tsdf_weights_kernel<kVoxPerThread>;
    kernel<<<blocks_for(n_voxels, 256 * per), 256, 0, as_stream(stream)>>>(knn_weights, radii, knn_idx, knn_dist, knn_counts, n_voxels,
                                                                          k);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_tsdf_vertices(float* vertices, const float voxel_size[3], const float volume_size[3], const int dims[3],
                      void* stream) {
    if (!vertices || !dims) return AFX_ERR_INVALID_ARGUMENT;
    Volume vol = make_volume(dims, voxel_size, volume_size);
    long S = (long)dims[0] * dims[1] * dims[2];
    if (dims[0] % 4 == 0 && !((size_t)vertices & 15))
        tsdf_vertices_rows_kernel<<<blocks_for((long)dims[1] * dims[2], 8), 256, 0, as_stream(stream)>>>(
            reinterpret_cast<float4*>(vertices), vol);
    else
        tsdf_vertices_kernel<<<blocks_for(S, 256), 256, 0, as_stream(stream)>>>(vertices, vol);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_warp_tsdf(float* vertices, const float* transforms, const uint32_t* knn_idx, const float* knn_weights,
                  const int* knn_counts, long n_voxels, int k, void* stream) {
    if (!vertices || !transforms || !knn_idx || !knn_weights || !knn_counts || k < 1 || k > kMaxK)
        return AFX_ERR_INVALID_ARGUMENT;
    if (n_voxels <= 0) return AFX_OK;
    warp_tsdf_kernel<<<blocks_for(n_voxels, 256), 256, 0, as_stream(stream)>>>(vertices, transforms, knn_idx,
                                                                               knn_weights, knn_counts, n_voxels, k);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_count_collisions(int* counts, const float* vertices, const int* knn_counts, const float voxel_size[3],
                         const float volume_size[3], const int dims[3], const float rotate[9], const float translate[3],
                         void* stream) {
    if (!counts || !vertices || !knn_counts || !dims || !rotate || !translate) return AFX_ERR_INVALID_ARGUMENT;
    DenseWarpArgs a;
    a.vol = make_volume(dims, voxel_size, volume_size);
    rotation_inverse(rotate, a.Rinv);
    for (int c = 0; c < 3; ++c) a.t[c] = translate[c];
    long S = (long)dims[0] * dims[1] * dims[2];
    count_collisions_kernel<<<blocks_for(S, 256 * kVoxPerThread), 256, 0, as_stream(stream)>>>(counts, vertices, knn_counts, a);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_integrate_warped_tsdf(float* tsdf, float* weights, const float* vertices, const int* collisions,
                              const int* knn_counts, const float* depth, int width, int height, float delta,
                              const float voxel_size[3], const float volume_size[3], const int dims[3],
                              const float rotate[9], const float translate[3], const float K[9], void* stream) {
    if (!tsdf || !weights || !vertices || !collisions || !knn_counts || !depth || !dims || !K)
        return AFX_ERR_INVALID_ARGUMENT;
    DenseWarpArgs a;
    a.vol = make_volume(dims, voxel_size, volume_size);
    rotation_inverse(rotate, a.Rinv);
    for (int c = 0; c < 3; ++c) a.t[c] = translate[c];
    long S = (long)dims[0] * dims[1] * dims[2];
    integrate_warped_kernel<<<blocks_for(S, 256 * kVoxPerThread), 256, 0, as_stream(stream)>>>(
        tsdf, weights, vertices, collisions, knn_counts, depth, width, height, delta, make_intrinsics(K), a);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

}  // extern "C"
