// afx_graph.cu -- motion graph on the device: greedy radius subsampling (af::buildGraph),
// exact K-nearest-node queries (af::getKnnData), graph-edge pruning
// (af::filterDisconnected), skinning weights, linear-blend warp and projective
// correspondences.  The reference does the first three on the host with nanoflann,
// copying the point cloud down and the results up every frame (src/VolumeFusion.cu:392-419).
#include <cfloat>
#include <cmath>
#include <cstring>
#include <mutex>

#include "afx_dqb.cuh"
#include "afx_host.h"
#include "afx_internal.h"

namespace afx {

// ------------------------------------------------------------------------------------
// Graph build
// ------------------------------------------------------------------------------------
//
// af::buildGraph visits the sorted point cloud in order and inserts a point as a node
// when none of its K nearest nodes lies closer than that node's radius.  With one radius
// for all nodes (what the pipeline uses) that is: insert p_i iff no node -- existing, or
// inserted earlier in the same call -- is within distance < r.  The device version inserts
// exactly those points:
//   1. points already covered by existing nodes are dropped in parallel; the others
//      (candidates) are bucketed by the cells of a grid whose cell is a little over r, so that
//      points within r of each other are in the same or in adjacent cells;
//   2. one CTA takes the candidates in rounds.  A candidate that is earlier than every other
//      undecided one of its own and the 26 adjacent cells has had every earlier point near it
//      decided, so it is inserted now as the sequential walk would insert it; the candidates it
//      covers are removed.  All such candidates of a round are independent of one another, and
//      the earliest one of all always is one, so rounds end.  A round costs about as much as one
//      step of the walk, and there are a few per node spacing along the cloud's order instead of
//      one per node;
//   3. a new node copies the transform of its nearest node at insertion time, that is among the
//      nodes before it (src/GraphBuilder.cpp:38-48; equal distances go to the lower node index):
//      searched for all new nodes in parallel once their order is known.

constexpr int kGridSlots = 32;
constexpr int kGridMaxCells = 1 << 18;
constexpr float kCellMargin = 1.02f;  // candidate cells over grid cells: more than the rounding of a cell index
constexpr int kSmallCells = 2048;     // candidate cells whose state fits in shared memory, with a neighbour table
constexpr int kGreedyThreads = 1024;
constexpr int kPickMax = 32;          // candidates inserted per round: a bit each of a cell's word
constexpr int kNearMax = 8;            // points of a round around a cell: their cells are not adjacent to one another
constexpr unsigned kNoCell = 0xffffffffu;
constexpr unsigned kGone = 0xffffffffu;  // point index of a decided candidate

struct Grid {
    float org[3];
    float cell;
    int dims[3];
    float ccell;   // candidate cells: same origin
    int cdims[3];
    int* cnt;    // [cells]
    int* slots;  // [cells * kGridSlots]
};

struct GraphCounters {  // cleared at the start of a build
    unsigned kmin[3], kmax[3];  // bounding box as ordered keys (the smallest as the largest complement)
    unsigned done[3];           // blocks finished: bounding box, candidates, nearest nodes
    unsigned ncell, ncand;
    int n_old;                  // nodes before the build
    int first_new;              // and the first node that copies a transform
};

struct GraphState {
    float* nodes;
    float* radii;
    float* T;
    int* n_nodes;
    int cap;
    const float* mesh;
    const unsigned* mesh_count;
    long mesh_max;
    float r;
    float r2;            // the smallest float whose square root is not below r: sqrtf(d) < r <=> d < r2
    Grid g;
    unsigned* pcell;     // [mesh_max] candidate cell of each point, kNoCell if covered
    unsigned* prank;     // [mesh_max] its place in the cell; from the end of the rounds: parent of each new node
    float4* sorted;      // [mesh_max] candidates by cell: position, point index
    unsigned* picked;    // [mesh_max / 32 + 1] bit per inserted point
    unsigned* ccnt;      // [kGridMaxCells] candidates per grid cell
    unsigned* cid;       // [kGridMaxCells] its index among the occupied ones
    unsigned* gcell;     // [kGridMaxCells] per occupied cell: grid cell,
    unsigned* cstart;    // first candidate,
    unsigned* ccount;    // number of them,
    unsigned* cmin;      // the earliest undecided one (0xffffffff: none),
    unsigned* cblock;    // the adjacent cell that holds an earlier one,
    unsigned* cnear;     // and the number of the round's inserted points around it
    unsigned* cwork;     // cells around the round's points
    float4* cpos;        // its position and index
    float4* cpick;       // [kNearMax] those of the round's inserted points around it
    unsigned short* nbr; // [kSmallCells * 32] adjacent occupied cells (27 used), 0xffff: none
    float* fac;          // [mesh_max] per new node: d / (0 + d)
    GraphCounters* k;
    int* error;          // [1]
};

AFX_D int ford(float f) {
    int i = __float_as_int(f);
    return i < 0 ? (int)(0x80000000u - (unsigned)i) : i;
}
AFX_D float ordf(int o) { return __int_as_float(o < 0 ? (int)(0x80000000u - (unsigned)o) : o); }

AFX_D int grid_cell(const Grid& g, const float* p, int* c3) {
    for (int c = 0; c < 3; ++c) {
        int v = (int)floorf((p[c] - g.org[c]) / g.cell);
        c3[c] = min(max(v, 0), g.dims[c] - 1);
    }
    return (c3[2] * g.dims[1] + c3[1]) * g.dims[0] + c3[0];
}

AFX_D void grid_insert(const Grid& g, const float* p, int idx, int* error) {
    int c3[3];
    int cell = grid_cell(g, p, c3);
    int k = atomicAdd(g.cnt + cell, 1);
    if (k < kGridSlots) g.slots[(long)cell * kGridSlots + k] = idx;
    else atomicOr(error, ERRF_CAPACITY);
}

// True in every thread of the block that finishes last (all blocks' writes are then visible to it).
AFX_D bool last_block(unsigned* done) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Chooses the grids from the bounding box and seeds the first node when the graph is empty
// (src/GraphBuilder.cpp:19-20).  One thread.
AFX_D void graph_setup(const GraphState& s, Grid* gout) {
    const long m = min((long)*s.mesh_count, s.mesh_max);
    const int n = *s.n_nodes;
    s.k->n_old = n;
    Grid g = s.g;
    float lo[3], hi[3], ext = 0.f;
    for (int c = 0; c < 3; ++c) {
        lo[c] = ordf((int)(~__ldcg(&s.k->kmin[c]) ^ 0x80000000u));
        hi[c] = ordf((int)(__ldcg(&s.k->kmax[c]) ^ 0x80000000u));
        if (!(lo[c] <= hi[c])) lo[c] = hi[c] = 0.f;
        ext = fmaxf(ext, hi[c] - lo[c]);
    }
    float cell = s.r > 0.f ? s.r : 1.f;
    if (!(ext < 1e6f)) {  // non-finite coordinates: refuse rather than size a grid from them
        atomicOr(s.error, ERRF_UNSUPPORTED);
        for (int c = 0; c < 3; ++c) lo[c] = hi[c] = 0.f;
    }
    for (int guard = 0; guard < 200; ++guard) {
        long cells = 1;
        for (int c = 0; c < 3; ++c) cells *= (long)((hi[c] - lo[c]) / cell) + 2;
        if (cells <= kGridMaxCells) break;
        cell *= 1.25f;
    }
    g.cell = cell;
    g.ccell = cell * kCellMargin;
    for (int c = 0; c < 3; ++c) {
        g.org[c] = lo[c] - cell * 0.5f;
        g.dims[c] = (int)((hi[c] - lo[c]) / cell) + 2;
        g.cdims[c] = min((int)((hi[c] - g.org[c]) / g.ccell) + 1, g.dims[c]);
    }
    if (cell > 2.0f * s.r) atomicOr(s.error, ERRF_CAPACITY);  // more than 32 nodes per cell possible
    *gout = g;
    s.k->first_new = n;
    if (n == 0 && m > 0) {
        if (s.cap < 1) {
            atomicOr(s.error, ERRF_CAPACITY);
            return;
        }
        for (int c = 0; c < 3; ++c) s.nodes[c] = s.mesh[c];
        s.radii[0] = s.r;
        for (int e = 0; e < 16; ++e) s.T[e] = (e % 5 == 0) ? 1.f : 0.f;
        *s.n_nodes = 1;
        s.k->first_new = 1;
    }
}

// Bounding box of the point cloud and the existing nodes (one atomic per block and side) and a check
// of the radii; the block that finishes last chooses the grids and enters the existing nodes.
__global__ void __launch_bounds__(1024) graph_bbox_kernel(GraphState s, Grid* gout) {
    __shared__ unsigned smn[3][32], smx[3][32];
    const long m = min((long)*s.mesh_count, s.mesh_max);
    const int n = min(*s.n_nodes, s.cap);
    unsigned mn[3] = {0u, 0u, 0u}, mx[3] = {0u, 0u, 0u};  // largest complement, largest key
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < m + n; i += (long)gridDim.x * blockDim.x) {
        const float* p = i < m ? s.mesh + 3 * i : s.nodes + 3 * (i - m);
        for (int c = 0; c < 3; ++c) {
            const unsigned u = (unsigned)ford(p[c]) ^ 0x80000000u;
            mn[c] = max(mn[c], ~u);
            mx[c] = max(mx[c], u);
        }
        if (i >= m && s.radii[i - m] != s.r) atomicOr(s.error, ERRF_UNSUPPORTED);
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int c = 0; c < 3; ++c) {
        mn[c] = __reduce_max_sync(0xffffffffu, mn[c]);
        mx[c] = __reduce_max_sync(0xffffffffu, mx[c]);
        if (lane == 0) {
            smn[c][w] = mn[c];
            smx[c][w] = mx[c];
        }
    }
    __syncthreads();
    if (w < 3) {
        const unsigned a = __reduce_max_sync(0xffffffffu, smn[w][lane]), b = __reduce_max_sync(0xffffffffu, smx[w][lane]);
        if (lane == 0) {
            atomicMax(&s.k->kmin[w], a);
            atomicMax(&s.k->kmax[w], b);
        }
    }
    if (!last_block(&s.k->done[0])) return;
    __shared__ int s_n;
    if (threadIdx.x == 0) {
        graph_setup(s, gout);
        s_n = min(*s.n_nodes, s.cap);
    }
    __syncthreads();
    const Grid g = *gout;
    for (int i = threadIdx.x; i < s_n; i += blockDim.x) grid_insert(g, s.nodes + 3 * (long)i, i, s.error);
}

// Any node in the grid with distance < r?  (radius test of src/GraphBuilder.cpp:28-34)  The counts of
// the cells, three in a row at a time, are loaded before the nodes of the occupied ones.
AFX_D bool grid_covered(const Grid& g, const float* nodes, const float* p, float r2) {
    int c3[3];
    grid_cell(g, p, c3);
    int cnt[27];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int y = c3[1] + q % 3 - 1, z = c3[2] + q / 3 - 1;
        const bool in = y >= 0 && z >= 0 && y < g.dims[1] && z < g.dims[2];
        const int* row = g.cnt + ((long)z * g.dims[1] + y) * g.dims[0] + c3[0];
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const int x = c3[0] + dx;
            cnt[3 * q + dx + 1] = (in && x >= 0 && x < g.dims[0]) ? __ldg(row + dx) : 0;
        }
    }
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int c = min(cnt[q], kGridSlots);
        if (c == 0) continue;
        const int x = c3[0] + q % 3 - 1, y = c3[1] + (q / 3) % 3 - 1, z = c3[2] + q / 9 - 1;
        const int* slot = g.slots + ((long)(z * g.dims[1] + y) * g.dims[0] + x) * kGridSlots;
        for (int k = 0; k < c; ++k)
            if (l2sq_nanoflann(p, nodes + 3 * (long)__ldg(slot + k)) < r2) return true;
    }
    return false;
}

// Candidates (live points no node covers), counted by cell; the block that finishes last gives the
// occupied cells their places in the bucketed order.
__global__ void __launch_bounds__(256) graph_candidates_kernel(GraphState s, const Grid* gp) {
    const long m = min((long)*s.mesh_count, s.mesh_max);
    const Grid g = *gp;
    const int lane = threadIdx.x & 31;
    const long t0 = blockIdx.x * (long)blockDim.x + threadIdx.x, nt = (long)gridDim.x * blockDim.x;
    for (long i = t0; i < (m + 31) / 32; i += nt) s.picked[i] = 0u;
    for (long i0 = t0 - lane; i0 < m; i0 += nt) {  // whole warps
        const long i = i0 + lane;
        unsigned cell = kNoCell;
        if (i < m) {
            const float p[3] = {s.mesh[3 * i], s.mesh[3 * i + 1], s.mesh[3 * i + 2]};
            if (!grid_covered(g, s.nodes, p, s.r2)) {
                int c3[3];
                for (int c = 0; c < 3; ++c) {
                    const int v = (int)floorf((p[c] - g.org[c]) / g.ccell);
                    c3[c] = min(max(v, 0), g.cdims[c] - 1);
                }
                cell = (unsigned)((c3[2] * g.cdims[1] + c3[1]) * g.cdims[0] + c3[0]);
            }
            s.pcell[i] = cell;
        }
        const unsigned same = __match_any_sync(0xffffffffu, cell);
        const int lead = __ffs(same) - 1;
        unsigned base = 0;
        if (lane == lead && cell != kNoCell) {
            base = atomicAdd(s.ccnt + cell, (unsigned)__popc(same));
            if (base == 0) {
                const unsigned c = atomicAdd(&s.k->ncell, 1u);
                s.cid[cell] = c;
                s.gcell[c] = cell;
            }
        }
        base = __shfl_sync(0xffffffffu, base, lead);
        if (i < m) s.prank[i] = base + __popc(same & ((1u << lane) - 1u));
    }
    if (!last_block(&s.k->done[1])) return;
    const unsigned nc = __ldcg(&s.k->ncell);
    for (unsigned c0 = 0; c0 < nc; c0 += blockDim.x) {
        const unsigned c = c0 + threadIdx.x;
        const unsigned n = c < nc ? __ldcg(s.ccnt + __ldcg(s.gcell + c)) : 0u;
        unsigned incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        unsigned base = 0;
        if (lane == 31) base = atomicAdd(&s.k->ncand, incl);
        base = __shfl_sync(0xffffffffu, base, 31);
        if (c < nc) {
            s.cstart[c] = base + incl - n;
            s.ccount[c] = n;
            s.cmin[c] = 0xffffffffu;
            s.cblock[c] = kNoCell;
            s.cnear[c] = 0u;
        }
    }
}

// Occupied cell adjacent to the occupied cell c in direction k (0 .. 26), or -1.
AFX_D int adjacent_cell(const GraphState& s, const Grid& g, unsigned c, int k) {
    const int cell = (int)s.gcell[c];
    const int x = cell % g.cdims[0] + k % 3 - 1, y = (cell / g.cdims[0]) % g.cdims[1] + (k / 3) % 3 - 1,
              z = cell / (g.cdims[0] * g.cdims[1]) + k / 9 - 1;
    if (x < 0 || y < 0 || z < 0 || x >= g.cdims[0] || y >= g.cdims[1] || z >= g.cdims[2]) return -1;
    const int q = (z * g.cdims[1] + y) * g.cdims[0] + x;
    return s.ccnt[q] ? (int)s.cid[q] : -1;
}

// The candidates in bucketed order, the earliest one of each cell, and the adjacent cells.
__global__ void __launch_bounds__(256) graph_bucket_kernel(GraphState s, const Grid* gp) {
    const unsigned nc = s.k->ncell;
    if (nc == 0) return;
    const long m = min((long)*s.mesh_count, s.mesh_max);
    const Grid g = *gp;
    const int lane = threadIdx.x & 31;
    const long t0 = blockIdx.x * (long)blockDim.x + threadIdx.x, nt = (long)gridDim.x * blockDim.x;
    for (long i0 = t0 - lane; i0 < m; i0 += nt) {
        const long i = i0 + lane;
        const unsigned cell = i < m ? s.pcell[i] : kNoCell;
        const unsigned c = cell != kNoCell ? s.cid[cell] : kNoCell;
        const unsigned same = __match_any_sync(0xffffffffu, c);
        if (c == kNoCell) continue;
        if (lane == __ffs(same) - 1) atomicMin(s.cmin + c, (unsigned)i);
        s.sorted[s.cstart[c] + s.prank[i]] =
            make_float4(s.mesh[3 * i], s.mesh[3 * i + 1], s.mesh[3 * i + 2], __uint_as_float((unsigned)i));
    }
    if (nc <= kSmallCells)
        for (long t = t0; t < (long)nc * 32; t += nt)
            if ((t & 31) < 27) s.nbr[t] = (unsigned short)adjacent_cell(s, g, (unsigned)(t >> 5), (int)(t & 31));
}

// The rounds, on one CTA.  A cell is examined again only when the adjacent cell that held it back no
// longer holds an earlier candidate.  Two barriers per round: (a) every warp goes through its share of
// the cells; a cell to examine either has its earliest candidate inserted, or is held back by the
// adjacent cell with the earliest one; (b) a warp per cell around an inserted point: the candidates it
// covers are marked and the earliest of the others found (a cell is gone through about five times;
// closing up its list instead wrote far more).
// Bound: the latency of a round -- two barriers, one load from L2 and about ten dependent accesses of
// shared memory, 2 to 3 us.  60,000 candidates and 295 nodes: 104 rounds, 0.30 ms (0.38 ms with 512
// threads: a warp then examines two cells in turn), where a walk in chunks of 1024 candidates, each
// tested against every node, took 1.76 ms.  The first frame of the 512^3 sequence, 28,761 candidates
// and 1,300 nodes: 232 rounds, 0.50 ms from 3.6 ms; a frame with nothing to insert: 2 us from 20 us.
struct GreedyCells {   // per occupied cell, in shared memory (up to kSmallCells of them)
    float4* pos;       // the earliest undecided candidate: position, point index
    unsigned* cmin;    // the index again (0xffffffff: none)
    unsigned* block;   // the adjacent cell that held an earlier one (kNoCell: to be examined)
    unsigned* near;    // the round's inserted points around it, a bit each
    unsigned* start;   // its candidates: first place in `sorted`
    unsigned* count;   // and number
    unsigned short* nbr;  // adjacent occupied cells, kNbr per cell (0xffff: none)
};
constexpr int kNbr = 28;  // 27 and a pad
__host__ __device__ constexpr unsigned padded_cells(unsigned n) { return n + n / 32 + 1; }
constexpr size_t kGreedySmem = (size_t)kSmallCells * (sizeof(float4) + 3 * sizeof(unsigned) + kNbr * sizeof(unsigned short)) +
                               2 * padded_cells(kSmallCells) * sizeof(unsigned) + 16;

struct GreedyLists {
    unsigned work[kPickMax * 27];
    float4 pick[kPickMax];
    unsigned npick[2], nwork[2];  // of odd and even rounds
    unsigned wsum[kGreedyThreads / 32];
};

// What a warp that goes through a cell's candidates keeps: those covered by the round's points around the cell (`near`: the
// lanes or places that hold one, point(i) gives it) are marked, the earliest of the others is returned in `best` of the
// lane whose `first` is the result.
template <class Point>
AFX_D unsigned mark_covered(float4* list, unsigned n, unsigned near, float r2, Point&& point, unsigned& first, float4& best) {
    const int lane = threadIdx.x & 31;
    constexpr int kAhead = 4;  // 32-candidate groups loaded together
    first = 0xffffffffu;
    for (unsigned i0 = 0; i0 < n; i0 += 32 * kAhead) {
        float4 v[kAhead];
        bool gone[kAhead];
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            const unsigned i = i0 + a * 32 + lane;
            v[a] = i < n ? list[i] : make_float4(0.f, 0.f, 0.f, __uint_as_float(kGone));
            gone[a] = false;
        }
        for (unsigned rest = near; rest; rest &= rest - 1) {
            const float4 q4 = point(__ffs(rest) - 1);
            const float q[3] = {q4.x, q4.y, q4.z};
#pragma unroll
            for (int a = 0; a < kAhead; ++a) {
                const float p[3] = {v[a].x, v[a].y, v[a].z};
                gone[a] |= l2sq_nanoflann(p, q) < r2 || __float_as_uint(v[a].w) == __float_as_uint(q4.w);
            }
        }
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            const unsigned id = __float_as_uint(v[a].w);
            if (id == kGone) continue;
            if (gone[a]) {
                list[i0 + a * 32 + lane].w = __uint_as_float(kGone);
            } else if (id < first) {
                first = id;
                best = v[a];
            }
        }
    }
    return __reduce_min_sync(0xffffffffu, first);
}

AFX_D void greedy_rounds(const GraphState& s, unsigned nc, const GreedyCells& C, GreedyLists& L) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned limit = s.k->ncand + 2;
    constexpr unsigned kWarps = kGreedyThreads / 32;
    // A warp's share are the cells w, w + kWarps, ...: cells to examine tend to be consecutive ones.  A word of
    // padding per 32 keeps that access free of bank conflicts.
    auto at = [](unsigned c) { return c + (c >> 5); };
    for (unsigned round = 1; round <= limit; ++round) {
        // (a)
        const int par = round & 1;
        bool some = false;  // a candidate is left
        for (unsigned c0 = w; c0 < nc; c0 += kGreedyThreads) {
            const unsigned mine = c0 + kWarps * lane;
            bool check = false;
            if (mine < nc) {
                const unsigned m = C.cmin[at(mine)], b = C.block[at(mine)];
                check = m != 0xffffffffu && (b == kNoCell || !(C.cmin[at(b)] < m));
                some |= m != 0xffffffffu;
            }
            for (unsigned rest = __ballot_sync(0xffffffffu, check); rest; rest &= rest - 1) {
                const unsigned c = c0 + kWarps * (__ffs(rest) - 1), m = C.cmin[at(c)];
                const int nb = lane < 27 && C.nbr[c * kNbr + lane] != 0xffff ? (int)C.nbr[c * kNbr + lane] : -1;
                const unsigned mm = nb >= 0 ? C.cmin[at(nb)] : 0xffffffffu;
                const unsigned wm = __reduce_min_sync(0xffffffffu, mm);
                if (wm < m) {
                    if (mm == wm) C.block[at(c)] = (unsigned)nb;
                    continue;
                }
                unsigned k = 0;
                if (lane == 0) {
                    k = atomicAdd(&L.npick[par], 1u);
                    C.block[at(c)] = kNoCell;
                    if (k < kPickMax) {
                        L.pick[k] = C.pos[c];
                        atomicOr(s.picked + (m >> 5), 1u << (m & 31));
                    }
                }
                k = __shfl_sync(0xffffffffu, k, 0);
                if (k >= kPickMax) continue;  // in a later round
                const bool first = nb >= 0 && mm != 0xffffffffu && atomicOr(C.near + nb, 1u << k) == 0u;
                const unsigned add = __ballot_sync(0xffffffffu, first);
                unsigned place = 0;
                if (lane == 0) place = atomicAdd(&L.nwork[par], (unsigned)__popc(add));
                place = __shfl_sync(0xffffffffu, place, 0) + __popc(add & ((1u << lane) - 1u));
                if (first) L.work[place] = (unsigned)nb;
            }
        }
        if (!__syncthreads_or(some)) break;
        // (b)
        const unsigned nwork = L.nwork[par];
        if (tid == 0) L.npick[par ^ 1] = L.nwork[par ^ 1] = 0;  // the next round's, unused in this one
        for (unsigned q = w; q < nwork; q += kWarps) {
            const unsigned c = L.work[q];
            unsigned first;
            float4 fp;
            const unsigned wf = mark_covered(s.sorted + C.start[c], C.count[c], C.near[c], s.r2,
                                             [&](int k) { return L.pick[k]; }, first, fp);
            if (wf != 0xffffffffu && first == wf) C.pos[c] = fp;
            if (lane == 0) {
                C.cmin[at(c)] = wf;
                C.near[c] = 0u;
            }
        }
        __syncthreads();
    }
}

// The same with the cells in global memory and no limit on the points of a round: each is left with the cells around it
// (at most kNearMax to a cell).  300,000 points in a plane, 29,000 nodes: 28 ms in the cloud's order, and 23,000
// nodes, 9 ms, in no order; with 32 points a round 42 and 90 ms (the walk in chunks: 45 and 39).
AFX_D void greedy_rounds_large(const GraphState& s, const Grid& g, unsigned nc, GreedyLists& L) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned limit = s.k->ncand + 2;
    constexpr unsigned kWarps = kGreedyThreads / 32;
    for (unsigned round = 1; round <= limit; ++round) {
        // (a)
        const int par = round & 1;
        bool some = false;
        for (unsigned c0 = w; c0 < nc; c0 += kGreedyThreads) {
            const unsigned mine = c0 + kWarps * lane;
            bool check = false;
            if (mine < nc) {
                const unsigned m = s.cmin[mine], b = s.cblock[mine];
                check = m != 0xffffffffu && (b == kNoCell || !(s.cmin[b] < m));
                some |= m != 0xffffffffu;
            }
            for (unsigned rest = __ballot_sync(0xffffffffu, check); rest; rest &= rest - 1) {
                const unsigned c = c0 + kWarps * (__ffs(rest) - 1), m = s.cmin[c];
                const int nb = lane < 27 ? adjacent_cell(s, g, c, lane) : -1;
                const unsigned mm = nb >= 0 ? s.cmin[nb] : 0xffffffffu;
                const unsigned wm = __reduce_min_sync(0xffffffffu, mm);
                if (wm < m) {
                    if (mm == wm) s.cblock[c] = (unsigned)nb;
                    continue;
                }
                if (lane == 0) {
                    s.cblock[c] = kNoCell;
                    atomicOr(s.picked + (m >> 5), 1u << (m & 31));
                }
                const float4 pick = s.cpos[c];
                unsigned k = kNearMax;
                if (nb >= 0 && mm != 0xffffffffu) k = atomicAdd(s.cnear + nb, 1u);
                if (k < kNearMax) s.cpick[(long)nb * kNearMax + k] = pick;
                const bool first = k == 0u;
                const unsigned add = __ballot_sync(0xffffffffu, first);
                unsigned place = 0;
                if (lane == 0) place = atomicAdd(&L.nwork[par], (unsigned)__popc(add));
                place = __shfl_sync(0xffffffffu, place, 0) + __popc(add & ((1u << lane) - 1u));
                if (first) s.cwork[place] = (unsigned)nb;
            }
        }
        if (!__syncthreads_or(some)) break;
        // (b)
        const unsigned nwork = L.nwork[par];
        if (tid == 0) L.nwork[par ^ 1] = 0;
        for (unsigned q = w; q < nwork; q += kWarps) {
            const unsigned c = s.cwork[q], near = min(s.cnear[c], (unsigned)kNearMax);
            const float4* picks = s.cpick + (long)c * kNearMax;
            unsigned first;
            float4 fp;
            const unsigned wf = mark_covered(s.sorted + s.cstart[c], s.ccount[c], (1u << near) - 1u, s.r2,
                                             [&](int k) { return picks[k]; }, first, fp);
            if (wf != 0xffffffffu && first == wf) s.cpos[c] = fp;
            if (lane == 0) {
                s.cmin[c] = wf;
                s.cnear[c] = 0u;
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kGreedyThreads) graph_greedy_kernel(GraphState s, const Grid* gp) {
    extern __shared__ float4 cells[];
    __shared__ GreedyLists L;
    const unsigned nc = s.k->ncell;
    if (nc == 0) return;
    const Grid g = *gp;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid < 2) L.npick[tid] = L.nwork[tid] = 0;
    unsigned* u = reinterpret_cast<unsigned*>(cells + nc);
    unsigned* v = u + 2 * padded_cells(nc);
    const GreedyCells S{cells, u, u + padded_cells(nc), v, v + nc, v + 2 * nc, reinterpret_cast<unsigned short*>(v + 3 * nc)};
    const bool small = nc <= kSmallCells;
    for (unsigned c = tid; c < nc; c += kGreedyThreads) {
        const unsigned m = s.cmin[c];
        const float4 p = make_float4(s.mesh[3 * (long)m], s.mesh[3 * (long)m + 1], s.mesh[3 * (long)m + 2], __uint_as_float(m));
        if (small) {
            S.pos[c] = p;
            S.cmin[c + (c >> 5)] = m;
            S.block[c + (c >> 5)] = kNoCell;
            S.near[c] = 0u;
            S.start[c] = s.cstart[c];
            S.count[c] = s.ccount[c];
        } else {
            s.cpos[c] = p;
        }
    }
    for (unsigned t = tid; small && t < nc * 32; t += kGreedyThreads)
        if ((t & 31) < 27) S.nbr[(t >> 5) * kNbr + (t & 31)] = s.nbr[t];
    __syncthreads();
    if (small) greedy_rounds(s, nc, S, L);
    else greedy_rounds_large(s, g, nc, L);
    __syncthreads();
    // the inserted points in order: nodes n0, n0 + 1, ...
    const long m = min((long)*s.mesh_count, s.mesh_max), words = (m + 31) / 32;
    const int n0 = *s.n_nodes, room = max(s.cap - n0, 0);
    unsigned before = 0;
    for (long w0 = 0; w0 < words; w0 += kGreedyThreads) {
        const long wi = w0 + tid;
        unsigned bits = wi < words ? __ldcg(s.picked + wi) : 0u;
        const unsigned n = (unsigned)__popc(bits);
        unsigned incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) L.wsum[w] = incl;
        __syncthreads();
        unsigned pre = lane < kGreedyThreads / 32 ? L.wsum[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += y;
        }
        const unsigned total = __shfl_sync(0xffffffffu, pre, 31);
        unsigned rank = before + incl - n + (w > 0 ? __shfl_sync(0xffffffffu, pre, w - 1) : 0u);
        for (; bits; bits &= bits - 1, ++rank) {
            if (rank >= (unsigned)room) break;
            const long i = wi * 32 + __ffs(bits) - 1;
            const long node = n0 + (long)rank;
            for (int c = 0; c < 3; ++c) s.nodes[3 * node + c] = s.mesh[3 * i + c];
            s.radii[node] = s.r;
        }
        before += total;
        __syncthreads();
    }
    if (tid == 0) {
        *s.n_nodes = n0 + (int)min(before, (unsigned)room);
        if (before > (unsigned)room) atomicOr(s.error, ERRF_CAPACITY);
    }
}

// Transforms of the new nodes.  A warp per node finds its parent, the nearest node before it; the
// block that finishes last copies T = 0 + T_parent * (d / (0 + d)) down from the nodes that were there
// before.  The factor is 1 unless d is zero or not finite, and 0 + (0 + x) = 0 + x, so with factors of
// 1 on the way a node's transform is 0 + that of the old node its parents lead to; otherwise the
// factors are applied one after the other from that node on.
__global__ void __launch_bounds__(256) graph_transforms_kernel(GraphState s) {
    const int first = s.k->first_new, n = min(*s.n_nodes, s.cap);
    if (first >= n) return;
    unsigned* parent = s.prank;
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5), nw = (int)((gridDim.x * (long)blockDim.x) >> 5);
    for (int i = first + gw; i < n; i += nw) {
        const float p[3] = {s.nodes[3 * (long)i], s.nodes[3 * (long)i + 1], s.nodes[3 * (long)i + 2]};
        float bs = FLT_MAX;
        int bj = 0x7fffffff;
        for (int q = lane; q < i; q += 32) {
            const float d = l2sq_nanoflann(p, s.nodes + 3 * (long)q);
            if (d < bs) {
                bs = d;
                bj = q;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float d = __shfl_xor_sync(0xffffffffu, bs, o);
            const int j = __shfl_xor_sync(0xffffffffu, bj, o);
            if (d < bs || (d == bs && j < bj)) {
                bs = d;
                bj = j;
            }
        }
        if (lane == 0) {
            const float d = sqrtf(bs);
            parent[i - first] = (unsigned)(bj < i ? bj : 0);
            s.fac[i - first] = d / (0.f + d);
        }
    }
    if (!last_block(&s.k->done[2])) return;
    const int cnt = n - first;
    auto up = [&](int i) { return (int)__ldcg(parent + (i - first)); };
    constexpr int kJump = 8192;  // new nodes whose ways up are shortened in shared memory, those of more in global memory
    constexpr unsigned kOdd = 0x80000000u;  // a factor other than 1 on the way
    __shared__ unsigned sp[kJump];
    unsigned* const gp = reinterpret_cast<unsigned*>(s.sorted);  // (not needed once the rounds are over)
    const bool small = cnt <= kJump;
    auto get = [&](int t) { return small ? sp[t] : __ldcg(gp + t); };
    auto put = [&](int t, unsigned v) {
        if (small) sp[t] = v;
        else __stcg(gp + t, v);
    };
    // each node's ancestor, doubled until it is one of the old nodes
    for (int t = threadIdx.x; t < cnt; t += blockDim.x)
        put(t, __ldcg(parent + t) | (__ldcg(s.fac + t) == 1.0f ? 0u : kOdd));
    bool more = true;
    while (__syncthreads_or(more)) {  // any ancestor another thread has moved up meanwhile is one too
        more = false;
        for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
            const unsigned a = get(t), q = a & ~kOdd;
            if ((int)q < first) continue;
            put(t, get((int)q - first) | (a & kOdd));
            more = true;
        }
    }
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
        const int i = first + t;
        bool plain = !(get(t) & kOdd);
        int root = (int)(get(t) & ~kOdd), hops = 0;
        if (!plain)
            for (root = i; root >= first; ++hops) root = up(root);
        float* out = s.T + 16 * (long)i;
        const float* in = s.T + 16 * (long)root;
        for (int e = 0; e < 16; ++e) {
            float v = in[e];
            if (plain) {
                v = 0.f + v * 1.0f;
            } else {
                for (int h = hops - 1; h >= 0; --h) {  // the node h hops above i
                    int a = i;
                    for (int q = 0; q < h; ++q) a = up(a);
                    v = 0.f + v * __ldcg(s.fac + (a - first));
                }
            }
            out[e] = v;
        }
    }
}

static size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

static size_t graph_cell_bytes() {  // counts of both grids (cleared together), then the per-cell arrays
    return al((size_t)kGridMaxCells * 4) * 13 + al((size_t)kSmallCells * 32 * 2);
}

size_t build_graph_ws(long mesh_max) {
    return 2 * al(mesh_max * 4) + al(mesh_max * sizeof(float4)) + al((mesh_max / 32 + 1) * 4) +
           graph_cell_bytes() + al((size_t)kGridMaxCells * kGridSlots * 4) + al(sizeof(Grid)) + al(sizeof(GraphCounters)) + 1024;
}

int build_graph_impl(float* nodes, float* radii, float* T, int* n_nodes, int cap, const float* mesh,
                     const unsigned* mesh_count, long mesh_max, float r, void* ws, size_t ws_bytes, int* error,
                     cudaStream_t st) {
    if (ws_bytes < build_graph_ws(mesh_max) || !ws) return AFX_ERR_WORKSPACE;
    char* p = static_cast<char*>(ws);
    auto take = [&](size_t n) {
        char* q = p;
        p += al(n);
        return q;
    };
    const size_t C = kGridMaxCells;
    GraphState s;
    s.nodes = nodes;
    s.radii = radii;
    s.T = T;
    s.n_nodes = n_nodes;
    s.cap = cap;
    s.mesh = mesh;
    s.mesh_count = mesh_count;
    s.mesh_max = mesh_max;
    s.r = r;
    s.r2 = r * r;
    while (sqrtf(s.r2) < r) s.r2 = std::nextafterf(s.r2, FLT_MAX);
    for (float d; s.r2 > 0.f && !(sqrtf(d = std::nextafterf(s.r2, 0.f)) < r);) s.r2 = d;
    // counters and both grids' counts side by side: one clear
    s.k = (GraphCounters*)take(sizeof(GraphCounters));
    s.g.cnt = (int*)take(C * 4);
    s.ccnt = (unsigned*)take(C * 4);
    const size_t clear = (size_t)(p - reinterpret_cast<char*>(s.k));
    s.cid = (unsigned*)take(C * 4);
    s.gcell = (unsigned*)take(C * 4);
    s.cstart = (unsigned*)take(C * 4);
    s.ccount = (unsigned*)take(C * 4);
    s.cmin = (unsigned*)take(C * 4);
    s.cblock = (unsigned*)take(C * 4);
    s.cnear = (unsigned*)take(C * 4);
    s.cpos = (float4*)take(C * sizeof(float4));
    s.nbr = (unsigned short*)take((size_t)kSmallCells * 32 * 2);
    s.g.slots = (int*)take(C * kGridSlots * 4);
    // the rounds of large graphs use the room of the node grid, which is not needed any more by then
    s.cwork = reinterpret_cast<unsigned*>(s.g.cnt);
    s.cpick = reinterpret_cast<float4*>(s.g.slots);
    static_assert(kGridSlots * sizeof(int) >= kNearMax * sizeof(float4), "they fit");
    s.pcell = (unsigned*)take(mesh_max * 4);
    s.prank = (unsigned*)take(mesh_max * 4);
    s.sorted = (float4*)take(mesh_max * sizeof(float4));
    s.picked = (unsigned*)take((mesh_max / 32 + 1) * 4);
    s.fac = reinterpret_cast<float*>(s.pcell);  // the buckets are not needed once the rounds are over
    Grid* gdev = (Grid*)take(sizeof(Grid));
    s.error = error;
    static ContextOnce once;
    const int rc = once_per_context(once, [](int) {
        return note_cuda_error(
            cudaFuncSetAttribute(graph_greedy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGreedySmem));
    });
    if (rc) return rc;
    AFX_CUDA(cudaMemsetAsync(s.k, 0, clear, st));
    graph_bbox_kernel<<<64, 1024, 0, st>>>(s, gdev);
    AFX_LAUNCH_CHECK();
    graph_candidates_kernel<<<grid_for(mesh_max, 256), 256, 0, st>>>(s, gdev);
    AFX_LAUNCH_CHECK();
    graph_bucket_kernel<<<grid_for(mesh_max, 256), 256, 0, st>>>(s, gdev);
    AFX_LAUNCH_CHECK();
    graph_greedy_kernel<<<1, kGreedyThreads, kGreedySmem, st>>>(s, gdev);
    AFX_LAUNCH_CHECK();
    graph_transforms_kernel<<<152, 256, 0, st>>>(s);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// ------------------------------------------------------------------------------------
// KNN (getKnnData<K>): the K[+1] nodes first by (nanoflann squared distance, node index).
// ------------------------------------------------------------------------------------
//
// Searches, by what the call brings:
//   few queries (kKnnFewQueries, as when the nodes are the queries): a warp per query.  Each lane finds its
//   smallest distance; the KK-th smallest of those bounds the KK-th of all, so a second pass
//   collects few candidates, which are then ranked;
//   many queries: a thread per query with its best KK in registers.  Every CTA sorts the nodes by x into shared
//   memory (bins: about 3 us), and a warp goes outwards from the x range of its 32 queries until the
//   gap exceeds every lane's KK-th distance.  Point clouds come sorted by x, so that range is narrow;
//   few nodes, a shape whose windows would be wide, coordinates that are not finite, or warps whose queries are in no
//   order: all nodes in index order, from shared memory;
//   more nodes than fit there: the same, as many at a time as fit.
// Bound: instructions, about 15 per distance and 25 per insertion, and below some thousand queries the latency of
// building and of one query.  In the 512^3 sequence (1,300 nodes): 330,000 points, K = 4, 83 -> 16 us; the nodes
// among themselves, K = 8, 99 -> 8 us; in the 256^3 sequence (170 nodes) 10.2 -> 8.3 and 15.4 -> 4.2 us (before:
// every thread walked all nodes).
// kKnnFewQueries: a warp per query takes 8.4, 12.7 and 31 us for 2,000 queries and 170, 1,300 and 5,000 nodes of
// a sphere, all nodes by a thread 12.7, 56 and 189; 10, 25 and 75 us for 8,000 (12.6, 56, 188, and a window 15, 35, 60),
// 31, 101 and 328 us for 40,000 (14.6, 66, 216, and a window 17, 36, 62).
// More nodes than fit, 20,000 and K = 4: 570 us for 20,000 queries, 780 for 60,000 and 2.57 ms for 300,000 (the queries in
// CTAs of 128, or of 1024 one after the other, and 1,024 nodes at a time: 770, 910 and 2.97 ms, and 1.28, 1.28 and 2.54 ms).
// kKnnWindowShare: 300 nodes, K = 4: on a sphere (0.39 by the estimate) a window takes 21 us for 16,000 queries and all
// nodes 17; on a tube along x (0.15) 13 and 17.

constexpr int kKnnThreads = 1024;
constexpr int kKnnWarps = kKnnThreads / 32;
constexpr long kKnnFewQueries = 8192;
constexpr int kKnnCandidates = 96;     // per query of the first search
constexpr int kKnnBins = 1024;
constexpr int kKnnScanNodes = 128;       // fewer are not worth sorting
constexpr float kKnnWindowShare = 0.35f;  // of the nodes: windows not narrower are not worth their bookkeeping
static_assert(kKnnBins == kKnnThreads, "a thread scans a bin");
constexpr size_t kKnnRoom = 220 * 1024;
constexpr size_t kKnnSide = (size_t)kKnnWarps * kKnnCandidates * 8;  // candidates, or the bins
constexpr int kKnnMaxNodes = (int)((kKnnRoom - kKnnSide) / sizeof(float4));

template <int KK>
struct KnnList {
    float d[KK];
    int i[KK];
    AFX_D void clear() {
#pragma unroll
        for (int s = 0; s < KK; ++s) {
            d[s] = INFINITY;
            i[s] = 0x7fffffff;  // empty: after every node at any distance
        }
    }
    // In any order of calls, for distances that are not NaN.
    AFX_D void offer(float nd, int ni) {
        if (!(nd <= d[KK - 1])) return;
        if (nd == d[KK - 1] && ni > i[KK - 1]) return;
        d[KK - 1] = nd;
        i[KK - 1] = ni;
#pragma unroll
        for (int p = KK - 1; p > 0; --p) {
            const bool up = d[p] < d[p - 1] || (d[p] == d[p - 1] && i[p] < i[p - 1]);
            const float dp = d[p], dq = d[p - 1];
            const int ip = i[p], iq = i[p - 1];
            d[p] = up ? dq : dp;
            d[p - 1] = up ? dp : dq;
            i[p] = up ? iq : ip;
            i[p - 1] = up ? ip : iq;
        }
    }
    // In ascending index order (any distances): a candidate that beats the last entry, or fills an empty
    // slot, replaces it and passes strictly larger distances, so equal ones keep the earlier index.
    AFX_D void offer_next(float nd, int ni) {
        if (i[KK - 1] != 0x7fffffff && !(nd < d[KK - 1])) return;
        d[KK - 1] = nd;
        i[KK - 1] = ni;
#pragma unroll
        for (int p = KK - 1; p > 0; --p) {
            if (i[p - 1] == 0x7fffffff || d[p] < d[p - 1]) {
                const float td = d[p];
                d[p] = d[p - 1];
                d[p - 1] = td;
                const int ti = i[p];
                i[p] = i[p - 1];
                i[p - 1] = ti;
            }
        }
    }
    AFX_D void store(uint32_t* idx, float* dist, long q, int k, int excl) const {
#pragma unroll
        for (int s = 0; s < KK; ++s) {
            const int o = s - excl;
            if (o < 0 || o >= k) continue;
            const bool have = i[s] != 0x7fffffff;
            idx[q * k + o] = have ? (uint32_t)i[s] : AFX_INVALID_INDEX;
            dist[q * k + o] = have ? sqrtf(d[s]) : FLT_MAX;
        }
    }
};

// One query by a warp over nodes in index order (`p`, in shared or global memory).
template <int KK>
AFX_D void knn_by_warp(const float (&q)[3], const float* p, int n, unsigned long long* cand, uint32_t* idx, float* dist, long i,
                       int k, int excl) {
    const int lane = threadIdx.x & 31;
    float least = INFINITY;
    bool nan = false;
#pragma unroll 4
    for (int j = lane; j < n; j += 32) {
        const float d = l2sq_nanoflann(q, p + 3 * j);
        nan |= d != d;
        least = fminf(least, d);
    }
    int rank = 0;
#pragma unroll 8
    for (int o = 0; o < 32; ++o) {
        const float v = __shfl_sync(0xffffffffu, least, o);
        rank += v < least || (v == least && o < lane);
    }
    const float bound = __shfl_sync(0xffffffffu, least, __ffs(__ballot_sync(0xffffffffu, rank == KK - 1)) - 1);
    int have = 0;
    if (!__any_sync(0xffffffffu, nan))
        for (int j0 = 0; j0 < n && have <= kKnnCandidates; j0 += 32) {
            const int j = j0 + lane;
            const float d = j < n ? l2sq_nanoflann(q, p + 3 * j) : INFINITY;
            const bool in = j < n && d <= bound;
            const unsigned bal = __ballot_sync(0xffffffffu, in);
            const int at = have + __popc(bal & ((1u << lane) - 1u));
            if (in && at < kKnnCandidates) cand[at] = (unsigned long long)__float_as_uint(d) << 32 | (unsigned)j;
            have += __popc(bal);
        }
    else
        have = kKnnCandidates + 1;
    if (have > kKnnCandidates) {  // distances that are not numbers, or a crowd of equal ones: in index order
        if (lane == 0) {
            KnnList<KK> best;
            best.clear();
            for (int j = 0; j < n; ++j) best.offer_next(l2sq_nanoflann(q, p + 3 * j), j);
            best.store(idx, dist, i, k, excl);
        }
        __syncwarp();
        return;
    }
    __syncwarp();
    for (int c = lane; c < have; c += 32) {
        const unsigned long long key = cand[c];
        int r = 0;
#pragma unroll 4
        for (int o = 0; o < have; ++o) r += cand[o] < key;
        r -= excl;
        if (r >= 0 && r < k) {
            idx[i * k + r] = (uint32_t)key;
            dist[i * k + r] = sqrtf(__uint_as_float((unsigned)(key >> 32)));
        }
    }
    for (int r = max(have - excl, 0) + lane; r < k; r += 32) {
        idx[i * k + r] = AFX_INVALID_INDEX;
        dist[i * k + r] = FLT_MAX;
    }
    __syncwarp();
}

AFX_D unsigned knn_key(float v) {  // ascending
    const unsigned b = __float_as_uint(v);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}
AFX_D float knn_unkey(unsigned k) { return __uint_as_float(k & 0x80000000u ? k & 0x7fffffffu : ~k); }

// The nodes by ascending bin of x, with their indices (the whole CTA; n <= kKnnMaxNodes).  Returns the x that a node
// may lie before another one further on by, or a negative value where nothing was sorted: a coordinate is not finite,
// or a window would not be much narrower than all nodes.
template <int KK>
AFX_D float knn_sort_x(const float* __restrict__ nodes, int n, float4* list, unsigned* bins, float& x0, float& scale) {
    __shared__ unsigned s_min[3], s_max[3], s_bad, s_sum[kKnnWarps];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid < 3) {
        s_min[tid] = 0xffffffffu;
        s_max[tid] = 0u;
    }
    if (tid == 3) s_bad = 0u;
    bins[tid] = 0u;
    __syncthreads();
    unsigned lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
    bool bad = false;
    for (int j = tid; j < n; j += kKnnThreads)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float v = nodes[3 * j + c];
            bad |= !isfinite(v);
            lo[c] = min(lo[c], knn_key(v));
            hi[c] = max(hi[c], knn_key(v));
        }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        lo[c] = __reduce_min_sync(0xffffffffu, lo[c]);
        hi[c] = __reduce_max_sync(0xffffffffu, hi[c]);
        if (lane == 0 && lo[c] <= hi[c]) {
            atomicMin(s_min + c, lo[c]);
            atomicMax(s_max + c, hi[c]);
        }
    }
    if (bad) s_bad = 1u;
    __syncthreads();
    x0 = knn_unkey(s_min[0]);
    const float ext = knn_unkey(s_max[0]) - x0, ey = knn_unkey(s_max[1]) - knn_unkey(s_min[1]),
                ez = knn_unkey(s_max[2]) - knn_unkey(s_min[2]);
    scale = ext > 0.f ? (kKnnBins - 0.5f) / ext : 0.f;
    if (s_bad || !isfinite(ext) || !isfinite(scale)) return -1.f;  // the same in every thread, as what follows
    // The distance of the KK-th node, if they lie evenly on a surface of half the bounding box's: a window is about
    // three of it wide (the farthest of 32 queries sets it).
    const float reach = sqrtf(0.41f * KK * (ext * ey + ey * ez + ext * ez) / (float)n);
    if (!(3.f * reach < kKnnWindowShare * ext)) return -1.f;
    auto bin = [&](float x) { return min(kKnnBins - 1, (int)((x - x0) * scale)); };
    for (int j = tid; j < n; j += kKnnThreads) atomicAdd(bins + bin(nodes[3 * j]), 1u);
    __syncthreads();
    const unsigned v = bins[tid];
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_sum[w] = x;
    __syncthreads();
    unsigned t = s_sum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
    }
    t = __shfl_sync(0xffffffffu, t, w > 0 ? w - 1 : 0);
    bins[tid] = x - v + (w > 0 ? t : 0u);
    __syncthreads();
    for (int j = tid; j < n; j += kKnnThreads) {
        const float p[3] = {nodes[3 * j], nodes[3 * j + 1], nodes[3 * j + 2]};
        list[atomicAdd(bins + bin(p[0]), 1u)] = make_float4(p[0], p[1], p[2], __int_as_float(j));
    }
    __syncthreads();
    return ext * (1.02f / kKnnBins);
}

// The nodes of a warp's 32 queries (those with `on`).  Bin b's nodes end at bins[b]; `copy`: the nodes in
// index order in shared memory, if they fit.
template <int KK>
AFX_D void knn_window(const float (&q)[3], bool on, const float4* list, const float* copy, const float* nodes, int n,
                      const unsigned* bins, float x0, float scale, float slack, KnnList<KK>& best) {
    const unsigned key = knn_key(q[0]);
    const float qlo = knn_unkey(__reduce_min_sync(0xffffffffu, on ? key : 0xffffffffu));
    const float qhi = knn_unkey(__reduce_max_sync(0xffffffffu, on ? key : 0u));
    auto look = [&](int a, int b) {
#pragma unroll 4
        for (int j = a; j < b; ++j) {
            const float4 v = list[j];
            const float p[3] = {v.x, v.y, v.z};
            best.offer(l2sq_nanoflann(q, p), __float_as_int(v.w));
        }
    };
    auto bin = [&](float x) { return (int)fminf(fmaxf((x - x0) * scale, 0.f), (float)(kKnnBins - 1)); };
    const int b0 = bin(qlo), b1 = bin(qhi);
    int left = b0 > 0 ? (int)bins[b0 - 1] : 0, right = (int)bins[b1];
    if (right - left > kKnnWindowShare * n) {  // queries in no order: all nodes, in theirs
        if (copy) {
#pragma unroll 4
            for (int j = 0; j < n; ++j) best.offer_next(l2sq_nanoflann(q, copy + 3 * j), j);
        } else {
#pragma unroll 4
            for (int j = 0; j < n; ++j) best.offer_next(l2sq_nanoflann(q, nodes + 3 * j), j);
        }
        return;
    }
    look(left, right);
    constexpr int kStep = 8;
    bool more_left = left > 0, more_right = right < n;
    while (more_left || more_right) {
        const float worst = __uint_as_float(__reduce_max_sync(0xffffffffu, on ? __float_as_uint(best.d[KK - 1]) : 0u));
        if (more_right) {
            const float gap = list[right].x - slack - qhi;
            if (gap > 0.f && gap * gap * 0.9999f > worst) {
                more_right = false;
            } else {
                const int to = min(right + kStep, n);
                look(right, to);
                right = to;
                more_right = right < n;
            }
        }
        if (more_left) {
            const float gap = qlo - slack - list[left - 1].x;
            if (gap > 0.f && gap * gap * 0.9999f > worst) {
                more_left = false;
            } else {
                const int to = max(left - kStep, 0);
                look(to, left);
                left = to;
                more_left = left > 0;
            }
        }
    }
}

template <int KK>
__global__ void __launch_bounds__(kKnnThreads, 1) knn_kernel(uint32_t* idx, float* dist, const float* __restrict__ nodes,
                                                             const int* n_nodes, int n_max, const float* __restrict__ pts,
                                                             const unsigned* count, long m_max, int k, int excl, size_t room) {
    extern __shared__ float4 knn_smem[];
    const int n = min(*n_nodes, n_max);
    const long m = count ? min((long)*count, m_max) : m_max;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long first = (long)w * gridDim.x + blockIdx.x, step = (long)gridDim.x * kKnnWarps;  // of warps, over all SMs first
    if ((long)blockIdx.x >= m) return;
    float4* const list = knn_smem + kKnnSide / sizeof(float4);
    if (m <= kKnnFewQueries) {
        unsigned long long* cand = reinterpret_cast<unsigned long long*>(knn_smem) + w * kKnnCandidates;
        const float* p = nodes;
        if (n <= kKnnMaxNodes) {
            float* s = reinterpret_cast<float*>(list);
            for (int t = threadIdx.x; t < 3 * n; t += kKnnThreads) s[t] = nodes[t];
            __syncthreads();
            p = s;
        }
        for (long i = first; i < m; i += step) {
            const float q[3] = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
            knn_by_warp<KK>(q, p, n, cand, idx, dist, i, k, excl);
        }
        return;
    }
    unsigned* const bins = reinterpret_cast<unsigned*>(knn_smem);
    float x0 = 0.f, scale = 0.f;
    bool scan = n <= kKnnScanNodes;
    const float slack = !scan && n <= kKnnMaxNodes ? knn_sort_x<KK>(nodes, n, list, bins, x0, scale) : -1.f;
    scan = scan || (n <= kKnnMaxNodes && slack < 0.f);
    if (scan || slack >= 0.f) {
        // in index order: the scan's nodes, or those of warps that leave the window (beside the sorted ones if there is room)
        float* const copy = reinterpret_cast<float*>(list + n);
        const bool copied = !scan && 28 * (size_t)n <= room;
        if (scan) {
            for (int j = threadIdx.x; j < n; j += kKnnThreads)
                list[j] = make_float4(nodes[3 * j], nodes[3 * j + 1], nodes[3 * j + 2], 0.f);
        } else if (copied) {
            for (int t = threadIdx.x; t < 3 * n; t += kKnnThreads) copy[t] = nodes[t];
        }
        __syncthreads();
        for (long t = first; t * 32 < m; t += step) {
            const long i = t * 32 + lane;
            float q[3] = {0.f, 0.f, 0.f};
            if (i < m)
#pragma unroll
                for (int c = 0; c < 3; ++c) q[c] = pts[3 * i + c];
            const bool on = i < m && isfinite(q[0]) && isfinite(q[1]) && isfinite(q[2]);
            KnnList<KK> best;
            best.clear();
            if (scan) {
#pragma unroll 4
                for (int j = 0; j < n; ++j) {
                    const float4 v = list[j];
                    const float p[3] = {v.x, v.y, v.z};
                    best.offer_next(l2sq_nanoflann(q, p), j);
                }
            } else if (__any_sync(0xffffffffu, on)) {
                knn_window<KK>(q, on, list, copied ? copy : nullptr, nodes, n, bins, x0, scale, slack, best);
            }
            if (!scan && i < m && !on) {
                best.clear();
                for (int j = 0; j < n; ++j) best.offer_next(l2sq_nanoflann(q, nodes + 3 * j), j);
            }
            if (i < m) best.store(idx, dist, i, k, excl);
            __syncwarp();
        }
        return;
    }
    // (the queries dealt to warps as above; every warp of a CTA loads nodes for those that have some)
    for (long t0 = blockIdx.x; t0 * 32 < m; t0 += step) {
        const long i = (t0 + (long)w * gridDim.x) * 32 + lane;
        const bool any = i - lane < m;
        float q[3] = {0.f, 0.f, 0.f};
        if (i < m)
#pragma unroll
            for (int c = 0; c < 3; ++c) q[c] = pts[3 * i + c];
        KnnList<KK> best;
        best.clear();
        for (int base = 0; base < n; base += kKnnMaxNodes) {
            const int nt = min(kKnnMaxNodes, n - base);
            __syncthreads();
            for (int j = threadIdx.x; j < nt; j += kKnnThreads) {
                const float* p = nodes + 3 * ((long)base + j);
                list[j] = make_float4(p[0], p[1], p[2], 0.f);
            }
            __syncthreads();
            if (any) {
#pragma unroll 8
                for (int j = 0; j < nt; ++j) {
                    const float4 v = list[j];
                    const float p[3] = {v.x, v.y, v.z};
                    best.offer_next(l2sq_nanoflann(q, p), base + j);
                }
            }
        }
        if (i < m) best.store(idx, dist, i, k, excl);
    }
}

template <int KK>
static int launch_knn(uint32_t* idx, float* dist, const float* nodes, const int* n_nodes, int n_max, const float* pts,
                      const unsigned* count, long m_max, int k, int excl, cudaStream_t st) {
    static ContextOnce once;
    const int rc = once_per_context(once, [](int) {
        return note_cuda_error(
            cudaFuncSetAttribute(knn_kernel<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kKnnRoom));
    });
    if (rc) return rc;
    // for the nodes: sorted, and in index order while both fit
    const size_t most = kKnnRoom - kKnnSide, room = 28 * (size_t)n_max < most ? 28 * (size_t)n_max : most;
    knn_kernel<KK><<<(unsigned)(m_max < 152 ? m_max : 152), kKnnThreads, kKnnSide + room, st>>>(
        idx, dist, nodes, n_nodes, n_max, pts, count, m_max, k, excl, room);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int knn_impl(uint32_t* idx, float* dist, const float* nodes, const int* n_nodes, int n_max, const float* pts,
             const unsigned* count, long m_max, int k, int excl, cudaStream_t st) {
    if (m_max <= 0) return AFX_OK;
    const int e = excl ? 1 : 0;
    const int kk = k + e;
#define AFX_KNN(KK) return launch_knn<KK>(idx, dist, nodes, n_nodes, n_max, pts, count, m_max, k, e, st)
    switch (kk) {
        case 1: AFX_KNN(1);
        case 2: AFX_KNN(2);
        case 3: AFX_KNN(3);
        case 4: AFX_KNN(4);
        case 5: AFX_KNN(5);
        case 6: AFX_KNN(6);
        case 7: AFX_KNN(7);
        case 8: AFX_KNN(8);
        case 9: AFX_KNN(9);
        default:
            if (kk <= 12) {
                AFX_KNN(12);
            } else if (kk <= 17) {
                AFX_KNN(17);
            } else {
                return AFX_ERR_UNSUPPORTED;
            }
    }
#undef AFX_KNN
}

__global__ void filter_disconnected_kernel(uint32_t* idx, float* dist, const int* n_nodes, int n_max, int k,
                                           const float* radii) {
    const int n = min(*n_nodes, n_max);
    AFX_GRID_STRIDE(t, (long)n * k) {
        const long i = t / k;
        const uint32_t nb = idx[t];
        if (nb >= (uint32_t)n) continue;
        if (dist[t] <= radii[i] * 1.3f) continue;
        idx[t] = AFX_INVALID_INDEX;
        dist[t] = FLT_MAX;
    }
}

// computeWarpWeightsKernel (src/VertexManipulation.cu:105-132)
// Weights of point i over its k nearest nodes; ws: its k weights.
AFX_D void warp_weights_of(const float* radii, const uint32_t* idx, const float* dist, int k, int n, float* ws) {
    float sum = 0.f;
    for (int j = 0; j < k; ++j) {
        const uint32_t nb = idx[j];
        float wj = 0.f;
        if (nb < (uint32_t)n) {
            const float r = radii[nb], d = dist[j];
            wj = (d >= r) ? 0.f : afx_expf(-(d * d) / (2.0f * (r * r)));
        }
        ws[j] = wj;
        sum = sum + wj;
    }
    for (int j = 0; j < k; ++j) ws[j] = (sum != 0.f) ? ws[j] / sum : ws[j];
}

__global__ void warp_weights_kernel(float* w, const float* radii, const uint32_t* idx, const float* dist,
                                    const unsigned* count, long m_max, int k, const int* n_nodes) {
    const long m = count ? min((long)*count, m_max) : m_max;
    const int n = *n_nodes;
    AFX_GRID_STRIDE(i, m) {
        float ws[17];
        warp_weights_of(radii, idx + i * k, dist + i * k, k, n, ws);
        for (int j = 0; j < k; ++j) w[i * k + j] = ws[j];
    }
}

// What follows the two searches of a frame, in one launch: the points' weights, the graph's edges without those
// too long (filter_disconnected_kernel), and how many entries and edges each node gets (the Gauss-Newton
// stage's lists; both counters start at zero).
__global__ void graph_weights_kernel(GraphWeightArgs a) {
    const long m = min((long)*a.count, a.m_max);
    const int n = min(*a.n_nodes, a.n_max);
    AFX_GRID_STRIDE(i, m) {
        float ws[17];
        warp_weights_of(a.radii, a.idx + i * a.k, a.dist + i * a.k, a.k, *a.n_nodes, ws);
        for (int j = 0; j < a.k; ++j) {
            a.w[i * a.k + j] = ws[j];
            const uint32_t node = a.idx[i * a.k + j];
            if (ws[j] != 0.f && node < (uint32_t)n) atomicAdd(a.entries + node, 1u);
        }
    }
    AFX_GRID_STRIDE(t, (long)n * a.kreg) {
        const uint32_t nb = a.gidx[t];
        if (nb >= (uint32_t)n) continue;
        if (a.gdist[t] <= a.radii[t / a.kreg] * 1.3f) {
            atomicAdd(a.edges + nb, 1u);
        } else {
            a.gidx[t] = AFX_INVALID_INDEX;
            a.gdist[t] = FLT_MAX;
        }
    }
}

int graph_weights_impl(const GraphWeightArgs& a, cudaStream_t st) {
    if (a.k > 17) return AFX_ERR_UNSUPPORTED;
    const long items = a.m_max > (long)a.n_max * a.kreg ? a.m_max : (long)a.n_max * a.kreg;
    if (items <= 0) return AFX_OK;
    graph_weights_kernel<<<grid_for(items, 256), 256, 0, st>>>(a);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// warpKernel (src/ComputeCorrespondence.cu:5-30)
__global__ void warp_kernel(float* out, const float* __restrict__ pts, const float* __restrict__ T,
                            const uint32_t* __restrict__ idx, const float* __restrict__ w, const unsigned* count,
                            long m_max, int k) {
    long m = count ? min((long)*count, m_max) : m_max;
    AFX_GRID_STRIDE(i, m) {
        float p[3] = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
        bool zero = true;
        for (int j = 0; j < k; ++j)
            if (!(fabsf(w[i * k + j]) <= 1e-5f)) zero = false;
        float acc[3] = {p[0], p[1], p[2]};
        if (!zero) {
            acc[0] = acc[1] = acc[2] = 0.f;
            for (int j = 0; j < k; ++j) {
                uint32_t nb = idx[i * k + j];
                if (nb == AFX_INVALID_INDEX) continue;
                float o[3];
                mat4_point(T + 16 * (long)nb, p, o);
                float wj = w[i * k + j];
                acc[0] = acc[0] + wj * o[0];
                acc[1] = acc[1] + wj * o[1];
                acc[2] = acc[2] + wj * o[2];
            }
        }
        out[3 * i] = acc[0];
        out[3 * i + 1] = acc[1];
        out[3 * i + 2] = acc[2];
    }
}

int warp_weights_impl(float* w, const float* radii, const uint32_t* idx, const float* dist, const unsigned* count,
                      long m_max, int k, const int* n_nodes, cudaStream_t st) {
    if (m_max <= 0) return AFX_OK;
    if (k > 17) return AFX_ERR_UNSUPPORTED;
    warp_weights_kernel<<<grid_for(m_max, 256), 256, 0, st>>>(w, radii, idx, dist, count, m_max, k, n_nodes);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// The same points moved by the dual-quaternion blend of their nodes (afx_dqb.cuh).
__global__ void warp_dqb_kernel(float* out, const float* __restrict__ pts, const float* __restrict__ T,
                                const uint32_t* __restrict__ idx, const float* __restrict__ w, const unsigned* count,
                                long m_max, int k) {
    long m = count ? min((long)*count, m_max) : m_max;
    AFX_GRID_STRIDE(i, m) {
        const float p[3] = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
        float o[3];
        dq_blend_point(T, idx + i * k, w + i * k, k, AFX_INVALID_INDEX, p, o);
        out[3 * i] = o[0];
        out[3 * i + 1] = o[1];
        out[3 * i + 2] = o[2];
    }
}

int warp_impl(float* out, const float* pts, const float* T, const uint32_t* idx, const float* w, const unsigned* count,
              long m_max, int k, cudaStream_t st, int blend) {
    if (m_max <= 0) return AFX_OK;
    if (blend == AFX_BLEND_DQB) {
        warp_dqb_kernel<<<grid_for(m_max, 256), 256, 0, st>>>(out, pts, T, idx, w, count, m_max, k);
        AFX_LAUNCH_CHECK();
        return AFX_OK;
    }
    warp_kernel<<<grid_for(m_max, 256), 256, 0, st>>>(out, pts, T, idx, w, count, m_max, k);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// ------------------------------------------------------------------------------------
// Correspondences (correspondencePairsKernel, src/ComputeCorrespondence.cu:45-81),
// compacted in vertex order.
// ------------------------------------------------------------------------------------

struct CorrArgs {
    const float* warped;
    const unsigned* count;
    long m_max;
    Intrinsics K;
    const float* depth;
    int rows, cols;
    const float* frame;
    float thresh;
};

AFX_D int corr_pixel(const CorrArgs& a, long i) {
    const float* v = a.warped + 3 * i;
    float y0 = v[1] / v[2];
    float x0 = v[0] / v[2];
    int y = f2i(y0 * a.K.fy + a.K.cy);
    int x = f2i(x0 * a.K.fx + a.K.cx);
    if (y < 0 || x < 0 || y >= a.rows || x >= a.cols) return -1;
    long px = (long)y * a.cols + x;
    const float* f = a.frame + 3 * px;
    float d[3] = {f[0] - v[0], f[1] - v[1], f[2] - v[2]};
    if (norm3(d) > a.thresh) return -1;
    if (!(a.depth[px] > 1.e-4f)) return -1;
    return (int)px;
}

// Pixels of the vertices, and how many of each tile of 256 have one.
constexpr int kCorrTile = 256;

__global__ void __launch_bounds__(kCorrTile) corr_pixel_kernel(CorrArgs a, int* pix, unsigned* sums) {
    const long m = a.count ? min((long)*a.count, a.m_max) : a.m_max;
    for (long tile = blockIdx.x; tile * kCorrTile < m; tile += gridDim.x) {
        const long i = tile * kCorrTile + threadIdx.x;
        const int px = i < m ? corr_pixel(a, i) : -1;
        if (i < m) pix[i] = px;
        const int n = __syncthreads_count(px >= 0);
        if (threadIdx.x == 0) sums[tile] = (unsigned)n;
    }
}

// The pairs in vertex order: a CTA adds up the tiles before its own (a few hundred numbers) instead of
// waiting for three launches of a prefix sum.
__global__ void __launch_bounds__(kCorrTile) corr_scatter_kernel(CorrArgs a, const int* pix, const unsigned* sums, int* corr,
                                                                 unsigned* corr_count, long cap, int* corr_of_vertex) {
    __shared__ unsigned s_before[2][kCorrTile / 32], s_have[2][kCorrTile / 32];
    const long m = a.count ? min((long)*a.count, a.m_max) : a.m_max;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (m <= 0 && blockIdx.x == 0 && threadIdx.x == 0) *corr_count = 0u;
    unsigned base = 0;
    long done = 0;
    int par = 0;
    for (long tile = blockIdx.x; tile * kCorrTile < m; tile += gridDim.x, par ^= 1) {
        unsigned v = 0;
        for (long t = done + threadIdx.x; t < tile; t += kCorrTile) v += sums[t];
        done = tile;
        v = warp_sum(v);
        const long i = tile * kCorrTile + threadIdx.x;
        const int px = i < m ? pix[i] : -1;
        const unsigned bal = __ballot_sync(0xffffffffu, px >= 0);
        if (lane == 0) {
            s_before[par][w] = v;
            s_have[par][w] = (unsigned)__popc(bal);
        }
        __syncthreads();  // the arrays alternate: the next tile's are written while these are read
        unsigned at = 0, all = 0;
#pragma unroll
        for (int q = 0; q < kCorrTile / 32; ++q) {
            base += s_before[par][q];
            if (q < w) at += s_have[par][q];
            all += s_have[par][q];
        }
        if (px >= 0) {
            const unsigned p = base + at + (unsigned)__popc(bal & ((1u << lane) - 1u));
            if (p < cap) {
                corr[2 * (long)p] = (int)i;
                corr[2 * (long)p + 1] = px;
            }
            if (corr_of_vertex) corr_of_vertex[i] = (int)p;
        } else if (corr_of_vertex && i < m) {
            corr_of_vertex[i] = -1;
        }
        if (threadIdx.x == 0 && (tile + 1) * kCorrTile >= m) *corr_count = base + all;
    }
}

size_t corr_ws(long m_max) { return al(m_max * 4) + al((m_max / kCorrTile + 1) * 4) + 256; }

int correspondences_impl(int* corr, unsigned* corr_count, long cap, const float* warped, const unsigned* count,
                         long m_max, const float* K, const float* depth, int rows, int cols, const float* frame,
                         float thresh, int* corr_of_vertex, void* ws, size_t ws_bytes, cudaStream_t st) {
    if (ws_bytes < corr_ws(m_max) || !ws) return AFX_ERR_WORKSPACE;
    if (m_max <= 0) {
        AFX_CUDA(cudaMemsetAsync(corr_count, 0, 4, st));
        return AFX_OK;
    }
    char* p = static_cast<char*>(ws);
    int* pix = (int*)p;
    p += al(m_max * 4);
    unsigned* sums = (unsigned*)p;
    CorrArgs a;
    a.warped = warped;
    a.count = count;
    a.m_max = m_max;
    a.K = make_intrinsics(K);
    a.depth = depth;
    a.rows = rows;
    a.cols = cols;
    a.frame = frame;
    a.thresh = thresh;
    corr_pixel_kernel<<<grid_for(m_max, kCorrTile), kCorrTile, 0, st>>>(a, pix, sums);
    AFX_LAUNCH_CHECK();
    corr_scatter_kernel<<<grid_for(m_max, kCorrTile), kCorrTile, 0, st>>>(a, pix, sums, corr, corr_count, cap, corr_of_vertex);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// Device scratch of the stand-alone entry points (error word, node count copy): one per host
// thread and device, allocated on the thread's first call and kept for the life of the process,
// so calls from different host threads never share it.
struct CallScratch {
    int error;
    int n;
    unsigned count;
};

static CallScratch* call_scratch() {
    thread_local CallScratch* s[kMaxDevices] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    if (!s[dev]) {
        CallScratch* p = nullptr;
        if (cudaMalloc(&p, sizeof(CallScratch)) != cudaSuccess) return nullptr;
        if (cudaMemset(p, 0, sizeof(CallScratch)) != cudaSuccess) {
            cudaFree(p);
            return nullptr;
        }
        s[dev] = p;
    }
    return s[dev];
}

}  // namespace afx

using namespace afx;

extern "C" {

size_t afx_build_graph_workspace_size(long mesh_max, int node_capacity) {
    (void)node_capacity;
    return build_graph_ws(mesh_max);
}

int afx_build_graph(float* nodes, float* radii, float* transforms, int* n_nodes, int node_capacity, const float* mesh,
                    const unsigned* mesh_count, long mesh_max, int knn, float radius, void* workspace,
                    size_t workspace_bytes, void* stream) {
    if (!nodes || !radii || !transforms || !n_nodes || !mesh || !mesh_count || knn < 1 || node_capacity < 1 ||
        mesh_max < 0 || !(radius > 0.f))
        return AFX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    CallScratch* cs = call_scratch();
    if (!cs) return AFX_ERR_NO_MEMORY;
    AFX_CUDA(cudaMemsetAsync(&cs->error, 0, sizeof(int), st));
    int rc = build_graph_impl(nodes, radii, transforms, n_nodes, node_capacity, mesh, mesh_count, mesh_max, radius,
                              workspace, workspace_bytes, &cs->error, st);
    if (rc) return rc;
    int err = 0;
    AFX_CUDA(cudaMemcpyAsync(&err, &cs->error, sizeof(int), cudaMemcpyDeviceToHost, st));
    AFX_CUDA(cudaStreamSynchronize(st));
    if (err & ERRF_UNSUPPORTED) return AFX_ERR_UNSUPPORTED;
    if (err & ERRF_CAPACITY) return AFX_ERR_CAPACITY;
    return AFX_OK;
}

int afx_knn(uint32_t* idx, float* dist, const float* nodes, const int* n_nodes, int n_nodes_max, const float* points,
            const unsigned* count, long n_points_max, int k, int exclude_closest, void* stream) {
    if (!idx || !dist || !nodes || !n_nodes || !points || k < 1 || n_points_max < 0) return AFX_ERR_INVALID_ARGUMENT;
    return knn_impl(idx, dist, nodes, n_nodes, n_nodes_max, points, count, n_points_max, k, exclude_closest,
                    as_stream(stream));
}

int afx_filter_disconnected(uint32_t* idx, float* dist, const int* n_nodes, int n_nodes_max, int k, const float* radii,
                            void* stream) {
    if (!idx || !dist || !n_nodes || !radii || k < 1) return AFX_ERR_INVALID_ARGUMENT;
    if (n_nodes_max <= 0) return AFX_OK;
    filter_disconnected_kernel<<<grid_for((long)n_nodes_max * k, 256), 256, 0, as_stream(stream)>>>(
        idx, dist, n_nodes, n_nodes_max, k, radii);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_warp_weights(float* weights, const float* radii, const uint32_t* idx, const float* dist, const unsigned* count,
                     long n_points_max, int k, const int* n_nodes, void* stream) {
    if (!weights || !radii || !idx || !dist || !n_nodes || k < 1) return AFX_ERR_INVALID_ARGUMENT;
    return warp_weights_impl(weights, radii, idx, dist, count, n_points_max, k, n_nodes, as_stream(stream));
}

int afx_warp(float* warped, const float* points, const float* transforms, const uint32_t* idx, const float* weights,
             const unsigned* count, long n_points_max, int k, void* stream) {
    if (!warped || !points || !transforms || !idx || !weights || k < 1) return AFX_ERR_INVALID_ARGUMENT;
    return warp_impl(warped, points, transforms, idx, weights, count, n_points_max, k, as_stream(stream));
}

int afx_warp_dqb(float* warped, const float* points, const float* transforms, const uint32_t* idx,
                 const float* weights, const unsigned* count, long n_points_max, int k, void* stream) {
    if (!warped || !points || !transforms || !idx || !weights || k < 1) return AFX_ERR_INVALID_ARGUMENT;
    return warp_impl(warped, points, transforms, idx, weights, count, n_points_max, k, as_stream(stream),
                     AFX_BLEND_DQB);
}

size_t afx_correspondences_workspace_size(long n_points_max) { return corr_ws(n_points_max); }

int afx_correspondences(int* corr, unsigned* corr_count, long capacity, const float* warped, const unsigned* count,
                        long n_points_max, const float K[9], const float* depth, int rows, int cols,
                        const float* frame_vertices, float thresh, void* workspace, size_t workspace_bytes,
                        void* stream) {
    if (!corr || !corr_count || !warped || !K || !depth || !frame_vertices || rows <= 0 || cols <= 0)
        return AFX_ERR_INVALID_ARGUMENT;
    return correspondences_impl(corr, corr_count, capacity, warped, count, n_points_max, K, depth, rows, cols,
                                frame_vertices, thresh, nullptr, workspace, workspace_bytes, as_stream(stream));
}

}  // extern "C"

// ------------------------------------------------------------------------------------
// Correspondence search without any allocation: the same two launches as
// afx_correspondences (pixels with the tiles' counts, scatter), with the scratch in a
// fixed file-scope device array instead of a caller-provided workspace.  Every scratch word
// is written before it is read within one call (a pixel for every live vertex, a count for
// every tile of them), so nothing has to start at zero and nothing is cleared.
// The array is shared by all calls on a device: calls that overlap in time race on it.
// ------------------------------------------------------------------------------------

namespace afx {

constexpr long kCorrStaticMaxPoints = AFX_CORR_STATIC_MAX_POINTS;
// the pixel of each vertex, and the tiles' counts with alignment slack
constexpr size_t kCorrStaticBytes = (size_t)kCorrStaticMaxPoints * 4 + 64 * 1024;

static __device__ __align__(256) unsigned char g_corr_static_scratch[kCorrStaticBytes];

constexpr int kCorrStaticMaxDevices = 64;
static std::mutex g_corr_static_mu;
struct CorrStaticSlot {
    unsigned long long ctx_id = 0;  // context the address belongs to (0: none yet)
    void* ptr = nullptr;
};
static CorrStaticSlot g_corr_static[kCorrStaticMaxDevices];

// Device address of the scratch array in the current device's context.  The lookup
// (cudaGetSymbolAddress, which loads the module into the context if needed and allocates
// nothing) runs on the first call in each context -- once per device unless the device is
// reset -- and its result is kept with the context's identifier, so an address from a
// context that has since been destroyed is never reused.
static int corr_static_scratch(void** out) {
    int dev = 0;
    AFX_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kCorrStaticMaxDevices) return AFX_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_corr_static_mu);
    CorrStaticSlot& slot = g_corr_static[dev];
    const unsigned long long id = current_context_id();
    if (!slot.ptr || id == 0 || id != slot.ctx_id) {
        void* p = nullptr;
        AFX_CUDA(cudaGetSymbolAddress(&p, g_corr_static_scratch));
        slot.ptr = p;
        slot.ctx_id = current_context_id();  // the lookup above made the context current if it was not
    }
    *out = slot.ptr;
    return AFX_OK;
}

}  // namespace afx

extern "C" int afx_correspondences_static(int* corr, unsigned* corr_count, long capacity, const float* warped,
                                          const unsigned* count, long n_points_max, const float K[9],
                                          const float* depth, int rows, int cols, const float* frame_vertices,
                                          float thresh, void* stream) {
    if (!corr || !corr_count || !warped || !K || !depth || !frame_vertices || rows <= 0 || cols <= 0)
        return AFX_ERR_INVALID_ARGUMENT;
    if (n_points_max > kCorrStaticMaxPoints) return AFX_ERR_CAPACITY;
    if (corr_ws(n_points_max) > kCorrStaticBytes) return AFX_ERR_CAPACITY;
    void* scratch = nullptr;
    int rc = corr_static_scratch(&scratch);
    if (rc) return rc;
    return correspondences_impl(corr, corr_count, capacity, warped, count, n_points_max, K, depth, rows, cols,
                                frame_vertices, thresh, nullptr, scratch, kCorrStaticBytes, as_stream(stream));
}
