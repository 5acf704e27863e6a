// afx_gn.cu -- Gauss-Newton for the motion graph: residuals, block-sparse J^T J / J^T r
// assembly and a block-Jacobi preconditioned conjugate-gradient solve.
//
// The reference fills a dense Jacobian ((C + 3 K_reg N) x N Vec6f), lists contributing
// node pairs with atomics, sorts and reduces them with thrust, scatters into a dense
// (6N)^2 matrix and solves it with cuSOLVER LU in FP32 (src/VolumeFusion.cu:454-691,
// src/MotionOptimization.cu).  Here J is never stored: a node's thread block stages the rows of
// the vertices that reference it (ascending vertex order, which is ascending correspondence
// order), and its 6x6 blocks J_a^T J_b, dealt over the warps, are summed in binary32 in a fixed
// order -- depth rows by ascending correspondence, then regularisation rows by ascending row.
// Diagonal blocks without any contribution keep the identity (runInitIdentityKernel).
// J^T J depends only on the canonical geometry, weights and correspondences, so it is
// assembled once per ICP iteration; J^T r is rebuilt every Gauss-Newton iteration.
// The solve is a block-Jacobi PCG in one kernel on one cluster: FP32 block SpMV, dot products in
// triple-binary32, FP64 6x6 block inverses.  Its exchanges between CTAs are bounded waits.
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <new>

#include "afx_dqb.cuh"
#include "afx_gn.h"
#include "afx_host.h"

namespace afx {

AFX_D void grad_rows(const float* p, float G[3][6]) {
    G[0][0] = 0.f;   G[0][1] = p[2];  G[0][2] = -p[1]; G[0][3] = 1.f; G[0][4] = 0.f; G[0][5] = 0.f;
    G[1][0] = -p[2]; G[1][1] = 0.f;   G[1][2] = p[0];  G[1][3] = 0.f; G[1][4] = 1.f; G[1][5] = 0.f;
    G[2][0] = p[1];  G[2][1] = -p[0]; G[2][2] = 0.f;   G[2][3] = 0.f; G[2][4] = 0.f; G[2][5] = 1.f;
}

// Depth-row Jacobian entry block for one slot (fill_J_DepthKernel, src/MotionOptimization.cu:51-60)
AFX_D void jdepth(const float* n, float w, const float G[3][6], float lam, float* J) {
    if (w < 1.e-4f) {
#pragma unroll
        for (int q = 0; q < 6; ++q) J[q] = 0.f;
        return;
    }
    float nw[3] = {n[0] * w, n[1] * w, n[2] * w};
#pragma unroll
    for (int q = 0; q < 6; ++q) J[q] = (nw[0] * G[0][q] + (nw[1] * G[1][q] + nw[2] * G[2][q])) * lam;
}

// ---- per-frame node lists ----
//
// Two sets of lists, both ascending: the (vertex, slot) entries of every node and its incoming
// regularisation edges.  The launches are what these steps cost (a few us each for tens of kB), so offsets,
// fill and sort take one each for the two sets together, and the counts are part of a launch before them
// (graph_weights_kernel in a session, gn_corr_of_vertex_kernel here).

AFX_D void list_counts(const GnArgs& a) {
    const long m = min((long)*a.mesh_count, a.m_max);
    const int n = min(*a.n_nodes, a.n_max);
    AFX_GRID_STRIDE(t, m * a.k) {
        if (a.mw[t] == 0.f) continue;
        const uint32_t node = a.midx[t];
        if (node < (uint32_t)n) atomicAdd(a.b.lcnt + node, 1u);
    }
    AFX_GRID_STRIDE(t, (long)n * a.kreg) {
        const uint32_t nb = a.gidx[t];
        if (nb < (uint32_t)n) atomicAdd(a.b.icnt + nb, 1u);
    }
}

// Exclusive prefix sums over the live nodes, one CTA per set: off[0..n].
__global__ void __launch_bounds__(1024) list_scan_kernel(GnArgs a) {
    __shared__ unsigned ws[32];
    const int n = min(*a.n_nodes, a.n_max);
    const unsigned* cnt = blockIdx.x ? a.b.icnt : a.b.lcnt;
    unsigned* off = blockIdx.x ? a.b.ioff : a.b.loff;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned carry = 0;
    for (int base = 0; base < n; base += 1024) {
        const int i = base + (int)threadIdx.x;
        const unsigned v = i < n ? cnt[i] : 0u;
        unsigned x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[wid] = x;
        __syncthreads();
        unsigned t = ws[lane];  // every warp scans the 32 warp sums for itself
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        const unsigned before = __shfl_sync(0xffffffffu, t, wid > 0 ? wid - 1 : 0);
        if (i < n) off[i] = carry + (wid > 0 ? before : 0u) + x - v;
        carry += __shfl_sync(0xffffffffu, t, 31);
        __syncthreads();
    }
    if (threadIdx.x == 0) off[n] = carry;
}

__global__ void list_fill_kernel(GnArgs a) {
    const long m = min((long)*a.mesh_count, a.m_max);
    const int n = min(*a.n_nodes, a.n_max);
    AFX_GRID_STRIDE(t, m * a.k) {
        if (a.mw[t] == 0.f) continue;
        const uint32_t node = a.midx[t];
        if (node >= (uint32_t)n) continue;
        const unsigned p = a.b.loff[node] + atomicAdd(a.b.lcur + node, 1u);
        a.b.lst[p] = (unsigned)t;
    }
    AFX_GRID_STRIDE(t, (long)n * a.kreg) {
        const uint32_t nb = a.gidx[t];
        if (nb >= (uint32_t)n) continue;
        const unsigned p = a.b.ioff[nb] + atomicAdd(a.b.icur + nb, 1u);
        a.b.ilst[p] = (unsigned)t;
    }
}

// Ascending bitonic steps of one value per lane: partners `from`, from / 2, .. 1 lanes apart.
AFX_D unsigned lane_merge(unsigned x, int from, bool asc) {
    const int lane = threadIdx.x & 31;
    for (int o = from; o > 0; o >>= 1) {
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, o);
        x = (((lane & o) == 0) == asc) ? min(x, y) : max(x, y);
    }
    return x;
}

// Bitonic sort of one list (len <= kSegMax) through shared memory, by the whole CTA.  Partners
// less than 32 apart are lanes of a warp: only the wider steps need a barrier (15 instead of 55
// for 1024 entries).
AFX_D void seg_sort_one(unsigned* lst, int len, unsigned* s) {
    int P = 32;
    while (P < len) P <<= 1;
    __syncthreads();  // the previous list's write-back is done with s
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        unsigned x = i < len ? lst[i] : 0xffffffffu;
        for (int size = 2; size <= 32; size <<= 1) x = lane_merge(x, size >> 1, (i & size) == 0);
        s[i] = x;
    }
    for (int size = 64; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride >= 32; stride >>= 1) {
            __syncthreads();
            for (int pidx = threadIdx.x; pidx < P / 2; pidx += blockDim.x) {
                const int i = 2 * stride * (pidx / stride) + (pidx % stride), j = i + stride;
                const bool asc = (i & size) == 0;
                const unsigned x = s[i], y = s[j];
                if ((y < x) == asc) {
                    s[i] = y;
                    s[j] = x;
                }
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < P; i += blockDim.x) s[i] = lane_merge(s[i], 16, (i & size) == 0);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < len; i += blockDim.x) lst[i] = s[i];
}

// Sort both sets: one CTA per node's entries at a time; the edge lists (about kreg entries) one per
// warp in registers, and by the whole CTA where one is longer than a warp.
__global__ void __launch_bounds__(256) list_sort_kernel(GnArgs a) {
    __shared__ unsigned s[kSegMax];
    const int n = min(*a.n_nodes, a.n_max);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int node = blockIdx.x; node < n; node += gridDim.x) {
        const unsigned o = a.b.loff[node];
        const int len = (int)(a.b.loff[node + 1] - o);
        if (len > kSegMax) {
            if (threadIdx.x == 0) atomicOr(a.error, ERRF_CAPACITY);
            continue;
        }
        if (len > 1) seg_sort_one(a.b.lst + o, len, s);
    }
    for (int base = blockIdx.x * 8; base < n; base += gridDim.x * 8) {
        const int node = base + w;
        if (node < n) {
            const unsigned o = a.b.ioff[node];
            const int len = (int)(a.b.ioff[node + 1] - o);
            if (len > 1 && len <= 32) {
                unsigned x = lane < len ? a.b.ilst[o + lane] : 0xffffffffu;
                for (int size = 2; size <= 32; size <<= 1) x = lane_merge(x, size >> 1, (lane & size) == 0);
                if (lane < len) a.b.ilst[o + lane] = x;
            }
        }
        for (int q = 0; q < 8 && base + q < n; ++q) {
            const unsigned o = a.b.ioff[base + q];
            const int len = (int)(a.b.ioff[base + q + 1] - o);
            if (len > kSegMax) {
                if (threadIdx.x == 0) atomicOr(a.error, ERRF_CAPACITY);
            } else if (len > 32) {
                seg_sort_one(a.b.ilst + o, len, s);
            }
        }
    }
}

// ---- per-ICP assembly ----

AFX_D int find_slot(const int* L, int cnt, int b) {
    int lo = 0, hi = cnt - 1;
    while (lo <= hi) {
        int mid = (lo + hi) >> 1;
        if (L[mid] == b) return mid;
        if (L[mid] < b) lo = mid + 1;
        else hi = mid - 1;
    }
    return -1;
}

// J^T J of one node per CTA: its neighbour list, its diagonal block D_a and its upper blocks
// (a, b > a).
//
// Neighbours: distinct nodes b != a sharing a corresponding vertex with a (both weights non-zero)
// or joined to a by a regularisation edge, as a bitmap in shared memory, so the list is sorted.
//
// Every block entry is a sum in a fixed order: depth rows by ascending node-list entry, then
// regularisation rows by ascending row.  Entries of different blocks are independent, so the rows
// are staged 256 at a time (one per thread, the Jacobian block of every slot formed: jdepth, or
// lam_r * G for a regularisation row) and the blocks are dealt over the CTA: warp 0 sums the
// diagonal, each of the other warps up to five upper blocks at a time, six lanes to a block, one
// row of it per lane in registers.  A group lists the rows of its block first (ballots over the slot
// bytes of 32 rows at a time), so that the loads of four rows are in flight while it sums in order; the
// diagonal takes eight rows at a time.  The bound is the serial sum of the longest lists:
// with one warp per node walking all rows and the upper blocks in shared memory, the graph of the
// 256^3 sequence took 70 us and 16 us for the neighbours, against 15 us for both so (and 20 us, or
// 115 instead of 57 us for 1,500 nodes over 60,000 points, with one row in flight per group).
constexpr int kAsmThreads = 256;
constexpr int kAsmUpWarps = kAsmThreads / 32 - 1;
constexpr int kAsmGroups = 5;
constexpr int kAsmPass = kAsmUpWarps * kAsmGroups;            // upper blocks in registers at a time
constexpr int kAsmPasses = (kMaxNbr + kAsmPass - 1) / kAsmPass;
constexpr unsigned kSlotDiag = 0xfeu, kSlotNone = 0xffu;       // else the number of the upper block

// Floats per staged row: even, so that pairs stay aligned, and not a multiple of four, so that
// rows 32 lanes write spread over the banks (two lanes to a bank).
AFX_HD int asm_stride(int k) {
    const int s = 6 * (k > 3 ? k : 3) + 2;
    return s % 4 == 0 ? s + 2 : s;
}

// Dynamic shared memory: the staged rows (or the neighbour bitmap before them), then a list of
// rows for every group (row << 6 | own slot << 3 | slot).
AFX_HD size_t asm_rows_bytes(int k, int words) {
    const size_t rows = (size_t)kAsmThreads * asm_stride(k) * 4, bits = ((size_t)words * 4 + 7) / 8 * 8;
    return rows > bits ? rows : bits;
}
constexpr size_t kAsmListBytes = (size_t)kAsmPass * kAsmThreads * sizeof(unsigned short);

template <int KM>  // at least k slots per vertex
__global__ void __launch_bounds__(kAsmThreads, KM <= 4 ? 4 : 3) jtj_assemble_kernel(GnArgs a) {
    extern __shared__ __align__(16) float2 asm_dyn[];
    float* const J = reinterpret_cast<float*>(asm_dyn);             // [256][stride]
    unsigned* const bm = reinterpret_cast<unsigned*>(asm_dyn);      // neighbour bitmap, before the rows
    __shared__ int s_L[kMaxNbr];
    __shared__ uint2 s_slot[kAsmThreads];
    __shared__ __align__(8) unsigned char s_own[kAsmThreads];
    __shared__ int s_rows[kAsmThreads / 32];
    __shared__ int s_cnt, s_first, s_touched;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int n = min(*a.n_nodes, a.n_max), k = a.k, stride = asm_stride(k);
    const int g = lane / 6, gi = lane % 6;                  // upper blocks: group and block row
    const int di = lane / 3, dj = (lane % 3) * 2;           // diagonal: lanes 0..17, two entries each
    unsigned short* const lists = reinterpret_cast<unsigned short*>(
        reinterpret_cast<char*>(asm_dyn) + asm_rows_bytes(k, (a.n_max + 31) / 32)) + (w - 1) * kAsmGroups * kAsmThreads;
    for (int node = blockIdx.x; node < n; node += gridDim.x) {
        const int words = (n + 31) / 32;
        for (int i = tid; i < words; i += kAsmThreads) bm[i] = 0u;
        if (tid == 0) s_touched = 0;
        __syncthreads();
        const unsigned o = a.b.loff[node], e = a.b.loff[node + 1];
        const unsigned io = a.b.ioff[node], nin = a.b.ioff[node + 1] - io;
        for (unsigned base = o + tid; base < e; base += 2 * kAsmThreads) {
            const unsigned t1 = base + kAsmThreads;
            const bool two = t1 < e;
            const unsigned ent[2] = {a.b.lst[base], two ? a.b.lst[t1] : 0u};
            long v[2] = {(long)(ent[0] / k), (long)(ent[1] / k)};
            bool on[2] = {a.corr_of_vertex[v[0]] >= 0, two && a.corr_of_vertex[v[1]] >= 0};
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (!on[j]) continue;
#pragma unroll 4
                for (int s = 0; s < k; ++s) {
                    const uint32_t b = a.midx[v[j] * k + s];
                    if (a.mw[v[j] * k + s] != 0.f && b != (uint32_t)node && b < (uint32_t)n)
                        atomicOr(bm + (b >> 5), 1u << (b & 31));
                }
            }
        }
        if (tid < a.kreg) {
            const uint32_t nb = a.gidx[(long)node * a.kreg + tid];
            if (nb < (uint32_t)n && nb != (uint32_t)node) atomicOr(bm + (nb >> 5), 1u << (nb & 31));
        }
        for (unsigned t = tid; t < nin; t += kAsmThreads) {
            const unsigned x = a.b.ilst[io + t] / a.kreg;
            if (x != (unsigned)node) atomicOr(bm + (x >> 5), 1u << (x & 31));
        }
        __syncthreads();
        if (w == 0) {  // ordered extraction
            int base = 0, first = 0;
            for (int w0 = 0; w0 < words; w0 += 32) {
                const int wi = w0 + lane;
                unsigned bits = wi < words ? bm[wi] : 0u;
                const int c = __popc(bits);
                int incl = c;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += y;
                }
                int pos = base + incl - c;
                while (bits) {
                    const int b = wi * 32 + __ffs(bits) - 1;
                    bits &= bits - 1;
                    if (pos < kMaxNbr) {
                        s_L[pos] = b;
                        a.b.nbr[(long)node * kMaxNbr + pos] = b;
                        first += b < node;
                    }
                    ++pos;
                }
                base += __shfl_sync(0xffffffffu, incl, 31);
            }
            first = warp_sum(first);
            if (lane == 0) {
                s_cnt = min(base, kMaxNbr);
                s_first = first;
                a.b.nbr_cnt[node] = min(base, kMaxNbr);
                if (base > kMaxNbr) atomicOr(a.error, ERRF_CAPACITY);
            }
        }
        __syncthreads();  // the list is complete, the bitmap's room is free
        const int first = s_first, nup = s_cnt - first;
        const int* up = s_L + first;
        float d0 = 0.f, d1 = 0.f;
        float acc[kAsmPasses][6];
#pragma unroll
        for (int p = 0; p < kAsmPasses; ++p)
#pragma unroll
            for (int q = 0; q < 6; ++q) acc[p][q] = 0.f;

        // The staged rows (s_rows of every 32) that the block of a group takes part in: a list per group of
        // this warp, in row order, for rows that name a block once; returns this lane's group's length.
        auto list_rows = [&](int pass) {
            int len[kAsmGroups] = {};
            for (int sub = 0; sub < kAsmThreads / 32; ++sub) {
                const int nr = s_rows[sub], row = sub * 32 + lane;
                if (nr == 0) continue;
                const uint2 x = lane < nr ? s_slot[row] : make_uint2(~0u, ~0u);
                const unsigned tag = lane < nr ? (unsigned)row << 6 | (unsigned)s_own[row] << 3 : 0u;
#pragma unroll
                for (int gg = 0; gg < kAsmGroups; ++gg) {
                    const int uu = pass * kAsmPass + gg * kAsmUpWarps + w - 1;
                    if (uu >= nup) break;
                    const unsigned r4 = (unsigned)uu * 0x01010101u;
                    const unsigned lo = __vcmpeq4(x.x, r4), hi = KM > 4 ? __vcmpeq4(x.y, r4) : 0u;
                    const unsigned bal = __ballot_sync(0xffffffffu, (lo | hi) != 0u);
                    if (lo | hi)
                        lists[gg * kAsmThreads + len[gg] + __popc(bal & ((1u << lane) - 1u))] =
                            (unsigned short)(tag | (lo ? (__ffs(lo) - 1) >> 3 : 4 + ((__ffs(hi) - 1) >> 3)));
                    len[gg] += __popc(bal);
                }
            }
            __syncwarp();
            int mine = 0;
#pragma unroll
            for (int gg = 0; gg < kAsmGroups; ++gg)
                if (g == gg) mine = len[gg];
            return mine;
        };
        // Upper blocks over the staged depth rows: listed rows, four in flight; or every row looked at
        // where a vertex of the chunk names a node twice.
        auto sum_listed = [&](int pass, float (&c)[6]) {
            const int len = list_rows(pass);
            const unsigned short* l = lists + min(g, kAsmGroups - 1) * kAsmThreads;
            for (int i0 = 0; i0 < len; i0 += 4) {
                float ja[4];
                float2 jb[4][3];
                const ushort4 q4 = *reinterpret_cast<const ushort4*>(l + i0);
                const unsigned q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const unsigned v = i0 + r < len ? q[r] : q[0];
                    const float* row = J + (v >> 6) * stride;
                    ja[r] = row[((v >> 3) & 7u) * 6 + gi];
#pragma unroll
                    for (int x = 0; x < 3; ++x) jb[r][x] = reinterpret_cast<const float2*>(row + (v & 7u) * 6)[x];
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    if (i0 + r >= len) break;
#pragma unroll
                    for (int x = 0; x < 3; ++x) {
                        c[2 * x] = c[2 * x] + ja[r] * jb[r][x].x;
                        c[2 * x + 1] = c[2 * x + 1] + ja[r] * jb[r][x].y;
                    }
                }
            }
            __syncwarp();
        };
        auto sum_all = [&](int pass, float (&c)[6]) {
            const int u = pass * kAsmPass + g * kAsmUpWarps + w - 1;
            if (g < kAsmGroups && u < nup)
                for (int sub = 0; sub < kAsmThreads / 32; ++sub)
                    for (int r = sub * 32; r < sub * 32 + s_rows[sub]; ++r) {
                        const float* row = J + r * stride;
                        const uint2 y = s_slot[r];
                        for (int tt = 0; tt < k; ++tt) {
                            if (((tt < 4 ? y.x >> (8 * tt) : y.y >> (8 * (tt - 4))) & 0xffu) != (unsigned)u) continue;
                            const float ja = row[s_own[r] * 6 + gi];
#pragma unroll
                            for (int q = 0; q < 6; ++q) c[q] = c[q] + ja * row[tt * 6 + q];
                        }
                    }
            __syncwarp();
        };

        for (unsigned base = o; base < e; base += kAsmThreads) {
            const unsigned t = base + tid;
            const unsigned ent = t < e ? a.b.lst[t] : 0u;
            const long v = ent / k;
            const int s = (int)(ent % k);
            const int c = t < e ? a.corr_of_vertex[v] : -1;
            if (t < e) a.b.jc[t] = c;
            const unsigned bal = __ballot_sync(0xffffffffu, c >= 0);
            bool dup = false;
            if (c >= 0) {
                const int row = (tid & ~31) + __popc(bal & ((1u << lane) - 1u));
                const int px = a.corr[2 * (long)c + 1];
                const float p[3] = {a.mesh[3 * v], a.mesh[3 * v + 1], a.mesh[3 * v + 2]};
                float wt[KM];
                uint32_t bn[KM];
#pragma unroll
                for (int tt = 0; tt < KM; ++tt) {
                    wt[tt] = tt < k ? a.mw[v * k + tt] : 0.f;
                    bn[tt] = tt < k ? a.midx[v * k + tt] : 0u;
                }
                const float nrm[3] = {a.normals[3 * (long)px], a.normals[3 * (long)px + 1], a.normals[3 * (long)px + 2]};
                float G[3][6];
                grad_rows(p, G);
                unsigned slots[2] = {~0u, ~0u};
                float2* out = reinterpret_cast<float2*>(J + row * stride);
#pragma unroll
                for (int tt = 0; tt < KM; ++tt) {
                    if (tt >= k) break;
                    unsigned sl = kSlotNone;
                    if (wt[tt] != 0.f && bn[tt] >= (uint32_t)node) {
                        if (bn[tt] == (uint32_t)node) {
                            sl = kSlotDiag;
                        } else {
                            const int f = find_slot(up, nup, (int)bn[tt]);
                            if (f >= 0) sl = (unsigned)f;
                        }
                    }
                    if (sl != kSlotNone)
                        dup = dup || ((__vcmpeq4(slots[0], sl * 0x01010101u) | __vcmpeq4(slots[1], sl * 0x01010101u)) != 0u);
                    slots[tt / 4] ^= (sl ^ 0xffu) << (8 * (tt % 4));
                    if (sl != kSlotNone || tt == s) {
                        float Jt[6];
                        jdepth(nrm, wt[tt], G, a.lam_d, Jt);
#pragma unroll
                        for (int q = 0; q < 3; ++q) out[tt * 3 + q] = make_float2(Jt[2 * q], Jt[2 * q + 1]);
                        if (tt == s) {  // this row's J block, for J^T r
                            float2* jr = reinterpret_cast<float2*>(a.b.jrow + (long)t * 6);
#pragma unroll
                            for (int q = 0; q < 3; ++q) jr[q] = make_float2(Jt[2 * q], Jt[2 * q + 1]);
                        }
                    }
                }
                s_slot[row] = make_uint2(slots[0], slots[1]);
                s_own[row] = (unsigned char)s;
                s_touched = 1;
            }
            if (lane == 0) s_rows[w] = __popc(bal);
            const bool twice = __syncthreads_or(dup);
            if (w == 0) {
                if (lane < 18)
                    for (int sub = 0; sub < kAsmThreads / 32; ++sub) {
                        const int nr = s_rows[sub];
                        if (!twice) {  // the row's own slot is the only one of this node
                            for (int r0 = 0; r0 < nr; r0 += 8) {
                                const uint2 own = *reinterpret_cast<const uint2*>(s_own + sub * 32 + r0);
                                float ja[8];
                                float2 jb[8];
#pragma unroll
                                for (int r = 0; r < 8; ++r) {
                                    const unsigned t8 = (r < 4 ? own.x >> (8 * r) : own.y >> (8 * (r - 4))) & 0xffu;
                                    const bool in = r0 + r < nr;
                                    const float* row = J + (in ? (sub * 32 + r0 + r) * stride + (int)t8 * 6 : 0);
                                    ja[r] = row[di];
                                    jb[r] = *reinterpret_cast<const float2*>(row + dj);
                                }
#pragma unroll
                                for (int r = 0; r < 8; ++r) {
                                    if (r0 + r >= nr) break;
                                    d0 = d0 + ja[r] * jb[r].x;
                                    d1 = d1 + ja[r] * jb[r].y;
                                }
                            }
                        } else {
                            for (int r = sub * 32; r < sub * 32 + nr; ++r) {
                                const float* row = J + r * stride;
                                const float ja = row[s_own[r] * 6 + di];
                                const uint2 y = s_slot[r];
                                for (int tt = 0; tt < k; ++tt) {
                                    const unsigned sl = ((tt < 4 ? y.x >> (8 * tt) : y.y >> (8 * (tt - 4))) & 0xffu);
                                    if (sl != kSlotDiag) continue;
                                    const float2 jb = *reinterpret_cast<const float2*>(row + tt * 6 + dj);
                                    d0 = d0 + ja * jb.x;
                                    d1 = d1 + ja * jb.y;
                                }
                            }
                        }
                    }
            } else {
#pragma unroll
                for (int pass = 0; pass < kAsmPasses; ++pass) {
                    if (pass * kAsmPass + w - 1 >= nup) break;
                    if (!twice) sum_listed(pass, acc[pass]);
                    else sum_all(pass, acc[pass]);
                }
            }
            __syncthreads();
        }
        // regularisation rows in ascending row order: incoming edges x -> node with x < node,
        // then node's own edges, then incoming edges with x > node (src/MotionOptimization.cu:298-340)
        unsigned nlo = 0;  // incoming rows with source below node (ilst is ascending)
        for (unsigned x = lane; x < nin; x += 32) nlo += (a.b.ilst[io + x] / a.kreg < (unsigned)node) ? 1u : 0u;
        nlo = warp_sum(nlo);
        const unsigned nrows = nin + (unsigned)a.kreg;
        for (unsigned base = 0; base < nrows; base += kAsmThreads) {
            const unsigned r = base + tid;
            if (r < nrows) {
                int src, kk;
                if (r < nlo) {
                    const unsigned ent = a.b.ilst[io + r];
                    src = (int)(ent / a.kreg);
                    kk = (int)(ent % a.kreg);
                } else if (r < nlo + (unsigned)a.kreg) {
                    src = node;
                    kk = (int)(r - nlo);
                } else {
                    const unsigned ent = a.b.ilst[io + r - a.kreg];
                    src = (int)(ent / a.kreg);
                    kk = (int)(ent % a.kreg);
                }
                const uint32_t nbk = a.gidx[(long)src * a.kreg + kk];
                const bool live = !(src == node && nbk >= (uint32_t)n);  // own edge filtered out
                float G[3][6];
                grad_rows(a.nodes + 3 * (long)src, G);
                float2* out = reinterpret_cast<float2*>(J + tid * stride);
#pragma unroll
                for (int ax = 0; ax < 3; ++ax)
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        out[ax * 3 + q] = make_float2(G[ax][2 * q] * a.lam_r, G[ax][2 * q + 1] * a.lam_r);
                const int other = (src == node) ? (int)nbk : src;
                unsigned sl = kSlotNone;
                if (live && other > node) {
                    const int f = find_slot(up, nup, other);
                    if (f >= 0) sl = (unsigned)f;
                }
                s_slot[tid] = make_uint2(0xffffff00u | sl, ~0u);
                s_own[tid] = live ? 1 : 0;  // skipped rows name no block and no diagonal
                if (live) s_touched = 1;
            }
            if (lane == 0) s_rows[w] = max(0, min(32, (int)(nrows - base) - w * 32));
            __syncthreads();
            // the node is an edge's source (coefficient +g) or its target (-g): g_i g_j on the
            // diagonal and -(g_i g_j) between the two either way
            if (w == 0) {
                if (lane < 18) {
                    const int nb = (int)min((unsigned)kAsmThreads, nrows - base);
                    for (int r2 = 0; r2 < nb; ++r2) {
                        if (!s_own[r2]) continue;
#pragma unroll
                        for (int ax = 0; ax < 3; ++ax) {
                            const float* row = J + r2 * stride + ax * 6;
                            const float ga = row[di];
                            const float2 gb = *reinterpret_cast<const float2*>(row + dj);
                            d0 = d0 + ga * gb.x;
                            d1 = d1 + ga * gb.y;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int pass = 0; pass < kAsmPasses; ++pass) {
                    if (pass * kAsmPass + w - 1 >= nup) break;
                    const int len = list_rows(pass);
                    const unsigned short* l = lists + min(g, kAsmGroups - 1) * kAsmThreads;
                    for (int x = 0; x < len; ++x) {
#pragma unroll
                        for (int ax = 0; ax < 3; ++ax) {
                            const float* row = J + (l[x] >> 6) * stride + ax * 6;
                            const float ga = row[gi];
#pragma unroll
                            for (int q = 0; q < 3; ++q) {
                                const float2 gb = reinterpret_cast<const float2*>(row)[q];
                                acc[pass][2 * q] = acc[pass][2 * q] - ga * gb.x;
                                acc[pass][2 * q + 1] = acc[pass][2 * q + 1] - ga * gb.y;
                            }
                        }
                    }
                    __syncwarp();
                }
            }
            __syncthreads();
        }
        if (w == 0) {
            if (!s_touched) {  // identity diagonal block (src/VolumeFusion.cu:637-640)
                d0 = di == dj ? 1.f : 0.f;
                d1 = di == dj + 1 ? 1.f : 0.f;
            }
            if (lane < 18) reinterpret_cast<float2*>(a.b.diag + (long)node * 36)[lane] = make_float2(d0, d1);
        } else if (g < kAsmGroups) {
#pragma unroll
            for (int pass = 0; pass < kAsmPasses; ++pass) {
                const int u = pass * kAsmPass + g * kAsmUpWarps + w - 1;
                if (u >= nup) continue;
                float2* B = reinterpret_cast<float2*>(a.b.blocks + ((long)node * kMaxNbr + first + u) * 36 + gi * 6);
#pragma unroll
                for (int q = 0; q < 3; ++q) B[q] = make_float2(acc[pass][2 * q], acc[pass][2 * q + 1]);
            }
        }
        __syncthreads();  // the shared state is the next node's
    }
}

// Inverses of the diagonal blocks of nodes `node` and `node` + 1: Gauss-Jordan with partial pivoting in FP64, half
// a warp per node with lane j < 12 of it owning column j of [D | I]; stored rounded to FP32 (the
// preconditioner is applied in FP32).  Bound: FP64 issue (16 cycles a warp) with many nodes, the chain of six
// pivots with few; so two nodes share a warp, and a pivot is searched by the lane that owns its column,
// on the bits of the magnitudes.  1,300 nodes: the launch took 23 us with a node per warp, 17 so.
AFX_D void diag_inverse_pair(const GnArgs& a, int node0, int n) {
    const int lane = threadIdx.x & 15, node = node0 + ((threadIdx.x >> 4) & 1);
    const bool on = node < n, own = on && lane < 12;
    const float* D = a.b.diag + (long)(on ? node : node0) * 36;
    constexpr unsigned long long kInf = 0x7ff0000000000000ull;
    double col[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) col[i] = !own ? 0.0 : (lane < 6 ? (double)D[i * 6 + lane] : (lane - 6 == i ? 1.0 : 0.0));
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        // pivot: the largest |m[r][c]|, r >= c (first on ties; one that is not a number is never larger or passed)
        int p = c;
        unsigned long long best = (unsigned long long)__double_as_longlong(fabs(col[c]));
#pragma unroll
        for (int r = c + 1; r < 6; ++r) {
            const unsigned long long v = (unsigned long long)__double_as_longlong(fabs(col[r]));
            if (v > best && v <= kInf) {
                best = v;
                p = r;
            }
        }
        p = __shfl_sync(0xffffffffu, best == 0ull ? -1 : p, c, 16);
        if (p < 0) ok = false;  // the rest is not used
        if (p != c) {
#pragma unroll
            for (int r = c + 1; r < 6; ++r)
                if (r == p) {
                    const double t = col[r];
                    col[r] = col[c];
                    col[c] = t;
                }
        }
        const double d = __shfl_sync(0xffffffffu, col[c], c, 16);
        col[c] /= d;
#pragma unroll
        for (int r = 0; r < 6; ++r)
            if (r != c) {
                const double f = __shfl_sync(0xffffffffu, col[r], c, 16);
                col[r] -= f * col[c];
            }
    }
    if (!on) return;
    float* out = a.b.minv + (long)node * 36;
    if (!ok) {
        if (lane == 0) atomicOr(a.error, ERRF_SINGULAR);
        if (lane < 6)
            for (int i = 0; i < 6; ++i) out[i * 6 + lane] = 0.f;
        return;
    }
    if (lane >= 6 && lane < 12)
#pragma unroll
        for (int i = 0; i < 6; ++i) out[i * 6 + lane - 6] = (float)col[i];
}

// The blocks of one node below the diagonal, as transposes of the owners' (one warp): with them a
// node's row of J^T J is its diagonal block and one contiguous run of blocks, in neighbour order.
AFX_D void lower_blocks_node(const GnArgs& a, int node) {
    const int lane = threadIdx.x & 31;
    const int* L = a.b.nbr + (long)node * kMaxNbr;
    const int cnt = a.b.nbr_cnt[node];
    for (int u0 = 0; u0 < cnt; u0 += 32) {
        const int u = u0 + lane;
        const int owner = u < cnt ? L[u] : node;
        int f = -1;
        if (owner < node) {
            f = find_slot(a.b.nbr + (long)owner * kMaxNbr, a.b.nbr_cnt[owner], node);
            if (f < 0) atomicOr(a.error, ERRF_CAPACITY);
        }
        const int lower = __popc(__ballot_sync(0xffffffffu, owner < node));  // lists ascend: the first ones
        float* dst = a.b.blocks + ((long)node * kMaxNbr + u0) * 36;
        const long from = f >= 0 ? ((long)owner * kMaxNbr + f) * 36 : -1;
#pragma unroll 4
        for (int e0 = 0; e0 < lower * 36; e0 += 32) {
            const int e = e0 + lane, q = e / 36, x = e - 36 * q;
            const long src = __shfl_sync(0xffffffffu, from, q & 31);
            if (e < lower * 36) dst[e] = src >= 0 ? a.b.blocks[src + (x % 6) * 6 + x / 6] : 0.f;
        }
        if (lower < 32) break;
    }
}

// What the Gauss-Newton loop needs besides the blocks, in one launch: the inverses (the first `half`
// CTAs: a serial chain in binary64), and meanwhile the lower blocks, the
// pending transforms as a copy of the committed ones and the loop's state.
__global__ void __launch_bounds__(128) gn_icp_finish_kernel(GnArgs a, float4* T_pending, const float4* T_committed,
                                                           int half) {
    const int n = min(*a.n_nodes, a.n_max);
    if ((int)blockIdx.x < half) {
        for (int node = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 2; node < n; node += half * 8) diag_inverse_pair(a, node, n);
        return;
    }
    const long first = (long)(blockIdx.x - half) * blockDim.x + threadIdx.x;
    const long step = (long)(gridDim.x - half) * blockDim.x;
    for (int node = (int)(first >> 5); node < n; node += (int)(step >> 5)) lower_blocks_node(a, node);
    if (T_pending)
        for (long t = first; t < (long)a.n_max * 4; t += step) T_pending[t] = T_committed[t];
    if (first == 0) {
        GnState* s = a.b.state;
        s->e_prev = 3.4028234663852886e+38;  // std::numeric_limits<float>::max() (src/VolumeFusion.cu:570)
        s->e_last = 0;
        s->e_depth = s->e_reg = 0;
        s->done = 0;
        s->commit = 0;
        s->iters = 0;
    }
}

// ---- Gauss-Newton loop: one thread-block cluster per ICP iteration ----
//
// All Gauss-Newton iterations of one ICP iteration (src/VolumeFusion.cu:571-691) run in one
// launch of a single cluster of kGnClusterMax CTAs (16 where the device allows non-portable
// cluster sizes, else 8).  Phases are separated by the hardware cluster barrier
// (barrier.cluster.arrive.release / wait.acquire), so no CTA spins on memory.  FP64
// reductions go through distributed shared memory: each CTA writes its block sum into a slot
// of its own shared memory and, after the barrier, reads every CTA's slot in rank order, so
// all CTAs hold bit-identical totals and take identical branches.  Values exchanged between
// CTAs through global memory (residuals, pending transforms, PCG vectors, warped vertices)
// are stored with st.global.cg and loaded with ld.global.cg, i.e. always from L2.
// Per iteration:
//   residuals + energies -> energy test and commit -> J^T r -> PCG (x = 0, block-Jacobi,
//   FP32 block SpMV; two exchanges through shared memory per PCG iteration, or three cluster barriers
//   where the vectors are in global memory)
//   -> T_pending -= [[x_rot]x, x_t; 0] -> re-warp the canonical vertices with T_pending.

constexpr int kLoopThreads = 512;
constexpr int kLoopWarps = kLoopThreads / 32;

AFX_D unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

AFX_D unsigned cluster_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

// All threads of all CTAs of the cluster; orders every prior memory access before every later one.
AFX_D void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Load a double from the shared memory of CTA `rank` of this cluster, at the offset of `p` here.
AFX_D double dsmem_load(const double* p, unsigned rank) {
    unsigned local = (unsigned)__cvta_generic_to_shared(p), remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote) : "memory");
    return v;
}

// Double-binary32 ("double-float") numbers: the unevaluated sum hi + lo of two binary32 numbers with
// |lo| <= ulp(hi) / 2, about 48 significant bits.  Knuth's TwoSum gives a binary32 sum and its exact rounding error,
// the same whatever the operands' order, so every lane of a butterfly ends with the same total; Dekker's Fast2Sum does
// so for |a| >= |b|; a product of two binary32 numbers is exact as p + fma(x, y, -p).  On this part a dependent
// binary64 add takes ~150-200 cycles.
struct DF {
    float hi, lo;
};

AFX_D DF two_sum(float a, float b) {
    const float s = a + b, v = s - a;
    return {s, (a - (s - v)) + (b - v)};
}

AFX_D DF fast_two_sum(float a, float b) {
    const float s = a + b;
    return {s, b - (s - a)};
}

// A sum under way: hi is the running binary32 sum, lo the running sum of its exact rounding errors and c
// that of lo's.  Adding two of them waits for one addition on hi and two on lo; the error terms follow
// behind, so a butterfly step costs a shuffle and two additions where adding double-floats takes
// thirteen, and the result carries more bits (errors of the PCG's dot products against exact sums, over
// 12 to 384 terms per CTA and 16 CTAs, relative to the sum of |x y|: about a third of a double-float's; with
// 66 terms at most 1.8e-15 and 3.2e-16 on average, against 4.7e-15 and 9.5e-16).
struct TF {
    float hi, lo, c;
};

AFX_D TF tf_add(TF a, TF b) {
    const DF h = two_sum(a.hi, b.hi), l = two_sum(a.lo, b.lo), m = two_sum(l.hi, h.lo);
    return {h.hi, m.hi, (a.c + b.c) + (l.lo + m.lo)};
}

AFX_D TF tf_add_prod(TF a, float x, float y) {
    const float p = x * y;
    return tf_add(a, {p, fmaf(x, y, -p), 0.f});
}

// Sum over the lanes that differ in bits kFrom, kFrom / 2, ..., 1 of their number, as a double-float.
template <int kFrom>
AFX_D DF tf_butterfly(TF v) {
#pragma unroll
    for (int o = kFrom; o > 0; o >>= 1) {
        const TF u = {__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o),
                      __shfl_xor_sync(0xffffffffu, v.c, o)};
        v = tf_add(v, u);
    }
    const DF s = fast_two_sum(v.hi, v.lo);
    return fast_two_sum(s.hi, s.lo + v.c);
}

// a / b rounded to binary32 (within about half an ulp): the binary32 quotient of the high parts,
// corrected once by the remainder, which fma forms exactly.
AFX_D float df_quotient(DF a, DF b) {
    const float q = a.hi / b.hi;
    if (q == 0.f || !isfinite(q)) return q;
    const float r = (fmaf(-q, b.hi, a.hi) + a.lo) - q * b.lo;
    return q + r / b.hi;
}

AFX_D bool df_zero_or_nan(DF v) { return v.hi == 0.f || v.hi != v.hi; }

constexpr int kClusterMax = 16;

struct ClusterSums {
    double slot[2][4];            // this CTA's block sums, double-buffered across calls
    double warp[kLoopWarps * 4];  // per-warp sums
    double total[4];
    double in[2][kClusterMax][2];  // every CTA's sums (cluster_sum_tf)
    int phase;
    int dead;  // a wait of some CTA ran out (gn_solve)
};

// Double-floats in this CTA's shared memory and in CTA `rank`'s (8-byte slots, hi first).
AFX_D void sts_df(double* local, DF v) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(local);
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.hi), "f"(v.lo) : "memory");
}
AFX_D DF lds_df_local(const double* local) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(local);
    DF v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.hi), "=f"(v.lo) : "r"(a) : "memory");
    return v;
}
AFX_D void dsmem_store_df(double* local, unsigned rank, DF v) {
    unsigned a = (unsigned)__cvta_generic_to_shared(local), ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(ra), "f"(v.hi), "f"(v.lo) : "memory");
}

// Sums over every thread of the cluster as double-floats, in fixed-shape trees (butterfly within each
// warp, the CTA's warps, the CTAs by rank): warp 0 puts the CTA's sums into slot [rank] of every
// CTA, and after the barrier every warp adds its CTA's slots, so all threads of all CTAs hold the same
// totals.  Contains one cluster barrier.
template <int NV>
AFX_D void cluster_sum_tf(const TF (&v)[NV], DF (&t)[NV], ClusterSums& cs) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const DF s = tf_butterfly<16>(v[i]);
        if (lane == 0) sts_df(&cs.warp[w * 4 + i], s);
    }
    __syncthreads();
    const int ph = cs.phase;
    if (w == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            DF s = lds_df_local(&cs.warp[(lane & (kLoopWarps - 1)) * 4 + i]);
            s = tf_butterfly<kLoopWarps / 2>({s.hi, s.lo, 0.f});
            if (lane < (int)cluster_size()) dsmem_store_df(&cs.in[ph][cluster_rank()][i], lane, s);
        }
    }
    cluster_barrier();
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int q = lane & (kClusterMax - 1);
        DF s = {0.f, 0.f};
        if (q < (int)cluster_size()) s = lds_df_local(&cs.in[ph][q][i]);
        t[i] = tf_butterfly<kClusterMax / 2>({s.hi, s.lo, 0.f});
    }
    if (threadIdx.x == 0) cs.phase = ph ^ 1;
}

// Sums v[0] and v[1] over every thread of the cluster; all threads of all CTAs get identical totals.
// Fixed-shape FP64 trees: butterfly within each warp, then over the CTA's warps, then over the
// CTAs by rank.  FP64 additions issue at one warp in about 20 cycles per SM, so a step of the trees adds
// both values, one in each half of the warp.  Contains one cluster barrier.
AFX_D void cluster_sum_pair(double (&v)[2], ClusterSums& cs) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    static_assert(kLoopWarps == 16, "half a warp per value");
    auto half_sum = [](double s) {  // over the 16 lanes of each half
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    };
    const int k = lane >> 4, q = lane & 15;  // value and item of this lane
    const double give = k ? v[0] : v[1], got = __shfl_xor_sync(0xffffffffu, give, 16);
    const double s = half_sum((k ? v[1] : v[0]) + got);
    if (q == 0) cs.warp[w * 4 + k] = s;
    __syncthreads();
    const int ph = cs.phase;
    if (w == 0) {
        const double t = half_sum(cs.warp[q * 4 + k]);
        if (q == 0) cs.slot[ph][k] = t;
    }
    cluster_barrier();
    if (w == 0) {
        const double t = half_sum(q < (int)cluster_size() ? dsmem_load(&cs.slot[ph][k], q) : 0.0);
        if (q == 0) cs.total[k] = t;
    }
    __syncthreads();
    v[0] = cs.total[0];
    v[1] = cs.total[1];
    if (threadIdx.x == 0) cs.phase = ph ^ 1;
}

struct LoopArgs {
    GnArgs g;
    const float* points;  // canonical vertices
    float* warped;
    float* T_committed;
    float* T_pending;
    int gn_iters, pcg_iters;
    double tol;      // <= 0: run exactly pcg_iters PCG iterations
    int wait_polls;  // polls of an exchange between CTAs before it gives up
    int* gave_up;    // set when one does (memory the host reads), or null
};

// J^T r of one node, one warp: lane l sums the node-list entries l, l+32, ... (depth rows, J
// rows formed once per ICP iteration by jtj_assemble_kernel) and then the regularisation rows
// l, l+32, ... (incoming edges, then the node's own); the 32 partial sums are combined by a
// butterfly, so every lane returns the same six totals.
AFX_D void jtr_node(const GnArgs& a, int node, int n, float (&acc)[6]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[q] = 0.f;
    const unsigned o = a.b.loff[node], e = a.b.loff[node + 1];
    constexpr int kAhead = 8;  // entries whose loads are in flight together
    for (unsigned t0 = o + lane; t0 < e; t0 += 32 * kAhead) {
        int c[kAhead];
        float J[kAhead][6], rd[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) c[k] = t0 + 32 * k < e ? a.b.jc[t0 + 32 * k] : -1;
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
#pragma unroll
            for (int q = 0; q < 6; ++q) J[k][q] = t0 + 32 * k < e ? a.b.jrow[(long)(t0 + 32 * k) * 6 + q] : 0.f;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) rd[k] = c[k] >= 0 ? __ldcg(a.b.rdepth + c[k]) : 0.f;
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
#pragma unroll
            for (int q = 0; q < 6; ++q) acc[q] = c[k] >= 0 ? acc[q] + J[k][q] * rd[k] : acc[q];
    }
    const unsigned io = a.b.ioff[node], nin = a.b.ioff[node + 1] - io;
    for (unsigned u = lane; u < nin + (unsigned)a.kreg; u += 32) {
        int src, kk;
        if (u < nin) {
            const unsigned ent = a.b.ilst[io + u];
            src = (int)(ent / a.kreg);
            kk = (int)(ent % a.kreg);
        } else {
            src = node;
            kk = (int)(u - nin);
            if (a.gidx[(long)node * a.kreg + kk] >= (uint32_t)n) continue;
        }
        float G[3][6];
        grad_rows(a.nodes + 3 * (long)src, G);
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const float r = __ldcg(a.b.rreg + ((long)src * a.kreg + kk) * 3 + ax);
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const float g = G[ax][q] * a.lam_r;
                const float jn = (src == node) ? g : -g;
                acc[q] = acc[q] + jn * r;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[q] = warp_sum(acc[q]);
}

// Row `i` of A z for node `node`: the node's blocks (diagonal first, then the neighbours in
// ascending order) times z, FP32, two elements a load (8,000 nodes, ten iterations: 536 us, 800 with one).
AFX_D float spmv_entry(const GnBuffers& b, int node, int i, const float* z) {
    const int cnt = b.nbr_cnt[node];
    auto product = [&](const float* block, int other) {  // row i of a block times the node's part of z, by pairs
        const float2* B = reinterpret_cast<const float2*>(block + i * 6);
        const float2* x = reinterpret_cast<const float2*>(z + (long)other * 6);
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const float2 v = B[j], y = __ldcg(x + j);
            s = s + v.x * y.x;
            s = s + v.y * y.y;
        }
        return s;
    };
    float acc = 0.f + product(b.diag + (long)node * 36, node);
#pragma unroll 4
    for (int u = 0; u < cnt; ++u)
        acc = acc + product(b.blocks + ((long)node * kMaxNbr + u) * 36, b.nbr[(long)node * kMaxNbr + u]);
    return acc;
}

// ---- PCG with the system resident in distributed shared memory ----
//
// For graphs up to kDsNpc nodes per CTA, each CTA of the cluster owns a contiguous node range
// and keeps, in its shared memory, the rows of J^T J for its nodes (diagonal block, then the
// neighbour blocks in ascending neighbour order, lower ones stored transposed so every block
// is row-major B_ij), their block inverses, its slices of x, r, p, A p, and a full copy of z.
// After each update a CTA writes its new z slice into every CTA's copy (st.async), so
// the SpMV reads only local shared memory.  Partial sums are written into every CTA's slot
// array the same way and summed locally in one fixed order: identical totals in all
// CTAs.  J^T J does not change during the Gauss-Newton loop, so the rows are staged once.

constexpr int kDsNodes = 1024;   // node limit of this path (full z copy)
constexpr int kDsNpc = 64;       // nodes per CTA
constexpr int kDsBlocks = 1024;  // blocks per CTA (diagonal included)
constexpr int kDsMaxCta = 16;

// Copies of 4 or 16 bytes from global to shared memory that no register waits for; stage_wait before the
// barrier after which they are read.
AFX_D void stage_word(int* dst, const int* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
AFX_D void stage_quad(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
AFX_D void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// rowptr[0..own] of the nodes from `start` on: a diagonal block and the neighbours' each (whole CTA).
AFX_D void stage_rowptr(const GnBuffers& b, int* rowptr, int start, int own) {
    for (int li = threadIdx.x; li < own; li += kLoopThreads) rowptr[li] = 1 + b.nbr_cnt[start + li];
    __syncthreads();
    if (threadIdx.x < 32) {
        int carry = 0;
        for (int base = 0; base < own; base += 32) {
            const int li = base + (int)threadIdx.x;
            const int c = li < own ? rowptr[li] : 0;
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += y;
            }
            if (li < own) rowptr[li] = carry + incl - c;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (threadIdx.x == 0) rowptr[own] = carry;
    }
    __syncthreads();
}

struct DsLayout {
    float* z;       // [kDsNodes * 6] full copy
    float* pf;      // [kDsNodes * 6] full copy of the search direction (each CTA forms it)
    float* x;       // [kDsNpc * 6] own slices
    float* r;
    float* ap;      // [kDsNpc * 6] own slice of A p
    float* minv;    // [kDsNpc * 36]
    float* blk;     // [kDsBlocks * 36]
    int* col;       // [kDsBlocks] neighbour node of each block
    int* rowptr;    // [kDsNpc + 1]
    double* slot;   // [2][kDsMaxCta][4]
    unsigned long long* bar;  // [2] mbarriers: p.Ap exchange, r.z exchange
    float* scal;    // [4] beta, stop, whether a wait of this CTA ran out (on 16 bytes, read together)
};

constexpr size_t kDsSmem = sizeof(float) * ((size_t)kDsNodes * 12 + 3 * kDsNpc * 6 + kDsNpc * 36 + (size_t)kDsBlocks * 36) +
                           sizeof(int) * (kDsBlocks + kDsNpc + 1 + 4) + sizeof(double) * (2 * kDsMaxCta * 4 + 4) + 64;

// `base` on 16 bytes: blocks, inverses, z and p are also copied and read 16 bytes at a time.
AFX_D DsLayout ds_layout(void* base) {
    static_assert(sizeof(double) * (2 * kDsMaxCta * 4 + 2) % 16 == 0 && sizeof(double) * (2 * kDsMaxCta * 4 + 4) % 16 == 0 && sizeof(float) * kDsNodes * 6 % 16 == 0 &&
                      sizeof(float) * kDsNpc * 6 % 16 == 0 && sizeof(float) * kDsNpc * 36 % 16 == 0,
                  "scal and every array from z on start on 16 bytes");
    DsLayout d;
    double* dp = static_cast<double*>(base);
    d.slot = dp;
    d.bar = reinterpret_cast<unsigned long long*>(dp + 2 * kDsMaxCta * 4);
    d.scal = reinterpret_cast<float*>(dp + 2 * kDsMaxCta * 4 + 2);
    float* f = reinterpret_cast<float*>(dp + 2 * kDsMaxCta * 4 + 4);
    d.z = f;
    f += kDsNodes * 6;
    d.pf = f;
    f += kDsNodes * 6;
    d.x = f;
    f += kDsNpc * 6;
    d.r = f;
    f += kDsNpc * 6;
    d.ap = f;
    f += kDsNpc * 6;
    d.minv = f;
    f += kDsNpc * 36;
    d.blk = f;
    f += (size_t)kDsBlocks * 36;
    int* ip = reinterpret_cast<int*>(f);
    d.col = ip;
    ip += kDsBlocks;
    d.rowptr = ip;
    return d;
}

// Store to the same shared-memory offset in CTA `rank` of this cluster.
AFX_D void dsmem_store_f64(double* local, unsigned rank, double v) {
    unsigned a = (unsigned)__cvta_generic_to_shared(local), ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
}
AFX_D void dsmem_store_int(int* local, unsigned rank, int v) {
    unsigned a = (unsigned)__cvta_generic_to_shared(local), ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(ra), "r"(v) : "memory");
}
// Asynchronous stores to the same shared-memory offset in CTA `rank` of this cluster, counted on that
// CTA's mbarrier: the receiver waits for the bytes it expects, so an exchange costs one trip
// through the cluster's network instead of a store, its acknowledgement and a cluster barrier
// (16 CTAs of 512 threads: 1,165 cycles that way; here the wait after a CTA's own last store is 230 to 310).
AFX_D unsigned cluster_addr(const void* local, unsigned rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(local), ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    return ra;
}
AFX_D void async_store_df(unsigned addr, unsigned bar, DF v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "f"(v.hi), "f"(v.lo), "r"(bar)
                 : "memory");
}

// The two exchanges of a PCG iteration.  Phases alternate: a CTA sends its part of an exchange only
// after it has received the other one of the step before from every CTA, that is after every CTA has
// read what this one overwrites.
//
// Waits are bounded.  A CTA one of whose waits runs out flags the error and leaves the solve at its next barrier,
// with no further sends; it then waits, again bounded, for what the others may have sent it until they
// run out too (ds_drain), so that no store is under way to a CTA that has left.  The others learn of it at the end of
// the solve (gn_solve), and nobody sends any more in that launch.
struct DsExchange {
    unsigned parity[2];  // phase of each mbarrier that the next wait is for
    bool dead;           // a wait ran out (this thread's within a solve, any CTA's after it)
};

constexpr int kDsWaitPolls = 1 << 20;
constexpr int kDsDrainPolls = 1 << 12;

// Before the cluster barrier at the start of the kernel (one thread).
AFX_D void ds_exchange_init(const DsLayout& d) {
    d.scal[2] = 0.f;
    for (int i = 0; i < 2; ++i)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(d.bar + i)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Expect `bytes` on mbarrier i in its current phase (one thread).
AFX_D void ds_expect(const DsLayout& d, int i, unsigned bytes) {
    const unsigned bar = (unsigned)__cvta_generic_to_shared(d.bar + i);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Whether the phase `parity` of mbarrier i ends within `polls` polls.
AFX_D bool ds_poll(const DsLayout& d, int i, unsigned parity, int polls) {
    const unsigned bar = (unsigned)__cvta_generic_to_shared(d.bar + i);
    unsigned ok = 0;
    for (int it = 0; it < polls && !ok; ++it)
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
    return ok != 0;
}

// Wait (bounded) for the current phase of mbarrier i.
AFX_D void ds_wait(const DsLayout& d, int i, DsExchange& x, const LoopArgs& L) {
    if (ds_poll(d, i, x.parity[i], L.wait_polls)) {
        x.parity[i] ^= 1u;
    } else {
        x.dead = true;
        d.scal[2] = 1.f;
        if (L.g.error) atomicOr(L.g.error, ERRF_TIMEOUT);
    }
}

// After a wait ran out (one thread, which has made every wait): what the other CTAs have sent or may still send before
// their own waits run out, that is at most the exchange that was waited for and the one after it.  `armed`: the
// mbarriers whose bytes are expected already.
AFX_D void ds_drain(const DsLayout& d, const DsExchange& x, unsigned armed, const unsigned (&bytes)[2]) {
    for (int i = 0; i < 2; ++i)
        if (!((armed >> i) & 1u)) ds_expect(d, i, bytes[i]);
    for (int i = 0; i < 2; ++i) ds_poll(d, i, x.parity[i], kDsDrainPolls);
}

// Cluster sum through the slot arrays: the CTA's block total is written into slot[ph][rank] of
// every CTA; after the barrier each CTA adds the slots in rank order.
template <int NV>
AFX_D void ds_sum(double (&v)[NV], const DsLayout& d, ClusterSums& cs, int& ph) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned rank = cluster_rank(), ncta = cluster_size();
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const double s = warp_sum(v[i]);
        if (lane == 0) cs.warp[w * 4 + i] = s;
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            double s = lane < kLoopWarps ? cs.warp[lane * 4 + i] : 0.0;
#pragma unroll
            for (int o = kLoopWarps / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            // lane q < ncta sends the total to CTA q
            if (lane < (int)ncta) dsmem_store_f64(d.slot + (ph * kDsMaxCta + rank) * 4 + i, lane, s);
        }
    }
    cluster_barrier();
    if (w == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            double t = lane < (int)ncta ? d.slot[(ph * kDsMaxCta + lane) * 4 + i] : 0.0;
#pragma unroll
            for (int o = kDsMaxCta / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) cs.total[i] = t;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = cs.total[i];
    ph ^= 1;
}

// Stage this CTA's rows; returns (uniformly over the cluster) whether every CTA's rows fit.
AFX_D bool ds_stage(const GnBuffers& b, int n, const DsLayout& d, ClusterSums& cs, int& ph) {
    const unsigned rank = cluster_rank(), ncta = cluster_size();
    const int npc = (n + (int)ncta - 1) / (int)ncta;
    const int start = min(n, (int)rank * npc), own = min(n, start + npc) - start;
    stage_rowptr(b, d.rowptr, start, own);
    double need[1] = {d.rowptr[own] > kDsBlocks ? 1.0 : 0.0};
    ds_sum<1>(need, d, cs, ph);
    if (need[0] != 0.0) return false;
    // the rows (block-major, 36 floats each) and the inverses
    for (int li = threadIdx.x >> 5; li < own; li += kLoopWarps) {
        const long node = start + li;
        const int lane = threadIdx.x & 31;
        const int r0 = d.rowptr[li], cnt = d.rowptr[li + 1] - r0 - 1;
        if (lane < 9) {
            stage_quad(d.blk + r0 * 36 + lane * 4, b.diag + node * 36 + lane * 4);
            stage_quad(d.minv + li * 36 + lane * 4, b.minv + node * 36 + lane * 4);
        }
        if (lane == 0) d.col[r0] = (int)node;
        for (int u = lane; u < cnt; u += 32) stage_word(d.col + r0 + 1 + u, b.nbr + node * kMaxNbr + u);
        for (int e = lane; e < cnt * 9; e += 32)
            stage_quad(d.blk + (r0 + 1) * 36 + e * 4, b.blocks + node * kMaxNbr * 36 + e * 4);
    }
    stage_wait();
    __syncthreads();
    return true;
}

// Dot products x[i] . y[i] of the CTA's own entries (cnt floats each, in shared memory), summed over the
// cluster (each product enters exactly; a CTA's sum travels as a double-float, 48 bits).  Warp 0 sends:
// lane l accumulates entries l, l + 32, ..., a butterfly gives the CTA's sum, and lane q puts it
// into slot [i][rank] of CTA q (i: the exchange, 0 for p.Ap, 1 for r.z).
template <int NV>
AFX_D void ds_dot_send(const float* const (&x)[NV], const float* const (&y)[NV], int cnt, const DsLayout& d, int i) {
    const int lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank(), ncta = cluster_size();
    const unsigned bar = cluster_addr(d.bar + i, lane < (int)ncta ? lane : 0);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        TF v = {0.f, 0.f, 0.f};
        constexpr int kAhead = 4;  // terms loaded together
        for (int o0 = lane; o0 < cnt; o0 += 32 * kAhead) {
            float xs[kAhead], ys[kAhead];
#pragma unroll
            for (int q = 0; q < kAhead; ++q) {
                const int o = o0 + 32 * q;
                xs[q] = o < cnt ? x[k][o] : 0.f;
                ys[q] = o < cnt ? y[k][o] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < kAhead; ++q)
                if (q == 0 || o0 - lane + 32 * q < cnt) v = tf_add_prod(v, xs[q], ys[q]);  // a zero product adds nothing
        }
        const DF s = tf_butterfly<16>(v);
        if (lane < (int)ncta) async_store_df(cluster_addr(d.slot + (i * kDsMaxCta + rank) * 4 + k, lane), bar, s);
    }
}

// The totals of exchange i, in every lane of every warp: the slots in one fixed tree, so all CTAs hold the
// same bits.
template <int NV>
AFX_D void ds_dot_total(const DsLayout& d, int i, DF (&t)[NV]) {
    const int lane = threadIdx.x & 31;
    const unsigned ncta = cluster_size();
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        // lanes 16 .. 31 hold the same slots again, so every lane ends with the total
        const int q = lane & (kDsMaxCta - 1);
        DF v = {0.f, 0.f};
        if (q < (int)ncta) v = lds_df_local(d.slot + (i * kDsMaxCta + q) * 4 + k);
        t[k] = tf_butterfly<kDsMaxCta / 2>({v.hi, v.lo, 0.f});
    }
}

// One PCG solve (same recurrences as the global-memory path), then T_pending -= [x] for the own
// nodes.  J^T r is read from b.jtr.  Per iteration: p = z + beta p over all nodes (each CTA keeps a
// full copy of p and of z), A p of the own rows with up to 32 lanes per row (each summing a fixed
// stride of the row's blocks, then a butterfly), p.Ap (exchange 0), the own x / r / z updates, and z to
// every CTA's copy -- one warp per destination -- while warp 0 sums r.z (and r.r when a tolerance is
// set; exchange 1).  A thread keeps its share of its row (up to kRegBlocks blocks), and its entry of x,
// r and the inverse, in registers for the whole solve.
// Bound: the chain of those steps, CTA barriers and two exchanges, about 6,000 cycles an iteration with 169 nodes
// on 16 CTAs (A p 750, the two sums with their sending 2,700, updates 700, waits 550).  gn_loop_kernel in
// the 256^3 sequence (169 nodes): 305 us with cluster barriers, double-float sums and the matrix rows read from
// shared memory in each iteration, 267 us so (232 with the transforms staged, NodeT below; the whole launch takes 203 us).
constexpr int kRegBlocks = 6;

template <bool kTol>
AFX_D void pcg_ds(const LoopArgs& L, int n, const DsLayout& d, DsExchange& ex) {
    const GnBuffers& b = L.g.b;
    const unsigned rank = cluster_rank(), ncta = cluster_size();
    const int npc = (n + (int)ncta - 1) / (int)ncta;
    const int start = min(n, (int)rank * npc), own = min(n, start + npc) - start;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int grp = lane / 6, ei = lane - 6 * grp;
    const int li = w * 5 + grp;  // kLoopWarps * 5 >= kDsNpc: one own node per lane group
    const bool act = lane < 30 && li < own;
    const int o = li * 6 + ei;
    const int cnt = own * 6;
    constexpr int NV = kTol ? 2 : 1;
    float* zown = d.z + (long)start * 6;
    float* pown = d.pf + (long)start * 6;
    // what arrives: every CTA's sums, and for exchange 1 every other CTA's z
    const unsigned dot_bytes = ncta * 8u, rz_bytes = ncta * 8u * NV + (unsigned)(n - own) * 24u;
    // SpMV lanes per row: the largest power of two with every own row covered at once
    int R = 1;
    while (R < 32 && 2 * R * cnt <= (int)blockDim.x) R <<= 1;
    static_assert(kDsNpc * 6 <= kLoopThreads, "a thread per row");
    const int row = (int)threadIdx.x / R, part = (int)threadIdx.x % R;
    const int re = row % 6;  // row within its block
    int b0 = 0, b1 = 0;
    if (row < cnt) {
        b0 = d.rowptr[row / 6] + part;
        b1 = d.rowptr[row / 6 + 1];
    }
    float A[kRegBlocks][6];
    int col[kRegBlocks];
#pragma unroll
    for (int k = 0; k < kRegBlocks; ++k) {
        const int bk = b0 + k * R;
        col[k] = bk < b1 ? d.col[bk] * 3 : 0;  // in float2
#pragma unroll
        for (int j = 0; j < 6; ++j) A[k][j] = bk < b1 ? d.blk[bk * 36 + re * 6 + j] : 0.f;
    }
    auto row_times = [&](const float (&B)[6], int c) {
        const float2* xv = reinterpret_cast<const float2*>(d.pf) + c;
        const float2 x0 = xv[0], x1 = xv[1], x2 = xv[2];
        float s = 0.f;
        s = s + B[0] * x0.x;
        s = s + B[1] * x0.y;
        s = s + B[2] * x1.x;
        s = s + B[3] * x1.y;
        s = s + B[4] * x2.x;
        s = s + B[5] * x2.y;
        return s;
    };
    float minv[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) minv[q] = act ? d.minv[li * 36 + ei * 6 + q] : 0.f;
    // z = M^-1 r of the own entry; r and z where warp 0 and the senders read them
    auto precondition = [&](float rv, bool stop) {
        float rq[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) rq[q] = __shfl_sync(0xffffffffu, rv, lane < 30 ? grp * 6 + q : q);
        float zi = 0.f;
#pragma unroll
        for (int q = 0; q < 6; ++q) zi = zi + minv[q] * rq[q];
        if (act) {
            d.r[o] = rv;
            zown[o] = zi;
        }
        if (__syncthreads_or(stop || ex.dead)) return false;
        if (w == 0) {
            if constexpr (kTol) ds_dot_send<2>({d.r, d.r}, {zown, d.r}, cnt, d, 1);
            else ds_dot_send<1>({d.r}, {zown}, cnt, d, 1);
        }
        for (unsigned k = (unsigned)w; k < ncta; k += kLoopWarps - 1) {  // warp w: the w-th CTA after this one
            if (k == 0) break;
            const unsigned q = rank + k < ncta ? rank + k : rank + k - ncta;
            const unsigned to = cluster_addr(zown, q), bar = cluster_addr(d.bar + 1, q);
            for (int i = lane; i < cnt / 2; i += 32) {
                const float2 v = reinterpret_cast<const float2*>(zown)[i];
                async_store_df(to + 8 * i, bar, {v.x, v.y});
            }
        }
        return true;
    };
    // x = 0, r = b, z = M^-1 r
    float x = 0.f, rv = act ? __ldcg(b.jtr + (long)(start + li) * 6 + ei) : 0.f;
    if (threadIdx.x == 0) ds_expect(d, 1, rz_bytes);
    precondition(rv, false);
    ds_wait(d, 1, ex, L);
    __syncthreads();
    const int iters = d.scal[2] != 0.f ? 0 : L.pcg_iters;
    DF t[NV];
    ds_dot_total<NV>(d, 1, t);
    DF rz = t[0];
    const bool mine = w * 5 < own;  // the warp has entries
    const float tol2 = kTol ? (float)(L.tol * L.tol) : 0.f, bn = t[NV - 1].hi;
    float beta = 0.f;
    int armed = -1;
    for (int it = 0; it < iters; ++it) {
        // p = z (first iteration) or z + beta p, formed for all nodes by every CTA from its copies
#pragma unroll 2
        for (int i = threadIdx.x; i < n * 3; i += kLoopThreads) {
            const float2 zv = reinterpret_cast<const float2*>(d.z)[i];
            float2* pv = reinterpret_cast<float2*>(d.pf) + i;
            if (it) {
                const float2 pp = *pv;
                *pv = make_float2(zv.x + beta * pp.x, zv.y + beta * pp.y);
            } else {
                *pv = zv;
            }
        }
        __syncthreads();
        // A p of the own rows
        float acc = 0.f, prod[kRegBlocks];
#pragma unroll
        for (int k = 0; k < kRegBlocks; ++k) prod[k] = row_times(A[k], col[k]);
#pragma unroll
        for (int k = 0; k < kRegBlocks; ++k) acc = b0 + k * R < b1 ? acc + prod[k] : acc;
        for (int bk = b0 + kRegBlocks * R; bk < b1; bk += R) {
            float B[6];
#pragma unroll
            for (int j = 0; j < 6; ++j) B[j] = d.blk[bk * 36 + re * 6 + j];
            acc = acc + row_times(B, d.col[bk] * 3);
        }
        for (int m = R / 2; m > 0; m >>= 1) acc = acc + __shfl_xor_sync(0xffffffffu, acc, m);
        if (row < cnt && part == 0) d.ap[row] = acc;
        if (threadIdx.x == 0) ds_expect(d, 0, dot_bytes);
        __syncthreads();
        if (w == 0) ds_dot_send<1>({pown}, {d.ap}, cnt, d, 0);
        const float pv = act ? pown[o] : 0.f, apv = act ? d.ap[o] : 0.f;
        // the totals and step sizes: alpha by the warps that have entries, beta by one warp (all warps
        // forming them costs more, by their instructions, than handing beta round)
        bool stop = false;
        if (mine || w == 0) {
            ds_wait(d, 0, ex, L);
            DF pap[1];
            ds_dot_total<1>(d, 0, pap);
            stop = df_zero_or_nan(pap[0]);  // the same in every CTA
            const float alpha = df_quotient(rz, pap[0]);
            x = stop ? x : x + alpha * pv;
            rv = rv - alpha * apv;
        } else {
            ex.parity[0] ^= 1u;
        }
        if (threadIdx.x == 0 && !stop && !ex.dead) ds_expect(d, 1, rz_bytes);
        // every CTA has read z (forming p) before it sent its part of p.Ap, so it can be overwritten here
        if (!precondition(rv, stop)) {  // no direction left, or the wait for p.Ap ran out
            armed = ex.dead ? 1 : (stop ? 0 : 2);
            break;
        }
        ds_wait(d, 1, ex, L);
        if (mine || w == 0) {
            ds_dot_total<NV>(d, 1, t);
            if (threadIdx.x == 0) {
                d.scal[0] = df_quotient(t[0], rz);
                d.scal[1] = kTol && t[NV - 1].hi <= tol2 * bn ? 1.f : 0.f;
            }
            rz = t[0];
        }
        __syncthreads();
        const float4 sc = *reinterpret_cast<const float4*>(d.scal);
        beta = sc.x;
        if ((kTol && sc.y != 0.f) || sc.z != 0.f) break;  // close enough, or the wait for r.z ran out
    }
    if (act) d.x[o] = x;
    // T_pending -= [[x_rot]x, x_t; 0] for the own nodes (updateTransformsKernel,
    // src/MotionOptimization.cu:483-498); x also to global memory for inspection.  After a wait that ran out there is
    // no x: the transforms stay.
    const bool mine_dead = ex.dead;
    ex.dead = __syncthreads_or(mine_dead);
    if (ex.dead) {
        if (threadIdx.x == 0) {
            if (armed < 0) armed = mine_dead ? 2 : 0;  // left after the wait for r.z
            const unsigned bytes[2] = {dot_bytes, rz_bytes};
            ds_drain(d, ex, (unsigned)armed, bytes);
            if (L.gave_up) {
                *(volatile int*)L.gave_up = 1;
                __threadfence_system();
            }
        }
        for (int t = threadIdx.x; t < own * 6; t += blockDim.x) __stcg(b.x + (long)start * 6 + t, NAN);
        return;
    }
    for (int t = threadIdx.x; L.T_pending && t < own * 16; t += blockDim.x) {
        const int l = t >> 4, e = t & 15;
        const float* u = d.x + l * 6;
        float U;
        switch (e) {
            case 1: U = u[2]; break;
            case 2: U = -u[1]; break;
            case 4: U = -u[2]; break;
            case 6: U = u[0]; break;
            case 8: U = u[1]; break;
            case 9: U = -u[0]; break;
            case 12: U = u[3]; break;
            case 13: U = u[4]; break;
            case 14: U = u[5]; break;
            default: U = 0.f;
        }
        float* T = L.T_pending + (long)(start + l) * 16 + e;
        __stcg(T, __ldcg(T) - U);
    }
    for (int t = threadIdx.x; t < own * 6; t += blockDim.x) __stcg(b.x + (long)start * 6 + t, d.x[t]);
}

// ---- phases of the Gauss-Newton loop (all CTAs of the cluster unless stated) ----

// The node transforms as the phases read them (rows 0 to 2; what the fourth row holds is never used):
// from global memory through L2 (T is written by other CTAs of the launch), or, when the system lives in
// shared memory, from a copy in the room of z and p, which are free between solves.  A vertex reads four
// transforms and an edge two, each transform many times: 3 loads of 16 bytes of shared memory instead of 12
// loads from L2.  With this, the loads of several items in flight in each phase, half the FP64 additions
// in the energy sum and the nodes of J^T r dealt over all CTAs, gn_loop_kernel in the 256^3 sequence went
// from 267 to 232 us.
template <bool kStaged>
struct NodeT {
    const float* T;     // [n][16]
    const float4* rows;  // kStaged: [n][3] rows (T[r], T[4 + r], T[8 + r], T[12 + r])
    int n;
    AFX_D void load(uint32_t i, float (&M)[16]) const {
        if (kStaged && i < (uint32_t)n) {
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const float4 v = rows[3 * i + r];
                M[r] = v.x;
                M[4 + r] = v.y;
                M[8 + r] = v.z;
                M[12 + r] = v.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) M[e] = (e & 3) < 3 ? __ldcg(T + 16 * (long)i + e) : 0.f;
        }
    }
};

// Stage the transforms of all n <= kDsNodes nodes (every thread of the CTA; ends with a CTA barrier).  Other CTAs
// must be past their last store into this CTA's z, and the next solve must begin after a cluster barrier.
AFX_D void stage_node_T(const float* T, int n, const DsLayout& d) {
    float4* rows = reinterpret_cast<float4*>(d.z);
    static_assert(kDsNodes * 12 * sizeof(float) == 2 * sizeof(float) * kDsNodes * 6, "z and p hold the rows");
#pragma unroll 2
    for (int t = threadIdx.x; t < 3 * n; t += kLoopThreads) {
        const float* p = T + 16 * (long)(t / 3) + t % 3;
        rows[t] = make_float4(__ldcg(p), __ldcg(p + 4), __ldcg(p + 8), __ldcg(p + 12));
    }
    __syncthreads();
}

// Residuals (fill_r_DepthKernel / fill_r_MRegKernel, src/MotionOptimization.cu:163-227) with
// the transforms T; partial FP64 energies of this thread (runSquareKernel + reductions,
// src/VolumeFusion.cu:575-588).
template <bool kStaged>
AFX_D void gn_residuals(const GnArgs& a, const float* warped, const NodeT<kStaged>& T, int n, long ncorr, long gt,
                        long gstride, double (&e2)[2]) {
    const GnBuffers& b = a.b;
    const long nreg = (long)n * a.kreg;
    constexpr int kAhead = 4;  // correspondences whose loads are in flight together
    for (long c0 = gt; c0 < ncorr; c0 += kAhead * gstride) {
        long v[kAhead], px[kAhead];
        float d[kAhead][3], nr[kAhead][3];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const long c = c0 + k * gstride < ncorr ? c0 + k * gstride : c0;
            v[k] = a.corr[2 * c];
            px[k] = a.corr[2 * c + 1];
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                d[k][ax] = __ldcg(warped + 3 * v[k] + ax) - a.frame[3 * px[k] + ax];
                nr[k][ax] = a.normals[3 * px[k] + ax];
            }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const long c = c0 + k * gstride;
            if (c >= ncorr) break;
            const float r = a.lam_d * dot3(nr[k], d[k]);
            __stcg(b.rdepth + c, r);
            e2[0] += (double)(r * r);
        }
    }
    for (long t = gt; t < nreg; t += gstride) {
        const int i = (int)(t / a.kreg);
        const uint32_t nb = a.gidx[t];
        float* rr = b.rreg + 3 * t;
        if (nb >= (uint32_t)n) {
            __stcg(rr, 0.f);
            __stcg(rr + 1, 0.f);
            __stcg(rr + 2, 0.f);
            continue;
        }
        float Ti[16], Tn[16], tc[3], tn[3];
        T.load((uint32_t)i, Ti);
        T.load(nb, Tn);
        mat4_point(Ti, a.nodes + 3 * (long)i, tc);
        mat4_point(Tn, a.nodes + 3 * (long)i, tn);
        for (int ax = 0; ax < 3; ++ax) {
            const float r = (tc[ax] - tn[ax]) * a.lam_r;
            __stcg(rr + ax, r);
            e2[1] += (double)(r * r);
        }
    }
}

// J^T r of every node into b.jtr (one node per warp).
AFX_D void gn_jtr(const GnArgs& a, int n, int gw, int nw) {
    const int lane = threadIdx.x & 31;
    for (int node = gw; node < n; node += nw) {
        float jv[6];
        jtr_node(a, node, n, jv);
        if (lane < 6) {
            float ji = jv[0];
#pragma unroll
            for (int q = 1; q < 6; ++q)
                if (lane == q) ji = jv[q];
            __stcg(a.b.jtr + (long)node * 6 + lane, ji);
        }
    }
}

// ---- PCG with the vectors in shared memory and the matrix where it fits ----
//
// For graphs past the path above: each CTA owns a contiguous node range and keeps in shared memory
// a full copy of the search direction, its own x, r and A p, its rows' neighbours, and as many of
// its blocks as there is room for (staged once per Gauss-Newton loop); the rest are read from L2.
// z travels through global memory: the CTA writes its slice before the barrier of the r.z sum,
// and after it every CTA forms p = z + beta p over all nodes, so an iteration has two cluster
// barriers.
// Bound: for 1,500 nodes the chain of barriers and sums, for 5,000 the blocks from L2 (16 SMs).
// 1,500 nodes, ten iterations: 103 us; 119 us with all blocks read from shared memory in each, and
// 298 us with all vectors in global memory (three barriers, one dependent load after the other).
constexpr int kWideFloats = kDsNodes * 12 + 3 * kDsNpc * 6 + kDsNpc * 36 + kDsBlocks * 36;  // the room from d.z on

struct WideLayout {
    float *pf, *x, *r, *ap;
    int *rowptr, *col;  // col: null where the neighbours did not fit
    float* blk;
    int cap;            // blocks [0, cap) of the CTA are in shared memory
};

AFX_D bool wide_fits(int n, int ncta) {
    const int npc = (n + ncta - 1) / ncta;
    return ((long)n * 6 + 3) / 4 * 4 + (long)npc * 19 + 1 <= kWideFloats;
}

AFX_D WideLayout wide_layout(float* room, int n, int npc) {
    WideLayout d;
    d.pf = room;
    d.x = room + (n * 6 + 3) / 4 * 4;
    d.r = d.x + npc * 6;
    d.ap = d.r + npc * 6;
    d.rowptr = reinterpret_cast<int*>(d.ap + npc * 6);
    return d;
}

// Row pointers, neighbours and blocks of the own rows; the layout is the same on later calls (`stage` false).
AFX_D void wide_stage(const GnBuffers& b, WideLayout& d, float* room, int start, int own, bool stage) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (stage) stage_rowptr(b, d.rowptr, start, own);
    const int nblk = d.rowptr[own];
    float* p = reinterpret_cast<float*>(d.rowptr + own + 1);
    float* const end = room + kWideFloats;
    d.col = nblk <= end - p ? reinterpret_cast<int*>(p) : nullptr;
    if (d.col) p += nblk;
    p = room + ((p - room) + 3) / 4 * 4;
    d.blk = p;
    d.cap = p < end ? min(nblk, (int)((end - p) / 36)) : 0;
    if (!stage) return;
    for (int li = w; li < own; li += kLoopWarps) {
        const long node = start + li;
        const int r0 = d.rowptr[li], cnt = d.rowptr[li + 1] - r0 - 1;
        if (d.col) {
            if (lane == 0) d.col[r0] = (int)node;
            for (int u = lane; u < cnt; u += 32) stage_word(d.col + r0 + 1 + u, b.nbr + node * kMaxNbr + u);
        }
        const int in = min(cnt + 1, max(0, d.cap - r0)) * 9;
        for (int e = lane; e < in; e += 32)
            stage_quad(d.blk + (long)r0 * 36 + e * 4, e < 9 ? b.diag + node * 36 + e * 4 : b.blocks + node * kMaxNbr * 36 + (e - 9) * 4);
    }
    stage_wait();
    __syncthreads();
}

// A p of the own rows from `first` on, into d.ap, and this thread's part of p.Ap.  kR lanes per row: each
// multiplies one of kR blocks and the products are added in block order in every lane, as one lane alone would.
template <int kR>
AFX_D void wide_spmv(const GnBuffers& b, const WideLayout& d, int start, int own, int first, TF& pap) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, part = lane % kR, cnt = own * 6;
    constexpr int kRows = 32 / kR;      // per warp
    constexpr int kH = kR == 1 ? 4 : 2;  // blocks of a lane in flight
    for (int base = first + w * kRows; base < cnt; base += kLoopWarps * kRows) {
        const int row = base + lane / kR;
        const bool on = row < cnt;
        const int li = on ? row / 6 : 0, i = on ? row - 6 * li : 0;
        const int r0 = d.rowptr[li], nb = on ? d.rowptr[li + 1] - r0 : 0;
        const int most = __reduce_max_sync(0xffffffffu, nb);
        float acc = 0.f;
        auto add = [&](const float2 (&B)[kH][3], const int (&c)[kH], int k0) {
            float s[kH];
#pragma unroll
            for (int h = 0; h < kH; ++h) {
                const float2* xv = reinterpret_cast<const float2*>(d.pf) + c[h] * 3;
                s[h] = 0.f;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const float2 x = xv[q];
                    s[h] = s[h] + B[h][q].x * x.x;
                    s[h] = s[h] + B[h][q].y * x.y;
                }
            }
#pragma unroll
            for (int h = 0; h < kH; ++h)
#pragma unroll
                for (int q = 0; q < kR; ++q) {
                    const float sq = kR == 1 ? s[h] : __shfl_sync(0xffffffffu, s[h], (lane & ~(kR - 1)) + q);
                    if (k0 + kR * h + q < nb) acc = acc + sq;
                }
        };
        if (__all_sync(0xffffffffu, r0 + nb <= d.cap) && d.col) {
            const float2* Bp = reinterpret_cast<const float2*>(d.blk) + r0 * 18 + i * 3;
            const int* cp = d.col + r0;
            for (int k0 = 0; k0 < most; k0 += kR * kH) {
                float2 B[kH][3];
                int c[kH];
#pragma unroll
                for (int h = 0; h < kH; ++h) {
                    const int u = k0 + kR * h + part < nb ? k0 + kR * h + part : 0;
                    c[h] = cp[u];
#pragma unroll
                    for (int q = 0; q < 3; ++q) B[h][q] = Bp[u * 18 + q];
                }
                add(B, c, k0);
            }
        } else {
            const long node = start + li;
            for (int k0 = 0; k0 < most; k0 += kR * kH) {
                float2 B[kH][3];
                int c[kH];
#pragma unroll
                for (int h = 0; h < kH; ++h) {
                    const int u = k0 + kR * h + part < nb ? k0 + kR * h + part : 0;
                    c[h] = d.col ? d.col[r0 + u] : (u ? b.nbr[node * kMaxNbr + u - 1] : (int)node);
                    const float2* src =
                        reinterpret_cast<const float2*>((u ? b.blocks + (node * kMaxNbr + u - 1) * 36 : b.diag + node * 36) + i * 6);
#pragma unroll
                    for (int q = 0; q < 3; ++q) B[h][q] = __ldg(src + q);
                }
                add(B, c, k0);
            }
        }
        if (on && part == 0) {
            d.ap[row] = acc;
            pap = tf_add_prod(pap, d.pf[start * 6 + row], acc);
        }
    }
}

template <bool kTol>
AFX_D void pcg_wide(const LoopArgs& L, int n, float* room, ClusterSums& cs, bool stage) {
    const GnBuffers& b = L.g.b;
    const unsigned rank = cluster_rank(), ncta = cluster_size();
    const int npc = (n + (int)ncta - 1) / (int)ncta;
    const int start = min(n, (int)rank * npc), own = min(n, start + npc) - start, cnt = own * 6;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int grp = lane / 6, ei = lane - 6 * grp;
    WideLayout d = wide_layout(room, n, npc);
    wide_stage(b, d, room, start, own, stage);
    constexpr int NV = kTol ? 2 : 1;
    TF sum[NV];
    DF tot[NV];
    // r -= alpha A p, x += alpha p (first: x = 0, r = b), z = M^-1 r to global memory, r.z (and r.r);
    // kAhead nodes of a lane group at a time, so that their loads are in flight together
    auto update = [&](bool first, float alpha) {
        constexpr int kAhead = 3;
#pragma unroll
        for (int i = 0; i < NV; ++i) sum[i] = {0.f, 0.f, 0.f};
        for (int base = w * 5; base < own; base += kAhead * kLoopWarps * 5) {
            float rv[kAhead];
            float2 M[kAhead][3];
            bool act[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
                const int li = base + k * kLoopWarps * 5 + grp;
                act[k] = lane < 30 && li < own;
                const float2* Mi = reinterpret_cast<const float2*>(b.minv + (long)(act[k] ? start + li : 0) * 36 + ei * 6);
#pragma unroll
                for (int q = 0; q < 3; ++q) M[k][q] = lane < 30 ? Mi[q] : make_float2(0.f, 0.f);
                const int o = li * 6 + ei;
                rv[k] = 0.f;
                if (!act[k]) continue;
                if (first) {
                    d.x[o] = 0.f;
                    rv[k] = __ldcg(b.jtr + (long)start * 6 + o);
                } else {
                    d.x[o] = d.x[o] + alpha * d.pf[start * 6 + o];
                    rv[k] = d.r[o] - alpha * d.ap[o];
                }
                d.r[o] = rv[k];
            }
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
                const int li = base + k * kLoopWarps * 5 + grp;
                float rq[6], zi = 0.f;
#pragma unroll
                for (int q = 0; q < 6; ++q) rq[q] = __shfl_sync(0xffffffffu, rv[k], lane < 30 ? grp * 6 + q : q);
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    zi = zi + M[k][q].x * rq[2 * q];
                    zi = zi + M[k][q].y * rq[2 * q + 1];
                }
                if (!act[k]) continue;
                __stcg(b.z + (long)(start + li) * 6 + ei, zi);
                sum[0] = tf_add_prod(sum[0], rv[k], zi);
                if constexpr (kTol) sum[NV - 1] = tf_add_prod(sum[NV - 1], rv[k], rv[k]);
            }
        }
        cluster_sum_tf<NV>(sum, tot, cs);
    };
    update(true, 0.f);
    // a thread keeps the first blocks of one of the first rows in registers for the whole solve
    constexpr int kRowBlocks = 6;
    const int row = threadIdx.x, re = row % 6;
    const int r0 = row < cnt ? d.rowptr[row / 6] : 0, nb = row < cnt ? d.rowptr[row / 6 + 1] - r0 : 0;
    auto block_row = [&](int u, int& c) {
        const long node = start + row / 6;
        c = d.col ? d.col[r0 + u] : (u ? b.nbr[node * kMaxNbr + u - 1] : (int)node);
        const float* B = r0 + u < d.cap ? d.blk + (r0 + u) * 36
                                        : (u ? b.blocks + (node * kMaxNbr + u - 1) * 36 : b.diag + node * 36);
        return reinterpret_cast<const float2*>(B + re * 6);
    };
    float2 A[kRowBlocks][3];
    int off[kRowBlocks];  // in float2
#pragma unroll
    for (int k = 0; k < kRowBlocks; ++k) {
        off[k] = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) A[k][q] = make_float2(0.f, 0.f);
        if (k >= nb) continue;
        int c;
        const float2* src = block_row(k, c);
        off[k] = c * 3;
#pragma unroll
        for (int q = 0; q < 3; ++q) A[k][q] = src[q];
    }
    DF rz = tot[0];
    const float tol2 = kTol ? (float)(L.tol * L.tol) : 0.f, bn = tot[NV - 1].hi;
    float beta = 0.f;
    for (int it = 0; it < L.pcg_iters; ++it) {
        // p = z (first iteration) or z + beta p for all nodes
        const float4* z4 = reinterpret_cast<const float4*>(b.z);
        float4* p4 = reinterpret_cast<float4*>(d.pf);
        constexpr int kBatch = 6;
        for (int i0 = threadIdx.x; i0 < n * 6 / 4; i0 += kBatch * kLoopThreads) {
            float4 v[kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const int i = i0 + q * kLoopThreads;
                v[q] = __ldcg(z4 + (i < n * 6 / 4 ? i : i0));
            }
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const int i = i0 + q * kLoopThreads;
                if (i >= n * 6 / 4) break;
                if (it) {
                    const float4 o = p4[i];
                    v[q] = make_float4(v[q].x + beta * o.x, v[q].y + beta * o.y, v[q].z + beta * o.z, v[q].w + beta * o.w);
                }
                p4[i] = v[q];
            }
        }
        for (int i = n * 6 / 4 * 4 + threadIdx.x; i < n * 6; i += kLoopThreads) {
            const float zi = __ldcg(b.z + i);
            d.pf[i] = it ? zi + beta * d.pf[i] : zi;
        }
        __syncthreads();
        TF pap[1] = {{0.f, 0.f, 0.f}};
        DF tp[1];
        if (row < cnt) {
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < kRowBlocks; ++k) {
                const float2* xv = reinterpret_cast<const float2*>(d.pf) + off[k];
                float s = 0.f;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const float2 x = xv[q];
                    s = s + A[k][q].x * x.x;
                    s = s + A[k][q].y * x.y;
                }
                if (k < nb) acc = acc + s;
            }
#pragma unroll 2
            for (int u = kRowBlocks; u < nb; ++u) {
                int c;
                const float2* src = block_row(u, c);
                const float2* xv = reinterpret_cast<const float2*>(d.pf) + c * 3;
                float s = 0.f;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const float2 B = src[q], x = xv[q];
                    s = s + B.x * x.x;
                    s = s + B.y * x.y;
                }
                acc = acc + s;
            }
            d.ap[row] = acc;
            pap[0] = tf_add_prod(pap[0], d.pf[start * 6 + row], acc);
        }
        // further rows: four lanes each while two passes take them all, else one (ten iterations, four lanes and one: 1,500
        // nodes, 52 rows, 96 and 105 us; 2,000, 238 rows, 110 both; 2,100, 280 rows, 125 and 115; 5,300 248 and 221)
        if (cnt - kLoopThreads > 2 * kLoopThreads / 4) wide_spmv<1>(b, d, start, own, kLoopThreads, pap[0]);
        else wide_spmv<4>(b, d, start, own, kLoopThreads, pap[0]);
        cluster_sum_tf<1>(pap, tp, cs);
        if (df_zero_or_nan(tp[0])) break;
        update(false, df_quotient(rz, tp[0]));
        beta = df_quotient(tot[0], rz);
        rz = tot[0];
        if (kTol && tot[NV - 1].hi <= tol2 * bn) break;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < cnt; t += kLoopThreads) __stcg(b.x + (long)start * 6 + t, d.x[t]);
}

// PCG with the vectors in global memory, for graphs whose search direction does not fit in shared memory
// either (past kWideFloats, about 7,300 nodes); J^T r from b.jtr, solution in b.x.  Same
// recurrences and arithmetic as pcg_wide.
__device__ __noinline__ void pcg_global(const LoopArgs& L, int n, ClusterSums& cs) {
    const GnBuffers& b = L.g.b;
    const unsigned rank = cluster_rank(), ncta = cluster_size();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gw = (int)rank * kLoopWarps + w, nw = (int)ncta * kLoopWarps;
    const int grp = lane / 6, ei = lane - 6 * grp;
    const bool glane = lane < 30;
    const int gstep = nw * 5;
    // x = 0, r = b, z = M^-1 r; rz = r.z, bb = b.b
    TF d2[2] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    DF tot[2], tp[1];
    for (int base = gw * 5; base < n; base += gstep) {  // warp-uniform trip count
        const int node = base + grp;
        const bool act = glane && node < n;
        const long o = (long)node * 6 + ei;
        const float ji = act ? __ldcg(b.jtr + o) : 0.f;
        float zi = 0.f;
        const float* Mi = b.minv + (long)(act ? node : 0) * 36 + ei * 6;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const float rq = __shfl_sync(0xffffffffu, ji, glane ? grp * 6 + q : q);
            if (act) zi = zi + Mi[q] * rq;
        }
        if (act) {
            __stcg(b.x + o, 0.f);
            __stcg(b.r + o, ji);
            __stcg(b.z + o, zi);
            d2[0] = tf_add_prod(d2[0], ji, zi);
            d2[1] = tf_add_prod(d2[1], ji, ji);
        }
    }
    cluster_sum_tf<2>(d2, tot, cs);
    // six lanes per node (entry i = lane % 6 of node group lane / 6, five groups per warp)
    DF rz = tot[0];
    const DF bnorm2 = tot[1];
    const float tol2 = L.tol > 0 ? (float)(L.tol * L.tol) : 0.f;
    float beta = 0.f;
    for (int it = 0; it < L.pcg_iters; ++it) {
        // p = z (first iteration) or z + beta p for the own entries, then A p once all are written
        for (int base = gw * 5; base < n; base += gstep) {
            const int node = base + grp;
            if (glane && node < n) {
                const long o = (long)node * 6 + ei;
                const float zi = __ldcg(b.z + o);
                __stcg(b.p + o, it ? zi + beta * __ldcg(b.p + o) : zi);
            }
        }
        cluster_barrier();
        TF pap[1] = {{0.f, 0.f, 0.f}};
        if (glane)
            for (int node = gw * 5 + grp; node < n; node += gstep) {
                const long o = (long)node * 6 + ei;
                const float api = spmv_entry(b, node, ei, b.p);
                __stcg(b.ap + o, api);
                pap[0] = tf_add_prod(pap[0], __ldcg(b.p + o), api);
            }
        cluster_sum_tf<1>(pap, tp, cs);
        if (df_zero_or_nan(tp[0])) break;
        const float alpha = df_quotient(rz, tp[0]);
        // x += alpha p; r -= alpha A p; z = M^-1 r; r.z, r.r
        TF q2[2] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
        for (int base = gw * 5; base < n; base += gstep) {
            const int node = base + grp;
            const bool act = glane && node < n;
            const long o = (long)node * 6 + ei;
            float rv = 0.f;
            if (act) {
                __stcg(b.x + o, __ldcg(b.x + o) + alpha * __ldcg(b.p + o));
                rv = __ldcg(b.r + o) - alpha * __ldcg(b.ap + o);
                __stcg(b.r + o, rv);
            }
            float zi = 0.f;
            const float* Mi = b.minv + (long)(act ? node : 0) * 36 + ei * 6;
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const float rq = __shfl_sync(0xffffffffu, rv, glane ? grp * 6 + q : q);
                if (act) zi = zi + Mi[q] * rq;
            }
            if (act) {
                __stcg(b.z + o, zi);
                q2[0] = tf_add_prod(q2[0], rv, zi);
                q2[1] = tf_add_prod(q2[1], rv, rv);
            }
        }
        cluster_sum_tf<2>(q2, tot, cs);
        beta = df_quotient(tot[0], rz);
        rz = tot[0];
        if (L.tol > 0 && tot[1].hi <= tol2 * bnorm2.hi) break;
    }
}

// T -= [[x_rot]x, x_t; 0] for nodes [lo, hi) with x in global memory (updateTransformsKernel,
// src/MotionOptimization.cu:483-498); entry e of node i by thread (i - lo) * 16 + e.
AFX_D void update_transforms_range(float* T, const float* x, int lo, int hi, long t0, long tstride) {
    for (long t = t0; t < (long)(hi - lo) * 16; t += tstride) {
        const long node = lo + t / 16;
        const int e = (int)(t & 15);
        const float* u = x + node * 6;
        float U;
        switch (e) {
            case 1: U = __ldcg(u + 2); break;
            case 2: U = -__ldcg(u + 1); break;
            case 4: U = -__ldcg(u + 2); break;
            case 6: U = __ldcg(u + 0); break;
            case 8: U = __ldcg(u + 1); break;
            case 9: U = -__ldcg(u + 0); break;
            case 12: U = __ldcg(u + 3); break;
            case 13: U = __ldcg(u + 4); break;
            case 14: U = __ldcg(u + 5); break;
            default: U = 0.f;
        }
        float* Te = T + node * 16 + e;
        __stcg(Te, __ldcg(Te) - U);
    }
}

// Canonical vertices warped by T (warpKernel, src/ComputeCorrespondence.cu:13-30, or the dual-quaternion
// blend of afx_dqb.cuh).
template <bool kStaged>
AFX_D void gn_rewarp(const GnArgs& a, const float* points, float* warped, const NodeT<kStaged>& T, long m, long gt,
                     long gstride) {
    if (a.blend == AFX_BLEND_DQB) {
        for (long i = gt; i < m; i += gstride) {
            const float p[3] = {points[3 * i], points[3 * i + 1], points[3 * i + 2]};
            float o[3];
            dq_blend_point([&](uint32_t nb, float(&Tn)[16]) { T.load(nb, Tn); }, a.midx + i * a.k, a.mw + i * a.k, a.k,
                           AFX_INVALID_INDEX, p, o);
            __stcg(warped + 3 * i, o[0]);
            __stcg(warped + 3 * i + 1, o[1]);
            __stcg(warped + 3 * i + 2, o[2]);
        }
        return;
    }
    // one neighbour's part of a point's sum
    auto blend = [&](const float (&p)[3], uint32_t nb, float wj, float (&acc)[3]) {
        if (nb == AFX_INVALID_INDEX) return;
        float Tn[16], o[3];
        T.load(nb, Tn);
        mat4_point(Tn, p, o);
        acc[0] = acc[0] + wj * o[0];
        acc[1] = acc[1] + wj * o[1];
        acc[2] = acc[2] + wj * o[2];
    };
    auto finish = [&](long i, const float (&p)[3], bool zero, const float (&acc)[3]) {
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) __stcg(warped + 3 * i + ax, zero ? p[ax] : acc[ax]);
    };
    if (kStaged && a.k == 4 && !(((size_t)a.midx | (size_t)a.mw) & 15)) {
        // four neighbours, rows on 16 bytes: whole rows, and the loads of several points in flight together
        constexpr int kAhead = 4;
        for (long i0 = gt; i0 < m; i0 += kAhead * gstride) {
            float p[kAhead][3];
            uint4 nb[kAhead];
            float4 w[kAhead];
#pragma unroll
            for (int q = 0; q < kAhead; ++q) {
                const long i = i0 + q * gstride < m ? i0 + q * gstride : i0;
                nb[q] = reinterpret_cast<const uint4*>(a.midx)[i];
                w[q] = reinterpret_cast<const float4*>(a.mw)[i];
#pragma unroll
                for (int ax = 0; ax < 3; ++ax) p[q][ax] = points[3 * i + ax];
            }
#pragma unroll
            for (int q = 0; q < kAhead; ++q) {
                const long i = i0 + q * gstride;
                if (i >= m) break;
                const bool zero = fabsf(w[q].x) <= 1e-5f && fabsf(w[q].y) <= 1e-5f && fabsf(w[q].z) <= 1e-5f &&
                                  fabsf(w[q].w) <= 1e-5f;
                float acc[3] = {0.f, 0.f, 0.f};
                if (!zero) {
                    blend(p[q], nb[q].x, w[q].x, acc);
                    blend(p[q], nb[q].y, w[q].y, acc);
                    blend(p[q], nb[q].z, w[q].z, acc);
                    blend(p[q], nb[q].w, w[q].w, acc);
                }
                finish(i, p[q], zero, acc);
            }
        }
        return;
    }
    for (long i = gt; i < m; i += gstride) {
        const float p[3] = {points[3 * i], points[3 * i + 1], points[3 * i + 2]};
        bool zero = true;
        for (int j = 0; j < a.k; ++j)
            if (!(fabsf(a.mw[i * a.k + j]) <= 1e-5f)) zero = false;
        float acc[3] = {0.f, 0.f, 0.f};
        if (!zero)
            for (int j = 0; j < a.k; ++j) blend(p, a.midx[i * a.k + j], a.mw[i * a.k + j], acc);
        finish(i, p, zero, acc);
    }
}

// One solve from b.jtr: x in b.x (and in the own slices of the shared-memory layout); with
// L.T_pending set, T_pending -= [x] as well.  Ends with a cluster barrier, after which every CTA knows whether a
// wait ran out.
// `first`: the first solve of the launch.
AFX_D void gn_solve(const LoopArgs& L, int n, bool ds, const DsLayout& dsl, ClusterSums& cs, DsExchange& ex, long gt,
                    long gstride, bool first) {
    if (ds) {
        if (!ex.dead) {
            if (L.tol > 0) pcg_ds<true>(L, n, dsl, ex);
            else pcg_ds<false>(L, n, dsl, ex);
        }
        if (ex.dead && threadIdx.x < cluster_size()) dsmem_store_int(&cs.dead, threadIdx.x, 1);
    } else {
        if (!wide_fits(n, (int)cluster_size())) pcg_global(L, n, cs);
        else if (L.tol > 0) pcg_wide<true>(L, n, dsl.z, cs, first);
        else pcg_wide<false>(L, n, dsl.z, cs, first);
        cluster_barrier();  // x complete
        if (L.T_pending) update_transforms_range(L.T_pending, L.g.b.x, 0, n, gt, gstride);
    }
    cluster_barrier();
    if (ds) ex.dead = cs.dead != 0;
}

__global__ void __launch_bounds__(kLoopThreads, 1) gn_loop_kernel(LoopArgs L) {
    const GnArgs& a = L.g;
    const GnBuffers& b = a.b;
    __shared__ ClusterSums cs;
    extern __shared__ __align__(16) double ds_smem[];
    const DsLayout dsl = ds_layout(ds_smem);
    if (threadIdx.x == 0) {
        cs.phase = 0;
        cs.dead = 0;
        ds_exchange_init(dsl);
    }
    // Every CTA of the cluster must be running before any thread touches another CTA's shared
    // memory (the first such store is in ds_stage).  Under load the CTAs of a cluster need not
    // start together; a store into a CTA that has not started is an SM fault.
    cluster_barrier();
    const unsigned rank = cluster_rank(), ncta = cluster_size();
    const int w = threadIdx.x >> 5;
    const long gt = (long)rank * kLoopThreads + threadIdx.x, gstride = (long)ncta * kLoopThreads;
    // nodes dealt to the CTAs in turn: a small graph's fill every CTA alike
    const int gw = w * (int)ncta + (int)rank, nw = (int)ncta * kLoopWarps;
    const bool leader = rank == 0 && threadIdx.x == 0;
    const int n = min(*a.n_nodes, a.n_max);
    const long ncorr = min((long)*a.corr_count, a.c_max);
    const long m = min((long)*a.mesh_count, a.m_max);
    GnState* s = b.state;
    double e_prev = s->e_prev;
    bool done = s->done != 0;
    // small graphs: the system lives in distributed shared memory for the whole loop
    int ds_ph = 0;
    DsExchange ex{{0u, 0u}, false};
    const bool ds = !done && n > 0 && (n + (int)ncta - 1) / (int)ncta <= kDsNpc && ds_stage(b, n, dsl, cs, ds_ph);
    const NodeT<true> Ts{L.T_pending, reinterpret_cast<const float4*>(dsl.z), n};
    const NodeT<false> Tg{L.T_pending, nullptr, n};
    if (ds) stage_node_T(L.T_pending, n, dsl);
    for (int iter = 0; iter < L.gn_iters && !done; ++iter) {
        double e2[2] = {0.0, 0.0};
        if (ds) gn_residuals(a, L.warped, Ts, n, ncorr, gt, gstride, e2);
        else gn_residuals(a, L.warped, Tg, n, ncorr, gt, gstride, e2);
        cluster_sum_pair(e2, cs);
        // ---- energy test and commit decision (src/VolumeFusion.cu:589-598)
        const double e = e2[0] + e2[1];
        if (leader) {
            s->e_last = e;
            s->e_depth = e2[0];
            s->e_reg = e2[1];
        }
        if (e_prev - e < (double)a.min_step) {
            if (leader) s->done = 1;
            done = true;
            break;
        }
        e_prev = e;
        const bool commit = iter != 0;
        if (leader) {
            s->e_prev = e;
            s->commit = commit;
            s->iters = iter + 1;
        }
        if (commit)
            for (long t = gstride - 1 - gt; t < (long)n * 16; t += gstride) L.T_committed[t] = __ldcg(L.T_pending + t);
        gn_jtr(a, n, gw, nw);
        cluster_barrier();
        gn_solve(L, n, ds, dsl, cs, ex, gt, gstride, iter == 0);
        if (ds) {
            stage_node_T(L.T_pending, n, dsl);
            gn_rewarp(a, L.points, L.warped, Ts, m, gt, gstride);
        } else {
            gn_rewarp(a, L.points, L.warped, Tg, m, gt, gstride);
        }
        cluster_barrier();
    }
    // no CTA leaves while another may still read its shared memory
    cluster_barrier();
}

// One PCG solve of a system assembled by afx_gn_build (J^T J blocks, inverses and J^T r in the
// workspace); x in b.x.
__global__ void __launch_bounds__(kLoopThreads, 1) gn_solve_kernel(LoopArgs L) {
    const GnArgs& a = L.g;
    __shared__ ClusterSums cs;
    extern __shared__ __align__(16) double ds_smem[];
    const DsLayout dsl = ds_layout(ds_smem);
    if (threadIdx.x == 0) {
        cs.phase = 0;
        cs.dead = 0;
        ds_exchange_init(dsl);
    }
    cluster_barrier();  // every CTA running before any access to another CTA's shared memory
    const unsigned rank = cluster_rank(), ncta = cluster_size();
    const long gt = (long)rank * kLoopThreads + threadIdx.x, gstride = (long)ncta * kLoopThreads;
    const int n = min(*a.n_nodes, a.n_max);
    int ds_ph = 0;
    DsExchange ex{{0u, 0u}, false};
    const bool ds = n > 0 && (n + (int)ncta - 1) / (int)ncta <= kDsNpc && ds_stage(a.b, n, dsl, cs, ds_ph);
    gn_solve(L, n, ds, dsl, cs, ex, gt, gstride, true);
    // no CTA leaves while another may still read its shared memory
    cluster_barrier();
}

}  // namespace afx

// ------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------

namespace afx {

struct GnSizes {
    long m_max;
    int n_max, k, kreg;
};

static size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

// Cluster size for gn_loop_kernel: 16 CTAs where the device runs non-portable clusters of
// that size, else the portable 8.
static int gn_cluster_size() {
    static ContextOnce once;
    static int cached_dev[kMaxDevices];
    once_per_context(once, [](int dev) {
        int cached = 0;
        cudaFuncSetAttribute(gn_loop_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaFuncSetAttribute(gn_loop_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDsSmem);
        cudaFuncSetAttribute(gn_solve_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaFuncSetAttribute(gn_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDsSmem);
        const int sizes[2] = {16, 8};
        for (int c : sizes) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(c);
            cfg.blockDim = dim3(kLoopThreads);
            cfg.dynamicSmemBytes = kDsSmem;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = c;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, gn_loop_kernel, &cfg) == cudaSuccess && clusters > 0) {
                cached = c;
                break;
            }
            cudaGetLastError();
        }
        cached_dev[dev] = cached ? cached : 8;
        return (int)AFX_OK;
    });
    int dev = 0;
    cudaGetDevice(&dev);
    return cached_dev[dev] ? cached_dev[dev] : 8;
}

size_t gn_workspace_size(long m_max, int n_max, int k, int kreg) {
    size_t s = 0;
    s += 3 * al((n_max + 1) * 4) + al(m_max * k * 4);           // lcnt loff lcur lst
    s += 3 * al((n_max + 1) * 4) + al((size_t)n_max * kreg * 4);  // icnt ioff icur ilst
    s += al(n_max * 4) + al((size_t)n_max * kMaxNbr * 4);         // nbr_cnt nbr
    s += al((size_t)n_max * kMaxNbr * 36 * 4) + al((size_t)n_max * 36 * 4) + al((size_t)n_max * 36 * 4);
    s += al((size_t)m_max * k * 6 * 4) + al((size_t)m_max * k * 4);  // jrow jc
    s += al((size_t)n_max * 6 * 4) * 6;                           // jtr x r z p ap
    s += al(m_max * 4) + al((size_t)n_max * kreg * 3 * 4);        // rdepth rreg
    s += al(sizeof(GnState));
    return s + 1024;
}

bool gn_carve(void* ws, size_t bytes, long m_max, int n_max, int k, int kreg, GnBuffers* b) {
    if (!ws || bytes < gn_workspace_size(m_max, n_max, k, kreg)) return false;
    char* p = static_cast<char*>(ws);
    auto take = [&](size_t n) {
        char* q = p;
        p += al(n);
        return q;
    };
    b->lcnt = (unsigned*)take((n_max + 1) * 4);  // the four counters together: cleared as one
    b->lcur = (unsigned*)take((n_max + 1) * 4);
    b->icnt = (unsigned*)take((n_max + 1) * 4);
    b->icur = (unsigned*)take((n_max + 1) * 4);
    b->loff = (unsigned*)take((n_max + 1) * 4);
    b->lst = (unsigned*)take(m_max * k * 4);
    b->ioff = (unsigned*)take((n_max + 1) * 4);
    b->ilst = (unsigned*)take((size_t)n_max * kreg * 4);
    b->nbr_cnt = (int*)take(n_max * 4);
    b->nbr = (int*)take((size_t)n_max * kMaxNbr * 4);
    b->blocks = (float*)take((size_t)n_max * kMaxNbr * 36 * 4);
    b->diag = (float*)take((size_t)n_max * 36 * 4);
    b->minv = (float*)take((size_t)n_max * 36 * 4);
    b->jrow = (float*)take((size_t)m_max * k * 6 * 4);
    b->jc = (int*)take((size_t)m_max * k * 4);
    b->jtr = (float*)take((size_t)n_max * 6 * 4);
    b->x = (float*)take((size_t)n_max * 6 * 4);
    b->r = (float*)take((size_t)n_max * 6 * 4);
    b->z = (float*)take((size_t)n_max * 6 * 4);
    b->p = (float*)take((size_t)n_max * 6 * 4);
    b->ap = (float*)take((size_t)n_max * 6 * 4);
    b->rdepth = (float*)take(m_max * 4);
    b->rreg = (float*)take((size_t)n_max * kreg * 3 * 4);
    b->state = (GnState*)take(sizeof(GnState));
    return true;
}

constexpr int kNodeCtas = 608;  // CTAs that take one node at a time: four of 256 threads per SM

// Per frame: node -> vertex lists and incoming regularisation edges.
size_t gn_counter_words(int n_max) { return 4 * al((n_max + 1) * 4) / 4; }

int gn_frame_setup(const GnArgs& a, cudaStream_t st) {
    const GnBuffers& b = a.b;
    const long items = std::max(a.m_max * a.k, (long)a.n_max * a.kreg);
    list_scan_kernel<<<2, 1024, 0, st>>>(a);
    AFX_LAUNCH_CHECK();
    list_fill_kernel<<<grid_for(items, 256), 256, 0, st>>>(a);
    AFX_LAUNCH_CHECK();
    list_sort_kernel<<<std::min(a.n_max, kNodeCtas), 256, 0, st>>>(a);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// Per ICP iteration (after correspondences): J^T J structure, blocks and block inverses.
int gn_icp_setup(const GnArgs& a, float* T_pending, const float* T_committed, cudaStream_t st) {
    const int words = (a.n_max + 31) / 32;
    if (words > kGnMaxWords) return AFX_ERR_UNSUPPORTED;
    const size_t smem = asm_rows_bytes(a.k, words) + kAsmListBytes;
    static ContextOnce once;  // the opt-in covers every size accepted above
    int rc = once_per_context(once, [](int) {
        const int most = (int)(std::max(asm_rows_bytes(8, 0), (size_t)kGnMaxWords * 4) + kAsmListBytes);
        const cudaError_t e = cudaFuncSetAttribute(jtj_assemble_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return note_cuda_error(e);
        return note_cuda_error(cudaFuncSetAttribute(jtj_assemble_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    });
    if (rc) return rc;
    if (a.k <= 4) jtj_assemble_kernel<4><<<std::min(a.n_max, kNodeCtas), kAsmThreads, smem, st>>>(a);
    else jtj_assemble_kernel<8><<<std::min(a.n_max, kNodeCtas), kAsmThreads, smem, st>>>(a);
    AFX_LAUNCH_CHECK();
    const int half = std::min((a.n_max + 7) / 8, kNodeCtas);
    gn_icp_finish_kernel<<<half + grid_for((long)a.n_max * 32, 128), 128, 0, st>>>(
        a, reinterpret_cast<float4*>(T_pending), reinterpret_cast<const float4*>(T_committed), half);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

// All Gauss-Newton iterations of one ICP iteration (src/VolumeFusion.cu:571-691): one launch
// of gn_loop_kernel.  On return (stream order) T_committed holds the last accepted transforms,
// T_pending the last update and `warped` the canonical vertices warped by T_pending.
static int launch_cluster(void (*kernel)(LoopArgs), const LoopArgs& L, cudaStream_t st) {
    const int c = gn_cluster_size();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kLoopThreads);
    cfg.dynamicSmemBytes = kDsSmem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    AFX_CUDA(cudaLaunchKernelEx(&cfg, kernel, L));
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int gn_loop(const GnArgs& a, const float* points, float* warped, float* T_committed, float* T_pending, int gn_iters,
            int pcg_iters, double tol, cudaStream_t st) {
    if (gn_iters <= 0) return AFX_OK;
    LoopArgs L;
    L.g = a;
    L.points = points;
    L.warped = warped;
    L.T_committed = T_committed;
    L.T_pending = T_pending;
    L.gn_iters = gn_iters;
    L.pcg_iters = pcg_iters;
    L.tol = tol;
    L.wait_polls = kDsWaitPolls;
    L.gave_up = nullptr;
    return launch_cluster(gn_loop_kernel, L, st);
}

}  // namespace afx

// ------------------------------------------------------------------------------------
// Stand-alone Gauss-Newton operators: residuals, J^T J / J^T r (exported in the reference's dense
// layout), the PCG solve and the transform update, for callers that drive the steps themselves.
// ------------------------------------------------------------------------------------

namespace afx {

// The start of a build in one launch (six copies and clears otherwise): the counts that later calls use, no error, no
// correspondence of any vertex, and the lists' counters at zero.
__global__ void gn_begin_kernel(unsigned* counts, const unsigned* n_points, const unsigned* n_corr, const int* n_nodes, int* error,
                                int* cov, long m_max, unsigned* counters, long words) {
    AFX_GRID_STRIDE(i, m_max) cov[i] = -1;
    AFX_GRID_STRIDE(i, words) counters[i] = 0u;
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    counts[0] = *n_points;
    counts[1] = *n_corr;
    counts[2] = (unsigned)*n_nodes;
    *error = 0;
}

// The correspondence of each vertex, and the lists' counts.
__global__ void gn_corr_of_vertex_kernel(const int* corr, const unsigned* n_corr, long c_max, int* cov, GnArgs a) {
    const long c = min((long)*n_corr, c_max);
    AFX_GRID_STRIDE(i, c) cov[corr[2 * i]] = (int)i;
    list_counts(a);
}

__global__ void __launch_bounds__(256) gn_residual_kernel(GnArgs a, const float* warped, const float* T) {
    const int n = min(*a.n_nodes, a.n_max);
    const long ncorr = min((long)*a.corr_count, a.c_max);
    double e2[2] = {0.0, 0.0};
    gn_residuals(a, warped, NodeT<false>{T, nullptr, n}, n, ncorr, blockIdx.x * (long)blockDim.x + threadIdx.x,
                 (long)gridDim.x * blockDim.x, e2);
}

__global__ void __launch_bounds__(256) gn_jtr_kernel(GnArgs a) {
    const int n = min(*a.n_nodes, a.n_max);
    const int gw = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5);
    gn_jtr(a, n, gw, (int)((gridDim.x * (long)blockDim.x) >> 5));
}

// Dense (6 n_host)^2 J^T J: diagonal blocks, upper blocks and their transposes (the layout
// fillJTJKernel writes over runInitIdentityKernel's identity).
__global__ void gn_dense_kernel(GnArgs a, int n_host, float* jtj) {
    const int n = min(min(*a.n_nodes, a.n_max), n_host);
    const long ld = 6L * n_host;
    const int lane = threadIdx.x & 31;
    for (long node = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5; node < n;
         node += (gridDim.x * (long)blockDim.x) >> 5) {
        for (int e = lane; e < 36; e += 32) {
            const int i = e / 6, j = e % 6;
            jtj[(node * 6 + i) * ld + node * 6 + j] = a.b.diag[node * 36 + e];
        }
        const int cnt = a.b.nbr_cnt[node];
        for (int u = 0; u < cnt; ++u) {
            const long other = a.b.nbr[node * kMaxNbr + u];
            if (other <= node) continue;
            const float* B = a.b.blocks + (node * kMaxNbr + u) * 36;
            for (int e = lane; e < 36; e += 32) {
                const int i = e / 6, j = e % 6;
                jtj[(node * 6 + i) * ld + other * 6 + j] = B[e];
                jtj[(other * 6 + j) * ld + node * 6 + i] = B[e];
            }
        }
    }
}

__global__ void gn_copy_residuals_kernel(GnArgs a, float* r_depth, float* r_reg) {
    const int n = min(*a.n_nodes, a.n_max);
    const long ncorr = min((long)*a.corr_count, a.c_max);
    const long nreg = (long)n * a.kreg * 3;
    AFX_GRID_STRIDE(t, ncorr + nreg) {
        if (t < ncorr) {
            if (r_depth) r_depth[t] = __ldcg(a.b.rdepth + t);
        } else if (r_reg) {
            r_reg[t - ncorr] = __ldcg(a.b.rreg + (t - ncorr));
        }
    }
}

__global__ void update_transforms_kernel(float* T, const float* x, const int* n_nodes, int n_max) {
    const int n = min(*n_nodes, n_max);
    update_transforms_range(T, x, 0, n, blockIdx.x * (long)blockDim.x + threadIdx.x, (long)gridDim.x * blockDim.x);
}

}  // namespace afx

struct afx_gn {
    long m_max;
    int n_max, k, kreg;
    void* arena;
    afx::GnBuffers b;
    int* cov;
    int* error;
    unsigned* counts;  // copies of the caller's counters at build time: points, correspondences, nodes
    int* gave_up;      // pinned: set by a solve one of whose waits ran out, until afx_gn_status reports it
    int wait_polls;
    afx::GnArgs last;
    bool built;
};

using namespace afx;

extern "C" {

int afx_gn_create(long n_points_max, int n_nodes_max, int k, int kreg, afx_gn** out) {
    if (!out || n_points_max < 1 || n_nodes_max < 1 || k < 1 || k > 8 || kreg < 1 || kreg > 8)
        return AFX_ERR_INVALID_ARGUMENT;
    afx_gn* g = new (std::nothrow) afx_gn();
    if (!g) return AFX_ERR_NO_MEMORY;
    g->m_max = n_points_max;
    g->n_max = n_nodes_max;
    g->k = k;
    g->kreg = kreg;
    const size_t ws = gn_workspace_size(n_points_max, n_nodes_max, k, kreg);
    const size_t bytes = ws + al((size_t)n_points_max * 4) + 512;
    if (cudaMalloc(&g->arena, bytes) != cudaSuccess) {
        cudaGetLastError();
        delete g;
        return AFX_ERR_NO_MEMORY;
    }
    if (cudaHostAlloc(reinterpret_cast<void**>(&g->gave_up), sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(g->arena);
        delete g;
        return AFX_ERR_NO_MEMORY;
    }
    *g->gave_up = 0;
    g->wait_polls = kDsWaitPolls;
    gn_carve(g->arena, ws, n_points_max, n_nodes_max, k, kreg, &g->b);
    g->cov = reinterpret_cast<int*>(static_cast<char*>(g->arena) + ws);
    g->error = reinterpret_cast<int*>(static_cast<char*>(g->arena) + ws + al((size_t)n_points_max * 4));
    g->counts = reinterpret_cast<unsigned*>(static_cast<char*>(g->arena) + ws + al((size_t)n_points_max * 4) + 256);
    if (cudaMemset(g->error, 0, 4) != cudaSuccess) {
        cudaFreeHost(g->gave_up);
        cudaFree(g->arena);
        delete g;
        return note_cuda_error(cudaGetLastError());
    }
    g->built = false;
    *out = g;
    return AFX_OK;
}

int afx_gn_destroy(afx_gn* g) {
    if (!g) return AFX_ERR_INVALID_ARGUMENT;
    cudaDeviceSynchronize();
    cudaFreeHost(g->gave_up);
    cudaError_t e = cudaFree(g->arena);
    delete g;
    return note_cuda_error(e);
}

int afx_gn_set_wait_limit(afx_gn* g, int polls) {
    if (!g || polls < 0) return AFX_ERR_INVALID_ARGUMENT;
    g->wait_polls = polls;
    return AFX_OK;
}

int afx_gn_status(afx_gn* g, void* stream) {
    if (!g) return AFX_ERR_INVALID_ARGUMENT;
    AFX_CUDA(cudaStreamSynchronize(as_stream(stream)));
    volatile int* w = g->gave_up;
    if (!*w) return AFX_OK;
    *w = 0;
    return AFX_ERR_TIMEOUT;
}

int afx_gn_build(afx_gn* g, const float* canonical, const unsigned* n_points, const uint32_t* knn_idx,
                 const float* knn_weights, const int* corr, const unsigned* n_corr, const float* frame_vertices,
                 const float* frame_normals, const float* warped, const float* nodes, const float* transforms,
                 const int* n_nodes, const uint32_t* graph_idx, float lambda_depth, float lambda_reg, void* stream) {
    if (!g || !canonical || !n_points || !knn_idx || !knn_weights || !corr || !n_corr || !frame_vertices ||
        !frame_normals || !warped || !nodes || !transforms || !n_nodes || !graph_idx)
        return AFX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    const long words = (long)gn_counter_words(g->n_max);
    gn_begin_kernel<<<grid_for(std::max(g->m_max, words), 256), 256, 0, st>>>(g->counts, n_points, n_corr, n_nodes, g->error,
                                                                              g->cov, g->m_max, g->b.lcnt, words);
    AFX_LAUNCH_CHECK();
    // later calls use these copies, not the caller's counters
    n_points = g->counts;
    n_corr = g->counts + 1;
    n_nodes = reinterpret_cast<const int*>(g->counts + 2);
    GnArgs a;
    std::memset(&a, 0, sizeof(a));
    a.mesh = canonical;
    a.mesh_count = n_points;
    a.m_max = g->m_max;
    a.midx = knn_idx;
    a.mw = knn_weights;
    a.k = g->k;
    a.normals = frame_normals;
    a.frame = frame_vertices;
    a.corr = corr;
    a.corr_count = n_corr;
    a.c_max = g->m_max;
    a.corr_of_vertex = g->cov;
    a.nodes = nodes;
    a.n_nodes = n_nodes;
    a.n_max = g->n_max;
    a.gidx = graph_idx;
    a.kreg = g->kreg;
    a.lam_d = lambda_depth;
    a.lam_r = lambda_reg;
    a.b = g->b;
    a.error = g->error;
    gn_corr_of_vertex_kernel<<<grid_for(std::max(g->m_max * g->k, (long)g->n_max * g->kreg), 256), 256, 0, st>>>(
        corr, n_corr, g->m_max, g->cov, a);
    AFX_LAUNCH_CHECK();
    int rc = gn_frame_setup(a, st);
    if (rc) return rc;
    rc = gn_icp_setup(a, nullptr, nullptr, st);
    if (rc) return rc;
    gn_residual_kernel<<<grid_for(g->m_max + (long)g->n_max * g->kreg, 256), 256, 0, st>>>(a, warped, transforms);
    AFX_LAUNCH_CHECK();
    gn_jtr_kernel<<<grid_for((long)g->n_max * 32, 256), 256, 0, st>>>(a);
    AFX_LAUNCH_CHECK();
    g->last = a;
    g->built = true;
    int err = 0;
    AFX_CUDA(cudaMemcpyAsync(&err, g->error, 4, cudaMemcpyDeviceToHost, st));
    AFX_CUDA(cudaStreamSynchronize(st));
    if (err & ERRF_SINGULAR) return AFX_ERR_SINGULAR;
    if (err & ERRF_CAPACITY) return AFX_ERR_CAPACITY;
    return AFX_OK;
}

int afx_gn_export(afx_gn* g, int n_nodes_host, float* jtj, float* jtr, float* r_depth, float* r_reg, void* stream) {
    if (!g || !g->built || n_nodes_host < 0 || n_nodes_host > g->n_max) return AFX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    const long dim = 6L * n_nodes_host;
    if (jtj && dim > 0) {
        AFX_CUDA(cudaMemsetAsync(jtj, 0, (size_t)dim * dim * 4, st));
        gn_dense_kernel<<<grid_for((long)n_nodes_host * 32, 256), 256, 0, st>>>(g->last, n_nodes_host, jtj);
        AFX_LAUNCH_CHECK();
    }
    if (jtr && dim > 0) AFX_CUDA(cudaMemcpyAsync(jtr, g->b.jtr, (size_t)dim * 4, cudaMemcpyDeviceToDevice, st));
    if (r_depth || r_reg) {
        gn_copy_residuals_kernel<<<grid_for(g->m_max + (long)g->n_max * g->kreg * 3, 256), 256, 0, st>>>(g->last, r_depth,
                                                                                                          r_reg);
        AFX_LAUNCH_CHECK();
    }
    return AFX_OK;
}

int afx_gn_solve(afx_gn* g, float* x, int iterations, double tol, void* stream) {
    if (!g || !g->built || !x || iterations < 0) return AFX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    LoopArgs L;
    std::memset(&L, 0, sizeof(L));
    L.g = g->last;
    L.pcg_iters = iterations;
    L.tol = tol;
    L.wait_polls = g->wait_polls;
    L.gave_up = g->gave_up;
    int rc = launch_cluster(gn_solve_kernel, L, st);
    if (rc) return rc;
    AFX_CUDA(cudaMemcpyAsync(x, g->b.x, (size_t)g->n_max * 6 * 4, cudaMemcpyDeviceToDevice, st));
    return AFX_OK;
}

int afx_update_transforms(float* transforms, const float* x, const int* n_nodes, int n_nodes_max, void* stream) {
    if (!transforms || !x || !n_nodes || n_nodes_max < 0) return AFX_ERR_INVALID_ARGUMENT;
    if (n_nodes_max == 0) return AFX_OK;
    update_transforms_kernel<<<grid_for((long)n_nodes_max * 16, 256), 256, 0, as_stream(stream)>>>(transforms, x, n_nodes,
                                                                                                  n_nodes_max);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

}  // extern "C"
