// afx_gn_dense.cu -- the reference's dense Gauss-Newton operators (src/MotionOptimization.cu:29-520)
// and its LU solve (src/LinearSolver.cu:179-223), for callers that keep the reference's dense
// Jacobian / (6N)^2 J^T J path.  The fused session does not use them: it assembles J^T J
// block-sparse and solves it with a preconditioned CG (afx_gn.cu).
//
// Layouts are the reference's: J is (rows x width) Vec6f, row-major (entry (row, node) at
// row * width + node); a contributing pair is a Vec2i (a <= b) with its row number; a 6x6 product
// is an Eigen Mat6f (column-major); J^T J is a dense (6 width)^2 float matrix whose rows are
// `jtj_width` floats apart; J^T r is width Vec6f.
//
// Where the reference appends pairs and J^T r elements with atomicAdd (in an order that varies from
// run to run, and which its caller then sorts), the entry points here append them in row order --
// row by row, and within a row in the reference's loop order -- so the lists are deterministic; they
// still append after the counters' current values, as the reference's do.
//
// The LU solve is partial-pivoting Gaussian elimination in binary32 on the column-major matrix the
// reference hands to cusolverDnSgetrf (pivot: the largest magnitude in the column, the first on
// ties), then the two triangular solves.  cuSOLVER's blocked factorisation rounds in a different
// order, so x agrees with the reference's to the conditioning of the system, not bit for bit.
#include <cfloat>
#include <cstring>
#include <type_traits>

#include "afx_gn.h"
#include "afx_host.h"
#include "afx_internal.h"

namespace afx {

namespace {

AFX_D void grad3x6(const float* p, float G[3][6]) {
    // gradOfTransfVertex (src/MotionOptimization.cu:22-27)
    G[0][0] = 0.f;   G[0][1] = p[2];  G[0][2] = -p[1]; G[0][3] = 1.f; G[0][4] = 0.f; G[0][5] = 0.f;
    G[1][0] = -p[2]; G[1][1] = 0.f;   G[1][2] = p[0];  G[1][3] = 0.f; G[1][4] = 1.f; G[1][5] = 0.f;
    G[2][0] = p[1];  G[2][1] = -p[0]; G[2][2] = 0.f;   G[2][3] = 0.f; G[2][4] = 0.f; G[2][5] = 1.f;
}

// fill_J_DepthKernel (src/MotionOptimization.cu:29-61): for every slot with weight >= 1e-4,
// J(row, node) = (n w)^T G(v) lambda.
__global__ void fill_j_depth_kernel(float* J, float lam, unsigned width, const int* corr, unsigned n_corr,
                                    const float* mesh, const uint32_t* knn_idx, const float* knn_w, int K,
                                    const float* normals) {
    AFX_GRID_STRIDE(c, (long)n_corr) {
        const long v = corr[2 * c], px = corr[2 * c + 1];
        const float* n = normals + 3 * px;
        float G[3][6];
        grad3x6(mesh + 3 * v, G);
        for (int i = 0; i < K; ++i) {
            const float w = knn_w[v * K + i];
            if (w < 1.e-4f) continue;
            const uint32_t node = knn_idx[v * K + i];
            if (node >= width) continue;  // not a column of J
            const float nw[3] = {n[0] * w, n[1] * w, n[2] * w};
            float* o = J + 6 * ((long)c * width + node);
#pragma unroll
            for (int q = 0; q < 6; ++q) o[q] = (nw[0] * G[0][q] + (nw[1] * G[1][q] + nw[2] * G[2][q])) * lam;
        }
    }
}

// fill_J_MRegKernel (src/MotionOptimization.cu:82-141): rows (node * Kreg + i) * 3 + axis get
// +lambda grad_axis(node) at the node and -lambda grad_axis(node) at its neighbour.
__global__ void fill_j_mreg_kernel(float* J, float lam, unsigned width, const float* nodes, unsigned n,
                                   const uint32_t* knn, int Kreg) {
    AFX_GRID_STRIDE(c, (long)n) {
        float G[3][6];
        grad3x6(nodes + 3 * c, G);
        for (int ax = 0; ax < 3; ++ax)
#pragma unroll
            for (int q = 0; q < 6; ++q) G[ax][q] = G[ax][q] * lam;
        for (int i = 0; i < Kreg; ++i) {
            const uint32_t nb = knn[c * Kreg + i];
            if (nb >= n) continue;
            const long row = (c * Kreg + i) * 3;
            for (int ax = 0; ax < 3; ++ax) {
                float* own = J + 6 * ((row + ax) * width + c);
                float* other = J + 6 * ((row + ax) * width + nb);
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    own[q] = G[ax][q];
                    other[q] = -G[ax][q];
                }
            }
        }
    }
}

// fill_r_DepthKernel (src/MotionOptimization.cu:163-181): lambda n . (warped - depth vertex)
__global__ void fill_r_depth_kernel(float* r, float lam, const int* corr, unsigned n_corr, const float* warped,
                                    const float* depth_mesh, const float* normals) {
    AFX_GRID_STRIDE(c, (long)n_corr) {
        const long v = corr[2 * c], px = corr[2 * c + 1];
        const float d[3] = {warped[3 * v] - depth_mesh[3 * px], warped[3 * v + 1] - depth_mesh[3 * px + 1],
                            warped[3 * v + 2] - depth_mesh[3 * px + 2]};
        r[c] = lam * dot3(normals + 3 * px, d);
    }
}

// fill_r_MRegKernel (src/MotionOptimization.cu:198-226): (T_node p - T_nb p) lambda; rows of a
// filtered neighbour are left as they are.
__global__ void fill_r_mreg_kernel(float* r, float lam, const float* nodes, const float* T, unsigned n,
                                   const uint32_t* knn, int Kreg) {
    AFX_GRID_STRIDE(c, (long)n) {
        float tc[3];
        mat4_point(T + 16 * c, nodes + 3 * c, tc);
        for (int i = 0; i < Kreg; ++i) {
            const uint32_t nb = knn[c * Kreg + i];
            if (nb >= n) continue;
            float tn[3];
            mat4_point(T + 16 * (long)nb, nodes + 3 * c, tn);
            const long row = (c * Kreg + i) * 3;
            for (int ax = 0; ax < 3; ++ax) r[row + ax] = (tc[ax] - tn[ax]) * lam;
        }
    }
}

// ---- contributing pairs (computeJTJAndJTrContrib*Kernel, src/MotionOptimization.cu:243-340) ----

__global__ void contrib_depth_count_kernel(unsigned* npairs, unsigned* njtr, const int* corr, unsigned n_corr,
                                           const float* knn_w, int K) {
    AFX_GRID_STRIDE(c, (long)n_corr) {
        const long v = corr[2 * c];
        unsigned nz = 0;
        for (int i = 0; i < K; ++i) nz += knn_w[v * K + i] != 0.f ? 1u : 0u;
        npairs[c] = nz * (nz + 1) / 2;
        njtr[c] = nz;
    }
}

__global__ void contrib_depth_write_kernel(int* pairs, unsigned* rows, const unsigned* n_pairs, int* jtr,
                                           const unsigned* n_jtr, const unsigned* poff, const unsigned* joff,
                                           const int* corr, unsigned n_corr, const uint32_t* knn_idx, const float* knn_w,
                                           int K) {
    const unsigned pbase = *n_pairs, jbase = *n_jtr;
    AFX_GRID_STRIDE(c, (long)n_corr) {
        const long v = corr[2 * c];
        unsigned p = pbase + poff[c], q = jbase + joff[c];
        for (int i = 0; i < K; ++i) {
            if (knn_w[v * K + i] == 0.f) continue;
            const int ni = (int)knn_idx[v * K + i];
            for (int j = i; j < K; ++j) {
                if (knn_w[v * K + j] == 0.f) continue;
                const int nj = (int)knn_idx[v * K + j];
                rows[p] = (unsigned)c;
                pairs[2 * p] = ni < nj ? ni : nj;
                pairs[2 * p + 1] = ni < nj ? nj : ni;
                ++p;
            }
            jtr[2 * q] = (int)c;
            jtr[2 * q + 1] = ni;
            ++q;
        }
    }
}

__global__ void contrib_mreg_count_kernel(unsigned* npairs, unsigned* njtr, unsigned n, const uint32_t* knn,
                                          int Kreg) {
    AFX_GRID_STRIDE(c, (long)n) {
        unsigned live = 0;
        for (int i = 0; i < Kreg; ++i) live += knn[c * Kreg + i] < n ? 1u : 0u;
        npairs[c] = 9 * live;
        njtr[c] = 6 * live;
    }
}

__global__ void contrib_mreg_write_kernel(int* pairs, unsigned* rows, unsigned row_offset, const unsigned* n_pairs,
                                          int* jtr, const unsigned* n_jtr, const unsigned* poff, const unsigned* joff,
                                          unsigned n, const uint32_t* knn, int Kreg) {
    const unsigned pbase = *n_pairs, jbase = *n_jtr;
    AFX_GRID_STRIDE(c, (long)n) {
        unsigned p = pbase + poff[c], q = jbase + joff[c];
        for (int i = 0; i < Kreg; ++i) {
            const uint32_t nb = knn[c * Kreg + i];
            if (nb >= n) continue;
            const unsigned row = (unsigned)(c * Kreg + i) * 3 + row_offset;
            const int a = (int)c, b = (int)nb;
            for (int j = 0; j < 3; ++j) {
                rows[p] = row + j;
                pairs[2 * p] = a < b ? a : b;
                pairs[2 * p + 1] = a < b ? b : a;
                rows[p + 1] = row + j;
                pairs[2 * (p + 1)] = a;
                pairs[2 * (p + 1) + 1] = a;
                rows[p + 2] = row + j;
                pairs[2 * (p + 2)] = b;
                pairs[2 * (p + 2) + 1] = b;
                p += 3;
                jtr[2 * q] = (int)(row + j);
                jtr[2 * q + 1] = a;
                jtr[2 * (q + 1)] = (int)(row + j);
                jtr[2 * (q + 1) + 1] = b;
                q += 2;
            }
        }
    }
}

__global__ void counters_add_kernel(unsigned* n_pairs, unsigned* n_jtr, const unsigned* tp, const unsigned* tj) {
    *n_pairs += *tp;
    *n_jtr += *tj;
}

// multiplyJTJContribPairsKernel (src/MotionOptimization.cu:342-356): J(row, a) J(row, b)^T, Mat6f
// column-major (entry (i, j) at j * 6 + i).
__global__ void multiply_pairs_kernel(float* out, const int* pairs, const unsigned* rows, unsigned n, const float* J,
                                      unsigned width) {
    AFX_GRID_STRIDE(t, (long)n * 36) {
        const long c = t / 36;
        const int e = (int)(t % 36), i = e % 6, j = e / 6;
        const long row = rows[c];
        const unsigned a = (unsigned)pairs[2 * c], b = (unsigned)pairs[2 * c + 1];
        if (a >= width || b >= width) continue;  // not a node of J: left unwritten
        const float* ja = J + 6 * (row * width + a);
        const float* jb = J + 6 * (row * width + b);
        out[c * 36 + e] = ja[i] * jb[j];
    }
}

// multiplyJTrContribElemsKernel (src/MotionOptimization.cu:371-383): J(row, node) r(row)
__global__ void multiply_jtr_kernel(float* out, const int* elems, unsigned n, const float* J, const float* r,
                                    unsigned width) {
    AFX_GRID_STRIDE(t, (long)n * 6) {
        const long c = t / 6;
        const int q = (int)(t % 6);
        const long row = elems[2 * c];
        const unsigned node = (unsigned)elems[2 * c + 1];
        if (node >= width) continue;  // not a node of J: left unwritten
        out[c * 6 + q] = J[6 * (row * width + node) + q] * r[row];
    }
}

// fillJTJKernel (src/MotionOptimization.cu:399-430): block (a, b) and, for a != b, its transpose at
// (b, a); rows jtj_width floats apart.
__global__ void fill_jtj_kernel(float* JTJ, const int* coords, const float* elems, unsigned n, unsigned ld) {
    AFX_GRID_STRIDE(t, (long)n * 36) {
        const long c = t / 36;
        const int e = (int)(t % 36), i = e % 6, j = e / 6;  // elems: Mat6f column-major
        const long a = coords[2 * c], b = coords[2 * c + 1];
        if (a < 0 || b < 0 || 6 * a + 5 >= (long)ld || 6 * b + 5 >= (long)ld) continue;  // outside the matrix
        const float v = elems[c * 36 + e];
        JTJ[(6 * a + i) * (long)ld + 6 * b + j] = v;
        if (a != b) JTJ[(6 * b + j) * (long)ld + 6 * a + i] = v;
    }
}

// fillJTrKernel (src/MotionOptimization.cu:447-456)
__global__ void fill_jtr_kernel(float* JTr, const int* coords, const float* elems, unsigned n) {
    AFX_GRID_STRIDE(t, (long)n * 6) {
        const long c = t / 6;
        const int q = (int)(t % 6);
        JTr[6 * (long)coords[2 * c + 1] + q] = elems[c * 6 + q];
    }
}

// ---- LU with partial pivoting (column-major, lda) ----
//
// Blocked right-looking elimination: a panel of NB columns is factorised by one CTA, then every other
// column gets the panel's row swaps and, right of the panel, the panel's updates.  An element still
// gets a[i][j] - l[i][k] u[k][j] for k = 0, 1, ... in that order, every product and difference
// rounded by itself, so the factors, pivots and solution are those of the column-by-column
// elimination bit for bit; only the passes over the matrix fall from one per column to one per NB.
// Bound: the chain of n pivots (a search over the column, one CTA barrier, a division and a rank-1
// update of registers each, about 1350 cycles).  At n = 822, ipiv and x read back: 8.9 ms with one
// search and one update launch per column, 1.37 ms now (a panel 25 us for up to 512 rows and 38 us for up
// to 1024, the update of the other columns 10 us, the triangular solves 0.27 ms).

// Best pivot of a warp: the largest key (bits of |a| + 1; 0: no candidate) and, among equal ones, the
// smallest position.
AFX_D unsigned redux_max(unsigned v) { return __reduce_max_sync(0xffffffffu, v); }
AFX_D unsigned redux_min(unsigned v) { return __reduce_min_sync(0xffffffffu, v); }

constexpr int kLuMaxPanelThreads = 512;

// Factorises columns k0 .. k0 + w - 1 (w = min(NB, n - k0)) of rows k0 .. n - 1, at most
// R * blockDim.x rows.  A thread keeps R rows of the panel in registers for the whole panel; rows
// are not moved: `pos` is the position a row has after the interchanges so far.  The register row
// moves down by one per column -- the update writes element j to j - 1, so element 0 is always the
// current column and the loop body does not depend on it -- and the multipliers go to shared memory.
// From the middle of the panel on only the lower half of the registers still holds columns.
// Every warp puts its best row in shared memory beside its key, so a column needs one CTA barrier:
// after it every thread knows the pivot and reads the pivot row.  NB x R is 64 registers at most
// (512 threads): 32 columns for up to 1024 rows, 16 up to 2048, 8 up to 4096.
// Where no pivot is left (all zero or NaN) the column is recorded in *info and, as cuSOLVER's caller
// treats the factorisation as failed, later columns are searched, swapped and divided but nothing is
// updated any more.
template <int NB, int R>
__global__ void __launch_bounds__(kLuMaxPanelThreads) lu_panel_kernel(float* A, int n, int lda, int k0, int* ipiv,
                                                                      int* info) {
    constexpr int kWarps = kLuMaxPanelThreads / 32;
    __shared__ alignas(16) float cand[2][kWarps][NB];  // each warp's best row, double-buffered over columns
    __shared__ unsigned ckey[2][kWarps], cpos[2][kWarps];
    __shared__ float prow[NB][NB + 1];                 // the chosen rows from their diagonal element on
    extern __shared__ __align__(16) float mult[];      // [NB][R * blockDim.x] multipliers of each row
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
    const int m = n - k0, w = min(NB, m);
    float a[R][NB];
    unsigned pos[R];
    bool live[R];  // a row of the matrix that is not a pivot yet
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int s = r * blockDim.x + t;
        pos[r] = (unsigned)s;
        live[r] = s < m;
        const float* col = A + (long)k0 * lda + k0 + s;
#pragma unroll
        for (int j = 0; j < NB; ++j) a[r][j] = (live[r] && j < w) ? col[(long)j * lda] : 0.f;
    }
    bool failed = *info != 0;
    const int rows = R * blockDim.x;
    auto column = [&](int c, auto width) {  // width: registers of a row that still hold columns
        constexpr int kW = decltype(width)::value;
        const int par = c & 1;
        unsigned key = 0, kp = 0xffffffffu;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float v = fabsf(a[r][0]);
            const unsigned kr = (live[r] && v == v) ? __float_as_uint(v) + 1u : 0u;
            if (kr > key || (kr == key && kr != 0u && pos[r] < kp)) {
                key = kr;
                kp = pos[r];
            }
        }
        const unsigned wk = redux_max(key);
        const unsigned wp = redux_min(key == wk ? kp : 0xffffffffu);
        if (wk != 0u && key == wk && kp == wp) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (pos[r] == wp) {
#pragma unroll
                    for (int j = 0; j < kW; j += 4)
                        *reinterpret_cast<float4*>(&cand[par][wid][j]) =
                            make_float4(a[r][j], a[r][j + 1], a[r][j + 2], a[r][j + 3]);
                }
        }
        if (lane == 0) {
            ckey[par][wid] = wk;
            cpos[par][wid] = wp;
        }
        __syncthreads();
        const unsigned bk = lane < nw ? ckey[par][lane] : 0u;
        const unsigned best = redux_max(bk);
        const unsigned bp = (lane < nw && bk == best) ? cpos[par][lane] : 0xffffffffu;
        const unsigned p = redux_min(bp);
        const int win = __ffs(__ballot_sync(0xffffffffu, lane < nw && bk == best && bp == p)) - 1;
        const float* u = cand[par][win];
        const float piv = best != 0u ? u[0] : 0.f;
        if (t == 0) ipiv[k0 + c] = best != 0u ? k0 + (int)p + 1 : n + 1;  // 1-based, as getrf
        if (piv == 0.f) {                                                 // uniform across the block
            if (t == 0 && !failed) *info = k0 + c + 1;
            failed = true;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (live[r] && pos[r] == (unsigned)c) {  // the row stays here: no candidate of a later column
                    live[r] = false;
#pragma unroll
                    for (int j = 0; j < kW; ++j) prow[c][j] = a[r][j];
                }
                mult[c * rows + r * blockDim.x + t] = a[r][0];
#pragma unroll
                for (int j = 1; j < kW; ++j) a[r][j - 1] = a[r][j];
            }
            return;
        }
        if (wid == win && lane < kW) prow[c][lane] = u[lane];
        float l[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (pos[r] == p) {
                live[r] = false;
                pos[r] = (unsigned)c;
            } else if (pos[r] == (unsigned)c) {
                pos[r] = p;
            }
            l[r] = a[r][0] / piv;  // of a row already chosen: not used
            if (live[r]) mult[c * rows + r * blockDim.x + t] = l[r];
        }
        if (failed) {
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int j = 1; j < kW; ++j) a[r][j - 1] = a[r][j];
        } else {
#pragma unroll
            for (int j0 = 0; j0 < kW; j0 += 4) {
                const float4 v = *reinterpret_cast<const float4*>(u + j0);
                const float uj[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = j0 > 0 ? j0 : 1; j < j0 + 4; ++j)
#pragma unroll
                    for (int r = 0; r < R; ++r) a[r][j - 1] = a[r][j] - l[r] * uj[j - j0];
            }
        }
    };
    const int half = min(w, NB / 2);
    for (int c = 0; c < half; ++c) column(c, std::integral_constant<int, NB>());
    for (int c = half; c < w; ++c) column(c, std::integral_constant<int, NB / 2>());
    __syncthreads();
    // the multipliers of each row at its position: all of them below the panel, those before its
    // column for a pivot row, whose other elements are prow's
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int s = r * blockDim.x + t;
        if (s >= m) continue;
        const int q = live[r] ? w : (int)pos[r];
        float* row = A + (long)k0 * lda + k0 + pos[r];
        for (int j = 0; j < q; ++j) row[(long)j * lda] = mult[j * rows + s];
        if (!live[r])
            for (int j = q; j < w; ++j) row[(long)j * lda] = prow[q][j - q];
    }
}

// The same panel (8 columns) for more rows than fit in registers: in place in global memory.
constexpr int kLuBigNB = 8;
constexpr int kLuThreads = 1024;

__global__ void __launch_bounds__(kLuThreads) lu_panel_big_kernel(float* A, int n, int lda, int k0, int* ipiv,
                                                                  int* info) {
    __shared__ unsigned ckey[32], cpos[32];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int w = min(kLuBigNB, n - k0);
    bool failed = *info != 0;
    for (int c = 0; c < w; ++c) {
        float* col = A + (long)(k0 + c) * lda;
        unsigned key = 0, kp = 0xffffffffu;
        for (int i = k0 + c + t; i < n; i += kLuThreads) {
            const float v = fabsf(col[i]);
            const unsigned kr = v == v ? __float_as_uint(v) + 1u : 0u;
            if (kr > key) {  // ascending i: the first of equal ones stays
                key = kr;
                kp = (unsigned)i;
            }
        }
        const unsigned wk = redux_max(key), wp = redux_min(key == wk ? kp : 0xffffffffu);
        if (lane == 0) {
            ckey[wid] = wk;
            cpos[wid] = wp;
        }
        __syncthreads();
        const unsigned best = redux_max(ckey[lane]);
        const unsigned p = redux_min(ckey[lane] == best ? cpos[lane] : 0xffffffffu);
        const float piv = best != 0u ? col[p] : 0.f;
        if (t == 0) ipiv[k0 + c] = best != 0u ? (int)p + 1 : n + 1;
        __syncthreads();  // every thread has read the pivot and the warps' keys
        if (piv == 0.f) {
            if (t == 0 && !failed) *info = k0 + c + 1;
            failed = true;
            continue;
        }
        if (t < w && (int)p != k0 + c) {
            float* q = A + (long)(k0 + t) * lda;
            const float x = q[k0 + c];
            q[k0 + c] = q[p];
            q[p] = x;
        }
        __syncthreads();
        for (int i = k0 + c + 1 + t; i < n; i += kLuThreads) {
            const float l = col[i] / piv;
            col[i] = l;
            if (!failed)
                for (int j = c + 1; j < w; ++j) {
                    float* q = A + (long)(k0 + j) * lda;
                    q[i] = q[i] - l * q[k0 + c];
                }
        }
        __syncthreads();
    }
}

// Where position d's row stood before the panel's swaps (k0 + i <-> p[i], i = 0 .. w - 1).
AFX_D int swap_source(int d, const int* p, int k0, int w) {
#pragma unroll 8
    for (int i = w - 1; i >= 0; --i) {
        const int a = k0 + i, b = p[i];
        d = d == a ? b : (d == b ? a : d);
    }
    return d;
}

// The columns outside a panel, kLuTC of them per CTA over all rows (so a CTA can move rows in place):
// the panel's row swaps and, for the columns right of it (the first tiles), U12 = L11^-1 A12 by one
// warp per column and A22 - L21 U12 with one row per thread and pass.  The last row below the panel is
// reached in ceil((n - k0 - w) / blockDim.x) passes.  NB: columns per panel.
constexpr int kLuTC = 8;

template <int NB>
__global__ void __launch_bounds__(kLuThreads) lu_update_kernel(float* A, int n, int lda, int k0, const int* ipiv,
                                                               const int* info, int right_tiles) {
    __shared__ int p[NB], dst[2 * NB], src[2 * NB];
    __shared__ float tmp[2 * NB][kLuTC];
    __shared__ float L11[NB][NB];               // [column][row]
    __shared__ alignas(16) float U[NB][kLuTC];
    const int t = threadIdx.x, nt = blockDim.x;
    const int w = min(NB, n - k0);
    const bool right = (int)blockIdx.x < right_tiles;
    const int c0 = right ? k0 + w + (int)blockIdx.x * kLuTC : ((int)blockIdx.x - right_tiles) * kLuTC;
    const int nc = min(kLuTC, (right ? n : k0) - c0);
    const int bad = *info;  // columns from bad - 1 on have no updates
    const int nk = bad == 0 ? w : max(0, min(w, bad - 1 - k0));
    if (t < w) {  // a column without a pivot (its diagonal element is zero or not a number) swaps nothing
        const int q = ipiv[k0 + t] - 1;
        const float d = bad != 0 ? A[k0 + t + (long)(k0 + t) * lda] : 1.f;
        p[t] = q < n && d == d && d != 0.f ? q : k0 + t;
    }
    __syncthreads();
    if (t < 2 * w) {
        const int d = t < w ? k0 + t : p[t - w];
        dst[t] = d;
        src[t] = swap_source(d, p, k0, w);
    }
    if (right)
        for (int e = t; e < w * w; e += nt) L11[e / w][e % w] = A[k0 + e % w + (long)(k0 + e / w) * lda];
    __syncthreads();
    for (int e = t; e < 2 * w * nc; e += nt) {
        const int q = e % (2 * w), j = e / (2 * w);
        tmp[q][j] = A[src[q] + (long)(c0 + j) * lda];
    }
    __syncthreads();
    for (int e = t; e < 2 * w * nc; e += nt) {
        const int q = e % (2 * w), j = e / (2 * w);
        if (dst[q] != src[q]) A[dst[q] + (long)(c0 + j) * lda] = tmp[q][j];
    }
    if (!right) return;
    for (int j = t >> 5; j < kLuTC; j += nt >> 5) {
        const int lane = t & 31;
        float u = (lane < w && j < nc) ? tmp[lane][j] : 0.f;
        for (int k = 0; k < nk; ++k) {
            const float uk = __shfl_sync(0xffffffffu, u, k);
            if (lane > k && lane < w) u = u - L11[k][lane] * uk;
        }
        if (lane < NB) U[lane][j] = u;
    }
    __syncthreads();  // U, and the moved rows of this CTA's columns
    for (int e = t; e < w * nc; e += nt) A[k0 + e % w + (long)(c0 + e / w) * lda] = U[e % w][e / w];
    for (int i = k0 + w + t; i < n; i += nt) {
        float acc[kLuTC];
#pragma unroll
        for (int j = 0; j < kLuTC; ++j) acc[j] = j < nc ? A[i + (long)(c0 + j) * lda] : 0.f;
        const float* L = A + i + (long)k0 * lda;
#pragma unroll 8
        for (int k = 0; k < nk; ++k) {
            const float l = L[(long)k * lda];
            const float4 u0 = *reinterpret_cast<const float4*>(&U[k][0]), u1 = *reinterpret_cast<const float4*>(&U[k][4]);
            acc[0] = acc[0] - l * u0.x;
            acc[1] = acc[1] - l * u0.y;
            acc[2] = acc[2] - l * u0.z;
            acc[3] = acc[3] - l * u0.w;
            acc[4] = acc[4] - l * u1.x;
            acc[5] = acc[5] - l * u1.y;
            acc[6] = acc[6] - l * u1.z;
            acc[7] = acc[7] - l * u1.w;
        }
#pragma unroll
        for (int j = 0; j < kLuTC; ++j)
            if (j < nc) A[i + (long)(c0 + j) * lda] = acc[j];
    }
}

// getrs (no transpose): row interchanges, L y = P b (unit diagonal), U x = y; one block.  Blocks of 32
// unknowns: a warp solves the diagonal block by shuffles while the other rows' coefficients, which do
// not depend on it, are already on their way to registers; then every row subtracts the block's 32
// terms in the order of the column-by-column substitution.  The unknowns stay in shared memory while
// they fit (kSolveSmem of them).
constexpr int kSolveNB = 32;
constexpr int kSolveSmem = 24576;

__global__ void __launch_bounds__(kLuThreads) lu_solve_kernel(const float* A, int n, int lda, const int* ipiv,
                                                              float* xg, const int* info, int in_smem) {
    __shared__ float D[kSolveNB][kSolveNB];  // [column][row]
    __shared__ float xb[kSolveNB];
    __shared__ int p[2][kSolveNB];
    extern __shared__ __align__(16) float xs[];
    if (*info) return;
    float* x = in_smem ? xs : xg;
    const int t = threadIdx.x, lane = t & 31, r = t & 31, c = t >> 5;  // 32 x 32 threads over a block
    if (in_smem)
        for (int i = t; i < n; i += kLuThreads) xs[i] = xg[i];
    if (t < kSolveNB) p[0][t] = t < n ? ipiv[t] - 1 : 0;
    __syncthreads();
    for (int k0 = 0, b = 0; k0 < n; k0 += kSolveNB, b ^= 1) {
        const int w = min(kSolveNB, n - k0), next = k0 + kSolveNB + t;
        int d = 0;
        float v = 0.f;
        const int pn = (t < kSolveNB && next < n) ? ipiv[next] - 1 : 0;
        if (t < 2 * w) {
            d = t < w ? k0 + t : p[b][t - w];
            v = x[swap_source(d, p[b], k0, w)];
        }
        __syncthreads();
        if (t < 2 * w) x[d] = v;
        if (t < kSolveNB) p[b ^ 1][t] = pn;
        __syncthreads();
    }
    // (the element of the next diagonal block that this thread stages is loaded a block ahead)
    float dn = r < n && c < n ? A[r + (long)c * lda] : 0.f;
    for (int k0 = 0; k0 < n; k0 += kSolveNB) {  // forward: x[i] -= l[i][k] x[k], i > k
        const int w = min(kSolveNB, n - k0), k1 = k0 + kSolveNB;
        const float* P = A + (long)k0 * lda;  // the block's columns
        D[c][r] = dn;
        const int i0 = k0 + w + t;
        float l[kSolveNB];
#pragma unroll
        for (int k = 0; k < kSolveNB; ++k) l[k] = (i0 < n && k < w) ? P[i0 + (long)k * lda] : 0.f;
        dn = (k1 + r < n && k1 + c < n) ? A[k1 + r + (long)(k1 + c) * lda] : 0.f;
        __syncthreads();
        if (t < 32) {
            float v = lane < w ? x[k0 + lane] : 0.f;
#pragma unroll 8
            for (int k = 0; k < w; ++k) {
                const float xk = __shfl_sync(0xffffffffu, v, k), d = D[k][lane];
                if (lane > k && lane < w) v = v - d * xk;
            }
            if (lane < w) x[k0 + lane] = v;
            xb[lane] = v;
        }
        __syncthreads();
        if (i0 < n) {
            float v = x[i0];
#pragma unroll
            for (int k = 0; k < kSolveNB; ++k)
                if (k < w) v = v - l[k] * xb[k];
            x[i0] = v;
        }
        for (int i = i0 + kLuThreads; i < n; i += kLuThreads) {
            float v = x[i];
#pragma unroll 8
            for (int k = 0; k < w; ++k) v = v - P[i + (long)k * lda] * xb[k];
            x[i] = v;
        }
        __syncthreads();
    }
    const int last = (n - 1) / kSolveNB * kSolveNB;
    dn = (last + r < n && last + c < n) ? A[last + r + (long)(last + c) * lda] : 0.f;
    for (int k0 = last; k0 >= 0; k0 -= kSolveNB) {  // backward
        const int w = min(kSolveNB, n - k0), k1 = k0 - kSolveNB;
        const float* P = A + (long)k0 * lda;
        D[c][r] = dn;
        float u[kSolveNB];
#pragma unroll
        for (int k = 0; k < kSolveNB; ++k) u[k] = (t < k0 && k < w) ? P[t + (long)k * lda] : 0.f;
        dn = k1 >= 0 ? A[k1 + r + (long)(k1 + c) * lda] : 0.f;
        __syncthreads();
        if (t < 32) {
            float v = lane < w ? x[k0 + lane] : 0.f;
#pragma unroll 4
            for (int k = w - 1; k >= 0; --k) {
                const float d = D[k][lane], xk = __shfl_sync(0xffffffffu, v / d, k);  // lane k: v / u[k][k]
                if (lane == k) v = xk;
                if (lane < k) v = v - d * xk;
            }
            if (lane < w) x[k0 + lane] = v;
            xb[lane] = v;
        }
        __syncthreads();
        if (t < k0) {
            float v = x[t];
#pragma unroll
            for (int k = kSolveNB - 1; k >= 0; --k)
                if (k < w) v = v - u[k] * xb[k];
            x[t] = v;
        }
        for (int i = t + kLuThreads; i < k0; i += kLuThreads) {
            float v = x[i];
#pragma unroll 8
            for (int k = w - 1; k >= 0; --k) v = v - P[i + (long)k * lda] * xb[k];
            x[i] = v;
        }
        __syncthreads();
    }
    if (in_smem)
        for (int i = t; i < n; i += kLuThreads) xg[i] = xs[i];
}

// One panel of NB columns, R rows per thread, and the update of the other columns.
template <int NB, int R>
int lu_step(float* A, int n, int lda, int k0, int* ipiv, int* info, cudaStream_t st) {
    const int m = n - k0, w = m < NB ? m : NB;
    if (m > R * kLuMaxPanelThreads) {
        lu_panel_big_kernel<<<1, kLuThreads, 0, st>>>(A, n, lda, k0, ipiv, info);
    } else {
        static ContextOnce once;  // the shared-memory opt-in: NB multipliers for every row
        const int rc = once_per_context(once, [](int) {
            return note_cuda_error(cudaFuncSetAttribute(lu_panel_kernel<NB, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        kLuMaxPanelThreads * R * NB * (int)sizeof(float)));
        });
        if (rc) return rc;
        const int threads = ((m + R - 1) / R + 31) / 32 * 32;
        lu_panel_kernel<NB, R><<<1, threads, threads * R * NB * sizeof(float), st>>>(A, n, lda, k0, ipiv, info);
    }
    AFX_LAUNCH_CHECK();
    const int right = (m - w + kLuTC - 1) / kLuTC, left = (k0 + kLuTC - 1) / kLuTC;
    if (right + left > 0) {
        int threads = (m - w + 31) / 32 * 32;
        threads = threads < 256 ? 256 : threads > kLuThreads ? kLuThreads : threads;
        lu_update_kernel<NB><<<right + left, threads, 0, st>>>(A, n, lda, k0, ipiv, info, right);
        AFX_LAUNCH_CHECK();
    }
    return AFX_OK;
}

}  // namespace

}  // namespace afx

using namespace afx;

extern "C" {

int afx_fill_j_depth(float* J, float weight, unsigned rows, unsigned width, const int* corr, unsigned n_corr,
                     const float* mesh, const uint32_t* knn_idx, const float* knn_w, int K, const float* normals,
                     void* stream) {
    if (!J || (n_corr && (!corr || !mesh || !knn_idx || !knn_w || !normals)) || K < 1 || K > 8 || n_corr > rows)
        return AFX_ERR_INVALID_ARGUMENT;
    if (!n_corr) return AFX_OK;
    fill_j_depth_kernel<<<grid_for(n_corr, 128), 128, 0, as_stream(stream)>>>(J, weight, width, corr, n_corr, mesh,
                                                                                 knn_idx, knn_w, K, normals);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_fill_j_mreg(float* J, float weight, unsigned rows, unsigned width, const float* nodes, unsigned n_nodes,
                    const uint32_t* knn_idx, int Kreg, void* stream) {
    if (!J || (n_nodes && (!nodes || !knn_idx)) || Kreg < 1 || Kreg > 8 || (unsigned long)n_nodes * Kreg * 3 > rows ||
        n_nodes > width)
        return AFX_ERR_INVALID_ARGUMENT;
    if (!n_nodes) return AFX_OK;
    fill_j_mreg_kernel<<<grid_for(n_nodes, 128), 128, 0, as_stream(stream)>>>(J, weight, width, nodes, n_nodes, knn_idx,
                                                                                Kreg);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_fill_r_depth(float* r, float weight, const int* corr, unsigned n_corr, const float* warped,
                     const float* depth_mesh, const float* normals, void* stream) {
    if (!r || (n_corr && (!corr || !warped || !depth_mesh || !normals))) return AFX_ERR_INVALID_ARGUMENT;
    if (!n_corr) return AFX_OK;
    fill_r_depth_kernel<<<grid_for(n_corr, 256), 256, 0, as_stream(stream)>>>(r, weight, corr, n_corr, warped,
                                                                                depth_mesh, normals);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_fill_r_mreg(float* r, float weight, const float* nodes, const float* transforms, unsigned n_nodes,
                    const uint32_t* knn_idx, int Kreg, void* stream) {
    if (!r || (n_nodes && (!nodes || !transforms || !knn_idx)) || Kreg < 1 || Kreg > 8) return AFX_ERR_INVALID_ARGUMENT;
    if (!n_nodes) return AFX_OK;
    fill_r_mreg_kernel<<<grid_for(n_nodes, 128), 128, 0, as_stream(stream)>>>(r, weight, nodes, transforms, n_nodes,
                                                                                knn_idx, Kreg);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

size_t afx_jtj_contrib_workspace_size(long rows) {
    if (rows < 0) return 0;
    const size_t a = (((size_t)rows * 4 + 255) / 256) * 256;
    const size_t s = ((scan_workspace_size(rows) + 255) / 256) * 256;
    return 4 * a + 2 * s + 512;
}

static int contrib_common(long rows, void* ws, size_t ws_bytes, unsigned** cp, unsigned** cj, unsigned** op,
                          unsigned** oj, unsigned** tp, unsigned** tj, void** sp, void** sj) {
    if (ws_bytes < afx_jtj_contrib_workspace_size(rows) || !ws) return AFX_ERR_WORKSPACE;
    const size_t a = (((size_t)rows * 4 + 255) / 256) * 256;
    const size_t s = ((scan_workspace_size(rows) + 255) / 256) * 256;
    char* q = static_cast<char*>(ws);
    *cp = (unsigned*)q;
    *cj = (unsigned*)(q + a);
    *op = (unsigned*)(q + 2 * a);
    *oj = (unsigned*)(q + 3 * a);
    *sp = q + 4 * a;
    *sj = q + 4 * a + s;
    *tp = (unsigned*)(q + 4 * a + 2 * s);
    *tj = (unsigned*)(q + 4 * a + 2 * s + 256);
    return AFX_OK;
}

int afx_jtj_contrib_depth(int* pairs, unsigned* rows, unsigned* n_pairs, int* jtr_elems, unsigned* n_jtr,
                          const int* corr, unsigned n_corr, const uint32_t* knn_idx, const float* knn_w, int K,
                          void* workspace, size_t workspace_bytes, void* stream) {
    if (!pairs || !rows || !n_pairs || !jtr_elems || !n_jtr || K < 1 || K > 8 ||
        (n_corr && (!corr || !knn_idx || !knn_w)))
        return AFX_ERR_INVALID_ARGUMENT;
    if (!n_corr) return AFX_OK;
    unsigned *cp, *cj, *op, *oj, *tp, *tj;
    void *sp, *sj;
    int rc = contrib_common(n_corr, workspace, workspace_bytes, &cp, &cj, &op, &oj, &tp, &tj, &sp, &sj);
    if (rc) return rc;
    cudaStream_t st = as_stream(stream);
    contrib_depth_count_kernel<<<grid_for(n_corr, 256), 256, 0, st>>>(cp, cj, corr, n_corr, knn_w, K);
    AFX_LAUNCH_CHECK();
    rc = scan_exclusive(cp, op, n_corr, tp, sp, st);
    if (!rc) rc = scan_exclusive(cj, oj, n_corr, tj, sj, st);
    if (rc) return rc;
    contrib_depth_write_kernel<<<grid_for(n_corr, 128), 128, 0, st>>>(pairs, rows, n_pairs, jtr_elems, n_jtr, op, oj,
                                                                         corr, n_corr, knn_idx, knn_w, K);
    AFX_LAUNCH_CHECK();
    counters_add_kernel<<<1, 1, 0, st>>>(n_pairs, n_jtr, tp, tj);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_jtj_contrib_mreg(int* pairs, unsigned* rows, unsigned row_offset, unsigned* n_pairs, int* jtr_elems,
                         unsigned* n_jtr, unsigned n_nodes, const uint32_t* knn_idx, int Kreg, void* workspace,
                         size_t workspace_bytes, void* stream) {
    if (!pairs || !rows || !n_pairs || !jtr_elems || !n_jtr || Kreg < 1 || Kreg > 8 || (n_nodes && !knn_idx))
        return AFX_ERR_INVALID_ARGUMENT;
    if (!n_nodes) return AFX_OK;
    unsigned *cp, *cj, *op, *oj, *tp, *tj;
    void *sp, *sj;
    int rc = contrib_common(n_nodes, workspace, workspace_bytes, &cp, &cj, &op, &oj, &tp, &tj, &sp, &sj);
    if (rc) return rc;
    cudaStream_t st = as_stream(stream);
    contrib_mreg_count_kernel<<<grid_for(n_nodes, 256), 256, 0, st>>>(cp, cj, n_nodes, knn_idx, Kreg);
    AFX_LAUNCH_CHECK();
    rc = scan_exclusive(cp, op, n_nodes, tp, sp, st);
    if (!rc) rc = scan_exclusive(cj, oj, n_nodes, tj, sj, st);
    if (rc) return rc;
    contrib_mreg_write_kernel<<<grid_for(n_nodes, 128), 128, 0, st>>>(pairs, rows, row_offset, n_pairs, jtr_elems,
                                                                        n_jtr, op, oj, n_nodes, knn_idx, Kreg);
    AFX_LAUNCH_CHECK();
    counters_add_kernel<<<1, 1, 0, st>>>(n_pairs, n_jtr, tp, tj);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_multiply_jtj_pairs(float* out, const int* pairs, const unsigned* rows, unsigned n_pairs, const float* J,
                           unsigned width, void* stream) {
    if (!out || (n_pairs && (!pairs || !rows || !J))) return AFX_ERR_INVALID_ARGUMENT;
    if (!n_pairs) return AFX_OK;
    multiply_pairs_kernel<<<grid_for((long)n_pairs * 36, 256), 256, 0, as_stream(stream)>>>(out, pairs, rows, n_pairs,
                                                                                               J, width);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_multiply_jtr_elems(float* out, const int* elems, unsigned n_elems, const float* J, const float* r,
                           unsigned width, void* stream) {
    if (!out || (n_elems && (!elems || !J || !r))) return AFX_ERR_INVALID_ARGUMENT;
    if (!n_elems) return AFX_OK;
    multiply_jtr_kernel<<<grid_for((long)n_elems * 6, 256), 256, 0, as_stream(stream)>>>(out, elems, n_elems, J, r,
                                                                                            width);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_fill_jtj(float* JTJ, const int* coords, const float* elems, unsigned n_elems, unsigned jtj_width,
                 void* stream) {
    if (!JTJ || (n_elems && (!coords || !elems))) return AFX_ERR_INVALID_ARGUMENT;
    if (!n_elems) return AFX_OK;
    fill_jtj_kernel<<<grid_for((long)n_elems * 36, 256), 256, 0, as_stream(stream)>>>(JTJ, coords, elems, n_elems,
                                                                                         jtj_width);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

int afx_fill_jtr(float* JTr, const int* coords, const float* elems, unsigned n_elems, void* stream) {
    if (!JTr || (n_elems && (!coords || !elems))) return AFX_ERR_INVALID_ARGUMENT;
    if (!n_elems) return AFX_OK;
    fill_jtr_kernel<<<grid_for((long)n_elems * 6, 256), 256, 0, as_stream(stream)>>>(JTr, coords, elems, n_elems);
    AFX_LAUNCH_CHECK();
    return AFX_OK;
}

size_t afx_lu_solve_workspace_size(int n, int lda) {
    if (n < 0 || lda < n) return 0;
    return (((size_t)lda * n * 4 + 255) / 256) * 256 + 256;
}

int afx_lu_solve(float* x, const float* A, int n, int lda, const float* b, int* ipiv, void* workspace,
                 size_t workspace_bytes, void* stream) {
    if (!x || !A || !b || !ipiv || n < 1 || lda < n) return AFX_ERR_INVALID_ARGUMENT;
    if (!workspace || workspace_bytes < afx_lu_solve_workspace_size(n, lda)) return AFX_ERR_WORKSPACE;
    cudaStream_t st = as_stream(stream);
    float* LU = static_cast<float*>(workspace);
    int* info = reinterpret_cast<int*>(static_cast<char*>(workspace) + (((size_t)lda * n * 4 + 255) / 256) * 256);
    AFX_CUDA(cudaMemcpyAsync(LU, A, (size_t)lda * n * 4, cudaMemcpyDeviceToDevice, st));
    AFX_CUDA(cudaMemsetAsync(info, 0, 4, st));
    for (int k0 = 0; k0 < n;) {
        // as many columns per panel as the registers of one CTA hold for the rows that are left
        const int m = n - k0, T = kLuMaxPanelThreads, nb = m <= 2 * T ? 32 : m <= 4 * T ? 16 : kLuBigNB;
        const int rc = m <= T       ? lu_step<32, 1>(LU, n, lda, k0, ipiv, info, st)
                       : m <= 2 * T ? lu_step<32, 2>(LU, n, lda, k0, ipiv, info, st)
                       : m <= 4 * T ? lu_step<16, 4>(LU, n, lda, k0, ipiv, info, st)
                                    : lu_step<kLuBigNB, 8>(LU, n, lda, k0, ipiv, info, st);
        if (rc) return rc;
        k0 += nb;
    }
    AFX_CUDA(cudaMemcpyAsync(x, b, (size_t)n * 4, cudaMemcpyDeviceToDevice, st));
    static ContextOnce once;
    const int rc = once_per_context(once, [](int) {
        return note_cuda_error(cudaFuncSetAttribute(lu_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    kSolveSmem * (int)sizeof(float)));
    });
    if (rc) return rc;
    const bool in_smem = n <= kSolveSmem;
    lu_solve_kernel<<<1, kLuThreads, in_smem ? n * sizeof(float) : 0, st>>>(LU, n, lda, ipiv, x, info, in_smem);
    AFX_LAUNCH_CHECK();
    int h_info = 0;
    AFX_CUDA(cudaMemcpyAsync(&h_info, info, 4, cudaMemcpyDeviceToHost, st));
    AFX_CUDA(cudaStreamSynchronize(st));
    return h_info ? AFX_ERR_SINGULAR : AFX_OK;
}

}  // extern "C"
