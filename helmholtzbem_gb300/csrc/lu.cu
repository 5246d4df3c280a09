// Batched LU with partial pivoting of complex128 matrices in global memory, and
// the two triangular-solve forms randomized_svd needs (T x = b and T^H x = b).
// It replaces Eigen::PartialPivLU at source/utilities/randsvd.cpp:104 (the LU of
// T(k)) and :205 (the bordered Wielandt system of sv_der2).
//
// Right-looking blocked factorisation, panel width 32, three launches per panel:
//   k_lu_panel      unblocked LU of the n-k0 x 32 panel, one CTA per matrix, or
//                   k_lu_panel_cluster, a cluster of up to 16
//   k_lu_swap_trsm  row exchanges on every column outside the panel and
//                   U12 = L11^-1 A12 on the columns right of it
//   k_lu_gemm       A22 -= L21 U12, 64 x 64 tiles, all matrices in one grid; large ones
//                   on the tensor cores (zgemm_tc.cu, tc_gemm.cu)
// Four complex128 matrices of order 1500: 43 panels on clusters 5.4 ms, exchanges and
// triangular solves 1.5 (71 us a launch with serial exchanges, 31 now: its FP64 steps), updates
// 3.6 (6.0 before the second tile buffer of zgemm_tc.cu).
// Matrices are column-major with leading dimension n (Eigen's layout); matrix m
// starts at A + m * stride.  piv[m*n + k] = row exchanged with row k at step k
// (LAPACK's ipiv, 0-based); perm[m*n + i] = source row of row i of P A; info[m]: 0, 1 + the first step
// with a zero pivot, or -1 where a wait of the complex128 tensor-core update ran out.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "hbem_device.cuh"

namespace cg = cooperative_groups;

namespace hbem {

constexpr int kLuNB = 32;
constexpr int kLuPanelThreads = 512;
constexpr int kLuClusterThreads = 512;   // a multiple of 128
constexpr int kLuTile = 64;
constexpr int kLuTcMin = 128;            // smallest trailing order the complex128 tensor-core update takes
constexpr int kLuSolveThreads = 512;
constexpr int kLuSolveChunk = 16;      // right-hand sides held in registers at a time

// Pivot candidates as integers: |x|^2 >= 0, so its bits order like its value, and an integer
// comparison costs 2 cycles a warp where an FP64 one costs 76 (the comparisons of the search
// were a third of a panel's time).  NaN counts as smaller than everything, as in a > best.
struct PivotKey {
    unsigned long long v;   // 0: no candidate; else 1 + the bits of |x|^2
    int i;
};
__device__ __forceinline__ unsigned long long pivot_key(cplx z) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(norm2(z));
    return b > 0x7ff0000000000000ull ? 0ull : b + 1;
}
__device__ __forceinline__ unsigned long long pivot_key(cplxf z) {
    const unsigned b = __float_as_uint(norm2(z));
    return b > 0x7f800000u ? 0ull : (unsigned long long)b + 1;
}
// the largest of a warp's candidates; ties: the smaller index
__device__ __forceinline__ PivotKey pivot_warp_max(PivotKey a) {
    const unsigned hi = (unsigned)(a.v >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)a.v : 0u);
    const unsigned long long v = ((unsigned long long)mh << 32) | ml;
    return PivotKey{v, (int)__reduce_min_sync(0xffffffffu, a.v == v ? (unsigned)a.i : 0xffffffffu)};
}

// Row i of the rank-1 update of a panel step, shared over the CTA: threads take (row, every
// fourth column).  lcol: the scaled column.  rows [i0, i1) of the panel storage P (leading
// dimension ld), columns j + 1 .. nb - 1.
template <class E>
__device__ __forceinline__ void panel_rank1(E* P, int ld, int i0, int i1, int j, int nb, const E* lcol, const E* prow) {
    const int tr = threadIdx.x & 127, cg = threadIdx.x >> 7;
    for (int i = i0 + tr; i < i1; i += 128) {
        const E l = lcol[i];
        for (int cc = j + 1 + cg; cc < nb; cc += kLuPanelThreads / 128) cfms(P[i + (long long)cc * ld], l, prow[cc]);
    }
}

// Unblocked LU of the panel rows [k0, n) x columns [k0, k0 + nb), one CTA per matrix.
// STAGED: the panel is copied to shared memory (column-major, leading dimension n - k0, the
// scaled column behind it), factored there and written back; otherwise it is factored in
// place in global memory (L2).
template <class E, bool STAGED>
__global__ void __launch_bounds__(kLuPanelThreads) k_lu_panel(int n, int k0, int nb, E* A, long long stride,
                                                              int* piv, int* info) {
    extern __shared__ double panel_sm[];
    E* M = A + (long long)blockIdx.x * stride;
    int* pv = piv + (long long)blockIdx.x * n;
    const int m = n - k0;
    E* P = STAGED ? reinterpret_cast<E*>(panel_sm) : M + k0 + (long long)k0 * n;
    const int ld = STAGED ? m : n;
    E* lcol = STAGED ? P + (long long)m * nb : nullptr;
    __shared__ PivotKey cand[kLuPanelThreads / 32];
    __shared__ E prow[kLuNB], s_id;
    __shared__ int s_p;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (STAGED) {
        for (int e = threadIdx.x; e < m * nb; e += blockDim.x) P[e] = M[(k0 + e % m) + (long long)(k0 + e / m) * n];
        __syncthreads();
    }
    for (int j = 0; j < nb; ++j) {
        PivotKey best{0ull, j};
        for (int i = j + threadIdx.x; i < m; i += blockDim.x) {
            const unsigned long long a = pivot_key(P[i + (long long)j * ld]);
            if (a > best.v) { best.v = a; best.i = i; }
        }
        best = pivot_warp_max(best);
        if (lane == 0) cand[warp] = best;
        __syncthreads();
        if (warp == 0) {
            best = lane < nw ? cand[lane] : PivotKey{0ull, m};
            best = pivot_warp_max(best);
            if (lane == 0) {
                if (best.v == 0ull) best.i = j;
                s_p = best.i;
                pv[k0 + j] = k0 + best.i;
                if (best.v == 1ull && info[blockIdx.x] == 0) info[blockIdx.x] = k0 + j + 1;
            }
            __syncwarp();
            const int p = s_p;
            E y = Elem<E>::zero();
            if (lane < nb) {
                E& xa = P[j + (long long)lane * ld];
                E& ya = P[p + (long long)lane * ld];
                const E x = xa;
                y = ya;
                if (p != j) { xa = y; ya = x; }
                prow[lane] = y;
            }
            if (lane == j) s_id = norm2(y) > 0 ? cdiv(Elem<E>::one(), y) : Elem<E>::one();   // zero pivot: unscaled
        }
        __syncthreads();
        const E id = s_id;
        if (STAGED) {
            for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) {
                const E l = P[i + j * m] * id;
                P[i + j * m] = l;
                lcol[i] = l;
            }
            __syncthreads();
            panel_rank1(P, m, j + 1, m, j, nb, lcol, prow);
        } else {
            for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) {
                const E l = P[i + (long long)j * ld] * id;
                P[i + (long long)j * ld] = l;
                for (int cc = j + 1; cc < nb; ++cc) cfms(P[i + (long long)cc * ld], l, prow[cc]);
            }
        }
        __syncthreads();
    }
    if (STAGED)
        for (int e = threadIdx.x; e < m * nb; e += blockDim.x) M[(k0 + e % m) + (long long)(k0 + e / m) * n] = P[e];
}

// The same on a cluster of CS CTAs per matrix (grid nmat * CS), CTA r holding panel rows
// [k0 + r R, k0 + (r + 1) R) in its shared memory (column-major, leading dimension R): for
// panels too tall for one CTA, and for few matrices because the FP64 rate of one SM bounds
// the rank-1 updates.  What is left is a chain of dependent steps per column, kept to one
// cluster barrier: before it every CTA writes its candidate into all the others' shared memory
// and posts that whole row in its own, and row c's owner posts row c; after it all read the
// winner's posted row through distributed shared memory, and the two owners write the exchanged
// rows.  The posts alternate between two buffers: a buffer is written again two columns on, past
// a barrier that every reader reached after its reads.  The next column's candidates come out of
// the rank-1 update, and the pivots go to global memory at the end (the barrier would wait for
// the write).
template <class E>
__global__ void __launch_bounds__(kLuClusterThreads) k_lu_panel_cluster(int n, int k0, int nb, int R, E* A,
                                                                      long long stride, int* piv, int* info) {
    cg::cluster_group cl = cg::this_cluster();
    const int ncta = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int mat = blockIdx.x / ncta;
    extern __shared__ double panel_sm[];
    E* P = reinterpret_cast<E*>(panel_sm);
    E* lcol = P + (long long)R * nb;
    __shared__ PivotKey post[2][16], cand[kLuClusterThreads / 32];
    __shared__ int s_piv[kLuNB], s_info;
    __shared__ E post_row[2][kLuNB], post_c[2][kLuNB], prow[kLuNB], s_id;
    E* M = A + (long long)mat * stride;
    int* pv = piv + (long long)mat * n;
    const int r0 = k0 + rank * R, r1 = min(n, r0 + R), rows = max(0, r1 - r0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int tr = threadIdx.x & 127, part = threadIdx.x >> 7;   // a row and every so many columns
    for (int e = threadIdx.x; e < rows * nb; e += blockDim.x)
        P[(e % rows) + (e / rows) * R] = M[(r0 + e % rows) + (long long)(k0 + e / rows) * n];
    if (threadIdx.x == 0) s_info = 0;
    cl.sync();   // every CTA runs before another writes into it
    {
        PivotKey best{0ull, n};
        for (int i = threadIdx.x; i < rows; i += blockDim.x) {
            const unsigned long long a = pivot_key(P[i]);
            if (a > best.v) { best.v = a; best.i = r0 + i; }
        }
        best = pivot_warp_max(best);
        if (lane == 0) cand[warp] = best;
    }
    __syncthreads();
    for (int j = 0; j < nb; ++j) {
        const int c = k0 + j, rc = j / R, b = j & 1;
        if (warp == 0) {
            const PivotKey mine = pivot_warp_max(lane < nw ? cand[lane] : PivotKey{0ull, n});
            if (lane < ncta) *cl.map_shared_rank(&post[b][rank], lane) = mine;
            if (lane < nb) {
                if (mine.v) post_row[b][lane] = P[(mine.i - r0) + lane * R];
                if (rank == rc) post_c[b][lane] = P[(c - r0) + lane * R];
            }
        }
        cl.sync();
        if (warp == 0) {
            PivotKey best = pivot_warp_max(lane < ncta ? post[b][lane] : PivotKey{0ull, n});
            if (best.v == 0ull) best.i = c;
            const int p = best.i, rp = (p - k0) / R;
            if (lane == 0) {
                s_piv[j] = p;
                if (best.v == 1ull && s_info == 0) s_info = c + 1;
            }
            E y = Elem<E>::zero();
            if (lane < nb) {
                y = p == c ? cl.map_shared_rank(&post_c[b][0], rc)[lane] : cl.map_shared_rank(&post_row[b][0], rp)[lane];
                prow[lane] = y;
                if (p != c) {
                    if (rank == rc) P[(c - r0) + lane * R] = y;
                    if (rank == rp) P[(p - r0) + lane * R] = cl.map_shared_rank(&post_c[b][0], rc)[lane];
                }
            }
            if (lane == j) s_id = norm2(y) > 0 ? cdiv(Elem<E>::one(), y) : Elem<E>::one();   // zero pivot: unscaled
        }
        __syncthreads();
        const E id = s_id;
        const int i0 = max(c + 1, r0) - r0;
        for (int i = i0 + threadIdx.x; i < rows; i += blockDim.x) {
            const E l = P[i + j * R] * id;
            P[i + j * R] = l;
            lcol[i] = l;
        }
        __syncthreads();
        PivotKey best{0ull, n};
        for (int i = i0 + tr; i < rows; i += 128) {
            const E l = lcol[i];
            // complex64: four loads, then four updates (latency; 129 -> 89 us a panel of order 3000
            // with the finer split).  complex128: the FP64 pipe is what waits, and alternates better
            // one by one (126 us; 150 in fours, order 1500)
            constexpr int kStep = kLuClusterThreads / 128, kBatch = std::is_same<E, cplxf>::value ? 4 : 1;
            for (int cc = j + 1 + part; cc < nb; cc += kBatch * kStep) {
                E z[kBatch];
#pragma unroll
                for (int q = 0; q < kBatch; ++q)
                    if (cc + q * kStep < nb) z[q] = P[i + (cc + q * kStep) * R];
#pragma unroll
                for (int q = 0; q < kBatch; ++q)
                    if (cc + q * kStep < nb) {
                        cfms(z[q], l, prow[cc + q * kStep]);
                        P[i + (cc + q * kStep) * R] = z[q];
                    }
                if (cc == j + 1) {
                    const unsigned long long a = pivot_key(z[0]);
                    if (a > best.v) { best.v = a; best.i = r0 + i; }
                }
            }
        }
        best = pivot_warp_max(best);
        if (lane == 0) cand[warp] = best;
        __syncthreads();
    }
    for (int e = threadIdx.x; e < rows * nb; e += blockDim.x)
        M[(r0 + e % rows) + (long long)(k0 + e / rows) * n] = P[(e % rows) + (e / rows) * R];
    if (rank == 0) {
        if (threadIdx.x < nb) pv[k0 + threadIdx.x] = s_piv[threadIdx.x];
        if (threadIdx.x == 0 && s_info && info[mat] == 0) info[mat] = s_info;
    }
    cl.sync();   // no CTA leaves while another may still read its shared memory
}

// Row exchanges of a panel's nb <= 32 columns on every column outside the panel, and
// U12 = L11^-1 A12 on the columns right of it.  grid (ceil(n / 16), nmat), 16 columns a CTA;
// columns from cmax on are left alone (the two-level factorisation exchanges and solves them
// once per 128-column block, k_lu_swap_trsm_block).
// The exchanges are composed into one gather over the at most 64 rows they touch (slot x < 32:
// row k0 + x; slot 32 + j: the pivot of step j where it lies below the panel), so that a column
// waits for memory once and not 32 times.  Eight lanes to a column, lane r holding rows r, r + 8,
// r + 16, r + 24: the substitution takes 80 FP64 steps for four columns where a warp per column,
// half idle, takes 128 for one.
// ek (complex128, or null): per matrix n integers, zero before, that take the biased exponents of
// the largest entries of U's rows right of their panel (the digit products' scales, zgemm_tc.cu).
constexpr int kLuSwapCols = 16;
__device__ __forceinline__ int abs_high(cplx z) {   // high words order like the sizes
    return max(__double2hiint(z.re) & 0x7fffffff, __double2hiint(z.im) & 0x7fffffff);
}
template <class E>
__global__ void __launch_bounds__(kLuSwapCols * 8) k_lu_swap_trsm(int n, int k0, int nb, E* A, long long stride,
                                                                  const int* piv, int cmax, int* ek) {
    const int col0 = blockIdx.x * kLuSwapCols;
    if ((col0 >= k0 && col0 < k0 + nb) || col0 >= cmax) return;   // the panel itself, or deferred
    E* M = A + (long long)blockIdx.y * stride;
    const int* pv = piv + (long long)blockIdx.y * n;
    __shared__ int pos[64], from[64];       // the slot's row (-1: none), the row its entry comes from
    __shared__ E L11[kLuNB][kLuNB + 1];     // [k][r]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {
        const int p = lane < nb ? pv[k0 + lane] : -1 - lane;
        const int first = __ffs(__match_any_sync(0xffffffffu, p)) - 1;
        const bool below = lane < nb && p >= k0 + nb;
        const int slot = lane >= nb ? lane : below ? 32 + first : p - k0;
        pos[lane] = lane < nb ? k0 + lane : -1;
        pos[32 + lane] = below && first == lane ? p : -1;
        int x = lane, y = 32 + lane;        // where the final entries of slots lane, 32 + lane were
        for (int j = nb - 1; j >= 0; --j) {
            const int s = __shfl_sync(0xffffffffu, slot, j);
            x = x == j ? s : x == s ? j : x;
            y = y == j ? s : y == s ? j : y;
        }
        __syncwarp();
        from[lane] = pos[x];
        from[32 + lane] = pos[y];
    }
    if (col0 > k0)
        for (int e = threadIdx.x; e < kLuNB * kLuNB; e += blockDim.x) {
            const int r = e % kLuNB, k = e / kLuNB;
            L11[k][r] = r < nb && k < nb ? M[(k0 + r) + (long long)(k0 + k) * n] : Elem<E>::zero();
        }
    __syncthreads();
    const int col = col0 + (threadIdx.x >> 3), r = lane & 7;
    const bool in = col < min(n, cmax);
    E* a = M + (long long)(in ? col : col0) * n;
    E v[4], w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int s = r + 8 * q;
        v[q] = in && pos[s] >= 0 ? a[from[s]] : Elem<E>::zero();
        w[q] = in && pos[32 + s] >= 0 ? a[from[32 + s]] : Elem<E>::zero();
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (in && pos[32 + r + 8 * q] >= 0) a[pos[32 + r + 8 * q]] = w[q];
    if (col0 > k0) {
#pragma unroll
        for (int k = 0; k < kLuNB; ++k) {
            if (k >= nb) break;
            E xk;
            xk.re = __shfl_sync(0xffffffffu, v[k >> 3].re, (lane & 24) + (k & 7));
            xk.im = __shfl_sync(0xffffffffu, v[k >> 3].im, (lane & 24) + (k & 7));
#pragma unroll
            for (int q = k >> 3; q < 4; ++q)
                if (q > (k >> 3) || r > (k & 7)) cfms(v[q], L11[k][r + 8 * q], xk);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (in && pos[r + 8 * q] >= 0) a[pos[r + 8 * q]] = v[q];
    if constexpr (std::is_same<E, cplx>::value) {
        if (!ek || col0 < k0) return;   // whole CTA
        __shared__ int high[kLuNB];
        if (threadIdx.x < kLuNB) high[threadIdx.x] = 0;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int h = in ? abs_high(v[q]) : 0;
            h = max(h, __shfl_xor_sync(0xffffffffu, h, 8));
            h = max(h, __shfl_xor_sync(0xffffffffu, h, 16));
            if (lane < 8) atomicMax(&high[r + 8 * q], h);
        }
        __syncthreads();
        if (threadIdx.x < nb) atomicMax(ek + (long long)blockIdx.y * n + k0 + threadIdx.x, high[threadIdx.x] >> 20);
    }
}

// Two-level factorisation, after the kb (<= 128) columns from K0 are factored: the
// row exchanges of those columns applied, in order, to the columns right of them
// (cbase on), and the block row solved with the kb x kb unit lower triangle,
// U12 = L11^-1 A12.  grid (ceil((n - cbase) / 32), nmat); L11 in shared memory
// (kb x (kb + 1)); a warp per column, lane l holding rows l, l + 32, l + 64, l + 96.
constexpr int kLuBlock = 128;
template <class E>
__global__ void __launch_bounds__(256) k_lu_swap_trsm_block(int n, int K0, int kb, E* A, long long stride,
                                                            const int* piv) {
    extern __shared__ double blk_sm[];
    E* L = reinterpret_cast<E*>(blk_sm);                  // [r][k], leading dimension kb + 1
    __shared__ int sp[kLuBlock];
    const int cbase = K0 + kb;
    const int col0 = cbase + blockIdx.x * kLuNB;
    E* M = A + (long long)blockIdx.y * stride;
    const int* pv = piv + (long long)blockIdx.y * n;
    const int ncols = min(kLuNB, n - col0);
    for (int j = threadIdx.x; j < kb; j += blockDim.x) sp[j] = pv[K0 + j];
    for (int e = threadIdx.x; e < kb * kb; e += blockDim.x) {
        const int r = e % kb, k = e / kb;
        L[r * (kb + 1) + k] = M[(K0 + r) + (long long)(K0 + k) * n];
    }
    __syncthreads();
    if (threadIdx.x < ncols) {
        E* a = M + (long long)(col0 + threadIdx.x) * n;
        for (int j = 0; j < kb; ++j) {
            const int p = sp[j];
            if (p != K0 + j) {
                const E t = a[K0 + j];
                a[K0 + j] = a[p];
                a[p] = t;
            }
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int cc = warp; cc < ncols; cc += (blockDim.x >> 5)) {
        E* a = M + (long long)(col0 + cc) * n + K0;
        E x[kLuBlock / 32];
#pragma unroll
        for (int s = 0; s < kLuBlock / 32; ++s) {
            const int r = lane + 32 * s;
            x[s] = r < kb ? a[r] : Elem<E>::zero();
        }
#pragma unroll
        for (int s0 = 0; s0 < kLuBlock / 32; ++s0) {
            for (int kk = 0; kk < 32; ++kk) {
                const int k = 32 * s0 + kk;
                if (k >= kb) break;
                E xk;
                xk.re = __shfl_sync(0xffffffffu, x[s0].re, kk);
                xk.im = __shfl_sync(0xffffffffu, x[s0].im, kk);
#pragma unroll
                for (int s = 0; s < kLuBlock / 32; ++s) {
                    const int r = lane + 32 * s;
                    if (s >= s0 && r > k && r < kb) cfms(x[s], L[r * (kb + 1) + k], xk);
                }
            }
        }
#pragma unroll
        for (int s = 0; s < kLuBlock / 32; ++s) {
            const int r = lane + 32 * s;
            if (r < kb) a[r] = x[s];
        }
    }
}

// grid (tiles over trailing rows, tiles over trailing columns below cend, nmat)
template <class E>
__global__ void __launch_bounds__(256) k_lu_gemm(int n, int k0, int nb, E* A, long long stride, int cend) {
    extern __shared__ double lu_smem[];
    E* La = reinterpret_cast<E*>(lu_smem);                // [k][i], 32 x 64
    E* Ub = La + kLuNB * kLuTile;                         // [k][j], 32 x 64
    const int t0 = k0 + nb;
    const int r0 = t0 + blockIdx.x * kLuTile, c0 = t0 + blockIdx.y * kLuTile;
    E* M = A + (long long)blockIdx.z * stride;
    for (int e = threadIdx.x; e < kLuNB * kLuTile; e += blockDim.x) {
        const int i = e % kLuTile, k = e / kLuTile;
        La[k * kLuTile + i] = (k < nb && r0 + i < n) ? M[(r0 + i) + (long long)(k0 + k) * n] : Elem<E>::zero();
        const int kk = e % kLuNB, j = e / kLuNB;
        Ub[kk * kLuTile + j] = (kk < nb && c0 + j < cend) ? M[(k0 + kk) + (long long)(c0 + j) * n] : Elem<E>::zero();
    }
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    E acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = Elem<E>::zero();
    for (int k = 0; k < nb; ++k) {
        E av[4], bv[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) av[a] = La[k * kLuTile + tx + 16 * a];
#pragma unroll
        for (int b = 0; b < 4; ++b) bv[b] = Ub[k * kLuTile + ty + 16 * b];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                acc[a][b].re = fma(av[a].re, bv[b].re, fma(-av[a].im, bv[b].im, acc[a][b].re));
                acc[a][b].im = fma(av[a].re, bv[b].im, fma(av[a].im, bv[b].re, acc[a][b].im));
            }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int j = c0 + ty + 16 * b;
        if (j >= cend) continue;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int i = r0 + tx + 16 * a;
            if (i < n) M[i + (long long)j * n] -= acc[a][b];
        }
    }
}

// perm from the exchange sequence: one CTA per matrix, the exchanges applied in
// shared memory by one thread.
__global__ void k_lu_perm(int n, const int* piv, int* perm) {
    extern __shared__ int pm[];
    const int* pv = piv + (long long)blockIdx.x * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) pm[i] = i;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < n; ++k) {
            const int p = pv[k];
            if (p != k) { const int t = pm[k]; pm[k] = pm[p]; pm[p] = t; }
        }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) perm[(long long)blockIdx.x * n + i] = pm[i];
}

size_t lu_solve_smem_bytes(int n, size_t esz) {
    return ((size_t)n + (size_t)kLuNB * (kLuNB + 1) + (size_t)kLuNB * kLuSolveChunk) * esz;
}

// Row permutation of the s columns of X in place through a shared-memory column
// buffer: forward (X <- P X) or inverse (X <- P^T X).
template <class E>
__device__ void permute_rows(E* X, int n, int s, const int* perm, E* buf, bool inverse) {
    for (int c = 0; c < s; ++c) {
        E* x = X + (long long)c * n;
        for (int i = threadIdx.x; i < n; i += blockDim.x) buf[i] = x[i];
        __syncthreads();
        if (!inverse)
            for (int i = threadIdx.x; i < n; i += blockDim.x) x[i] = buf[perm[i]];
        else
            for (int i = threadIdx.x; i < n; i += blockDim.x) x[perm[i]] = buf[i];
        __syncthreads();
    }
}

// X <- T^-1 X (s columns), P T = L U stored in M.  Right-looking by 32-row blocks.
template <class E, int CH>
__device__ void lu_solve_n(const E* M, const int* perm, int n, E* X, int s, E* sm) {
    E* buf = sm;
    E (*D)[kLuNB + 1] = reinterpret_cast<E (*)[kLuNB + 1]>(sm + n);
    E* xb = sm + n + kLuNB * (kLuNB + 1);            // [c][k], CH x 32
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    permute_rows(X, n, s, perm, buf, false);
    for (int b0 = 0; b0 < n; b0 += kLuNB) {
        const int bs = min(kLuNB, n - b0);
        for (int e = threadIdx.x; e < bs * bs; e += blockDim.x) {
            const int r = e % bs, k = e / bs;
            D[r][k] = M[(b0 + r) + (long long)(b0 + k) * n];
        }
        __syncthreads();
        for (int cb = 0; cb < s; cb += CH) {
            const int cs = min(CH, s - cb);
            for (int c = warp; c < cs; c += nw) {
                E* x = X + (long long)(cb + c) * n + b0;
                E v = lane < bs ? x[lane] : Elem<E>::zero();
                for (int k = 0; k < bs; ++k) {
                    E vk;
                    vk.re = __shfl_sync(0xffffffffu, v.re, k);
                    vk.im = __shfl_sync(0xffffffffu, v.im, k);
                    if (lane > k && lane < bs) cfms(v, D[lane][k], vk);
                }
                if (lane < bs) { x[lane] = v; xb[c * kLuNB + lane] = v; }
            }
            __syncthreads();
            for (int i = b0 + bs + threadIdx.x; i < n; i += blockDim.x) {
                E acc[CH];
#pragma unroll
                for (int c = 0; c < CH; ++c) acc[c] = Elem<E>::zero();
                for (int k = 0; k < bs; ++k) {
                    const E l = M[i + (long long)(b0 + k) * n];
#pragma unroll
                    for (int c = 0; c < CH; ++c)
                        if (c < cs) cfma(acc[c], l, xb[c * kLuNB + k]);
                }
#pragma unroll
                for (int c = 0; c < CH; ++c)
                    if (c < cs) X[i + (long long)(cb + c) * n] -= acc[c];
            }
            __syncthreads();
        }
    }
    for (int b0 = ((n - 1) / kLuNB) * kLuNB; b0 >= 0; b0 -= kLuNB) {
        const int bs = min(kLuNB, n - b0);
        for (int e = threadIdx.x; e < bs * bs; e += blockDim.x) {
            const int r = e % bs, k = e / bs;
            D[r][k] = M[(b0 + r) + (long long)(b0 + k) * n];
        }
        __syncthreads();
        for (int cb = 0; cb < s; cb += CH) {
            const int cs = min(CH, s - cb);
            for (int c = warp; c < cs; c += nw) {
                E* x = X + (long long)(cb + c) * n + b0;
                E v = lane < bs ? x[lane] : Elem<E>::zero();
                for (int k = bs - 1; k >= 0; --k) {
                    if (lane == k) v = cdiv(v, D[k][k]);
                    E vk;
                    vk.re = __shfl_sync(0xffffffffu, v.re, k);
                    vk.im = __shfl_sync(0xffffffffu, v.im, k);
                    if (lane < k) cfms(v, D[lane][k], vk);
                }
                if (lane < bs) { x[lane] = v; xb[c * kLuNB + lane] = v; }
            }
            __syncthreads();
            for (int i = threadIdx.x; i < b0; i += blockDim.x) {
                E acc[CH];
#pragma unroll
                for (int c = 0; c < CH; ++c) acc[c] = Elem<E>::zero();
                for (int k = 0; k < bs; ++k) {
                    const E u = M[i + (long long)(b0 + k) * n];
#pragma unroll
                    for (int c = 0; c < CH; ++c)
                        if (c < cs) cfma(acc[c], u, xb[c * kLuNB + k]);
                }
#pragma unroll
                for (int c = 0; c < CH; ++c)
                    if (c < cs) X[i + (long long)(cb + c) * n] -= acc[c];
            }
            __syncthreads();
        }
    }
}

// Warp-wide dot products sum_{k in [k_lo, k_hi)} conj(a[k]) X[k, c] for the cs
// columns of a chunk; the sums end up in every lane.
template <class E, int CH>
__device__ __forceinline__ void warp_dots_h(const E* a, const E* X, int n, int k_lo, int k_hi, int cs,
                                            E (&acc)[CH]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < CH; ++c) acc[c] = Elem<E>::zero();
    for (int k = k_lo + lane; k < k_hi; k += 32) {
        const E u = conj(a[k]);
#pragma unroll
        for (int c = 0; c < CH; ++c)
            if (c < cs) cfma(acc[c], u, X[k + (long long)c * n]);
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        if (c >= cs) break;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            acc[c].re += __shfl_xor_sync(0xffffffffu, acc[c].re, o);
            acc[c].im += __shfl_xor_sync(0xffffffffu, acc[c].im, o);
        }
    }
}

// X <- T^-H X:  T^H = U^H L^H P, so x = P^T L^-H U^-H b.  Left-looking by 32-row
// blocks (the sums run down columns of U and L, which are contiguous).
template <class E, int CH>
__device__ void lu_solve_h(const E* M, const int* perm, int n, E* X, int s, E* sm) {
    E* buf = sm;
    E (*D)[kLuNB + 1] = reinterpret_cast<E (*)[kLuNB + 1]>(sm + n);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int b0 = 0; b0 < n; b0 += kLuNB) {               // U^H y = b
        const int bs = min(kLuNB, n - b0);
        for (int e = threadIdx.x; e < bs * bs; e += blockDim.x) {
            const int r = e % bs, k = e / bs;
            D[r][k] = M[(b0 + r) + (long long)(b0 + k) * n];
        }
        for (int cb = 0; cb < s; cb += CH) {
            const int cs = min(CH, s - cb);
            E* Xc = X + (long long)cb * n;
            if (b0 > 0)
                for (int r = warp; r < bs; r += nw) {
                    E acc[CH];
                    warp_dots_h<E, CH>(M + (long long)(b0 + r) * n, Xc, n, 0, b0, cs, acc);
                    if (lane == 0)
#pragma unroll
                        for (int c = 0; c < CH; ++c)
                            if (c < cs) Xc[b0 + r + (long long)c * n] -= acc[c];
                }
            __syncthreads();
            for (int c = warp; c < cs; c += nw) {
                E* x = Xc + (long long)c * n + b0;
                E v = lane < bs ? x[lane] : Elem<E>::zero();
                for (int k = 0; k < bs; ++k) {
                    if (lane == k) v = cdiv(v, conj(D[k][k]));
                    E vk;
                    vk.re = __shfl_sync(0xffffffffu, v.re, k);
                    vk.im = __shfl_sync(0xffffffffu, v.im, k);
                    if (lane > k && lane < bs) cfms_c(v, D[k][lane], vk);
                }
                if (lane < bs) x[lane] = v;
            }
            __syncthreads();
        }
    }
    for (int b0 = ((n - 1) / kLuNB) * kLuNB; b0 >= 0; b0 -= kLuNB) {   // L^H z = y
        const int bs = min(kLuNB, n - b0);
        for (int e = threadIdx.x; e < bs * bs; e += blockDim.x) {
            const int r = e % bs, k = e / bs;
            D[r][k] = M[(b0 + r) + (long long)(b0 + k) * n];
        }
        for (int cb = 0; cb < s; cb += CH) {
            const int cs = min(CH, s - cb);
            E* Xc = X + (long long)cb * n;
            if (b0 + bs < n)
                for (int r = warp; r < bs; r += nw) {
                    E acc[CH];
                    warp_dots_h<E, CH>(M + (long long)(b0 + r) * n, Xc, n, b0 + bs, n, cs, acc);
                    if (lane == 0)
#pragma unroll
                        for (int c = 0; c < CH; ++c)
                            if (c < cs) Xc[b0 + r + (long long)c * n] -= acc[c];
                }
            __syncthreads();
            for (int c = warp; c < cs; c += nw) {
                E* x = Xc + (long long)c * n + b0;
                E v = lane < bs ? x[lane] : Elem<E>::zero();
                for (int k = bs - 1; k >= 0; --k) {
                    E vk;
                    vk.re = __shfl_sync(0xffffffffu, v.re, k);
                    vk.im = __shfl_sync(0xffffffffu, v.im, k);
                    if (lane < k) cfms_c(v, D[k][lane], vk);
                }
                if (lane < bs) x[lane] = v;
            }
            __syncthreads();
        }
    }
    permute_rows(X, n, s, perm, buf, true);
}

// One CTA per matrix: X_m <- T_m^-1 X_m (trans = 0) or T_m^-H X_m (trans = 1).
// grid (column groups, nmat): CTA (g, m) solves columns [g cpc, g cpc + cpc) of X_m,
// so that small batches still occupy the GPU (the factors are then re-read from L2).
template <class E, int CH>
__global__ void __launch_bounds__(kLuSolveThreads) k_lu_solve(int n, int s, int cpc, int trans, const E* LU,
                                                              long long stride, const int* perm, E* X,
                                                              long long xstride) {
    extern __shared__ double lu_solve_sm[];
    E* sm = reinterpret_cast<E*>(lu_solve_sm);
    const int c0 = blockIdx.x * cpc, cs = min(cpc, s - c0);
    if (cs <= 0) return;
    const E* M = LU + (long long)blockIdx.y * stride;
    const int* pm = perm + (long long)blockIdx.y * n;
    E* Xm = X + (long long)blockIdx.y * xstride + (long long)c0 * n;
    if (trans) lu_solve_h<E, CH>(M, pm, n, Xm, cs, sm);
    else lu_solve_n<E, CH>(M, pm, n, Xm, cs, sm);
}

// ---- few matrices or columns: one launch per 32-row block over all SMs
//
// k_lu_solve keeps a column group on one CTA, which reads all the factors by itself: a
// single matrix of order 3000 (complex64, 16 columns) took 4.4 ms that way, order 802
// (six matrices, 12 columns, complex128) 1.54 ms.  Here launch b of a triangular sweep
// subtracts the solved block b from the rows left (a CTA per 32 rows, CPC columns and
// matrix, its four warps splitting the block's columns), and the CTAs that hold the next
// block's rows multiply them at once by the inverse of its triangle.  The 32 x 32 inverses
// are made once per factorisation (k_diag_inv): substitution there, 32 dependent steps of
// FP64 FMAs and shuffles on one warp, was two thirds of a launch (14.8 us; 6 with them).
// A multiplication by a rounded inverse D of a triangle B leaves a residual of |B| |D| |B| |x|
// roundings where substitution leaves |B| |x|: with the nearly dependent columns of a smooth kernel
// inside a block, 1e5 times more.  So k_diag_cond estimates the norm of |D| |B| for each triangle.
// Up to kInvAlone the residuals are substitution's to a factor of about two (T(k), orders 160 to 240:
// half of the blocks below 20 to 55, the largest 55 to 215); up to kInvRefined one step of
// iterative refinement inside the block brings them there (its two products more); beyond, where
// the refinement need not converge, the block is solved by substitution.
// The launches of a sweep are programmatic dependents of one another: a launch comes up and
// reads its part of the factors, which no launch of the sweep writes, while the one before it
// still runs, and waits for that one's end before it touches X.
enum SolveSweep { kSweepL = 0, kSweepU = 1, kSweepUH = 2, kSweepLH = 3 };   // L y = b, U x = y; U^H y = b, L^H x = y

constexpr int kDinvBlock = kLuNB * kLuNB + 2;   // a block's inverses, then the estimates: L, U; L^H, U^H
constexpr float kInvAlone = 64.f;
template <class E>
constexpr float kInvRefined = std::is_same<E, cplx>::value ? 16777216.f : 1024.f;

size_t lu_dinv_elems(int n) { return (size_t)((n + kLuNB - 1) / kLuNB) * kDinvBlock; }

// Inverses of the diagonal blocks of L (unit: strictly lower part stored) and U (upper
// part) of every matrix: dinv[matrix][block][column][row].  grid (blocks, nmat, 4): a warp
// per column, eight columns a CTA, by substitution.
template <class E>
__global__ void __launch_bounds__(256) k_diag_inv(int n, const E* LU, long long stride, E* dinv) {
    __shared__ E W[kLuNB][kLuNB + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r0 = blockIdx.x * kLuNB, nr = min(kLuNB, n - r0);
    const E* M = LU + (long long)blockIdx.y * stride;
    E* out = dinv + ((long long)blockIdx.y * gridDim.x + blockIdx.x) * kDinvBlock;
    for (int e = threadIdx.x; e < kLuNB * kLuNB; e += blockDim.x) {   // beyond the matrix: the unit matrix
        const int r = e % kLuNB, k = e / kLuNB;
        W[r][k] = (r < nr && k < nr) ? M[(r0 + r) + (long long)(r0 + k) * n] : r == k ? Elem<E>::one() : Elem<E>::zero();
    }
    __syncthreads();
    const int c = blockIdx.z * 8 + warp;
    E v = lane == c ? Elem<E>::one() : Elem<E>::zero();               // L x = e_c
    for (int k = c; k < kLuNB; ++k) {
        E vk;
        vk.re = __shfl_sync(0xffffffffu, v.re, k);
        vk.im = __shfl_sync(0xffffffffu, v.im, k);
        if (lane > k) cfms(v, W[lane][k], vk);
    }
    const E lower = v;
    const E id = cdiv(Elem<E>::one(), W[lane][lane]);
    v = lane == c ? Elem<E>::one() : Elem<E>::zero();                 // U x = e_c
    for (int k = c; k >= 0; --k) {
        if (lane == k) v = v * id;
        E vk;
        vk.re = __shfl_sync(0xffffffffu, v.re, k);
        vk.im = __shfl_sync(0xffffffffu, v.im, k);
        if (lane < k) cfms(v, W[lane][k], vk);
    }
    out[c * kLuNB + lane] = lane > c ? lower : v;
}

// max(|re|, |im|) = f 2^e, 1 <= f < 2 (zero and subnormal: f = 0; Inf and NaN: f infinite)
__device__ __forceinline__ int size_of(cplx z, float& f) {
    const int m = max(__double2hiint(z.re) & 0x7fffffff, __double2hiint(z.im) & 0x7fffffff), e = m >> 20;
    f = e == 0 ? 0.f : e == 0x7ff ? INFINITY : __int_as_float(0x3f800000 | (m & 0xfffff) << 3);
    return e - 1023;
}
__device__ __forceinline__ int size_of(cplxf z, float& f) {
    const int m = max(__float_as_int(z.re) & 0x7fffffff, __float_as_int(z.im) & 0x7fffffff), e = m >> 23;
    f = e == 0 ? 0.f : e == 0xff ? INFINITY : __int_as_float(0x3f800000 | (m & 0x7fffff));
    return e - 127;
}
__device__ __forceinline__ float scaled(float f, int e) { return f > 0.f ? ldexpf(f, max(-300, min(300, e))) : 0.f; }

// The largest row sum of |D| |B| for the triangles B of a diagonal block as the sweeps apply them (L, U,
// L^H, U^H: a warp each) and their inverses D, to a factor of two, in FP32; rows of B and then its
// columns brought to the size of one by powers of two, so that the scaling of the matrix does not
// count.  grid (blocks, nmat); lane r has row r.
template <class E>
__global__ void __launch_bounds__(128) k_diag_cond(int n, const E* LU, long long stride, E* dinv) {
    const int lane = threadIdx.x & 31, up = (threadIdx.x >> 5) & 1, herm = threadIdx.x >> 6;
    const int r0 = blockIdx.x * kLuNB, nr = min(kLuNB, n - r0);
    const E* M = LU + (long long)blockIdx.y * stride;
    E* D = dinv + ((long long)blockIdx.y * gridDim.x + blockIdx.x) * kDinvBlock;
    float f[kLuNB];
    int e[kLuNB], re = -(1 << 20);
#pragma unroll
    for (int k = 0; k < kLuNB; ++k) {
        const int row = herm ? k : lane, col = herm ? lane : k;   // of the stored block
        const bool in = row < nr && col < nr;
        E z = in ? M[(r0 + row) + (long long)(r0 + col) * n] : Elem<E>::zero();
        if (up ? row > col : row < col) z = Elem<E>::zero();
        if (row == col && (!up || !in)) z = Elem<E>::one();
        e[k] = size_of(z, f[k]);
        if (f[k] > 0.f) re = max(re, e[k]);
    }
    int ce = 0;                    // column lane's exponent
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < kLuNB; ++k) {
        const int c = __reduce_max_sync(0xffffffffu, f[k] > 0.f ? e[k] - re : -(1 << 20));
        if (lane == k) ce = c;
        v += scaled(f[k], e[k] - re - c);
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kLuNB; ++k) {
        const int row = herm ? k : lane, col = herm ? lane : k;
        E z = D[col * kLuNB + row];
        if (up ? row > col : row < col) z = Elem<E>::zero();
        if (!up && row == col) z = Elem<E>::one();
        const int rk = __shfl_sync(0xffffffffu, re, k);
        const float vk = __shfl_sync(0xffffffffu, v, k);
        float g;
        const int q = size_of(z, g);
        s = fmaf(scaled(g, q + ce + rk), vk, s);
    }
    s = s >= 0.f ? s : INFINITY;   // NaN: 0 times infinity
    const float top = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(s)));
    if (lane == 0) {
        E* est = D + kLuNB * kLuNB + herm;
        (up ? est->im : est->re) = top;
    }
}

template <class E, int SWEEP, int CPC>
__global__ void __launch_bounds__(128) k_solve_step(int n, int s, int cur, const E* LU, long long stride,
                                                    const E* dinv, E* X, long long xstride) {
    constexpr bool ASC = SWEEP == kSweepL || SWEEP == kSweepUH, HERM = SWEEP >= 2;
    __shared__ E W[kLuNB][kLuNB + 1], D[kLuNB][kLuNB + 1];   // D[k][r]: entry (r, k) of the inverse as applied
    __shared__ E xs[CPC][kLuNB], part[4][CPC][kLuNB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = blockIdx.x;
    const int nb = (n + kLuNB - 1) / kLuNB;
    const int blk = ASC ? cur + 1 + t : cur - 1 - t;               // this CTA's rows
    const int c0 = blockIdx.y * CPC, cs = min(CPC, s - c0);
    const E* M = LU + (long long)blockIdx.z * stride;
    E* Xm = X + (long long)blockIdx.z * xstride + (long long)c0 * n;
    const int r0 = blk * kLuNB, nr = min(kLuNB, n - r0);
    asm volatile("griddepcontrol.launch_dependents;");
    float cond = 0.f;
    if (t == 0) {
        const E* Db = dinv + ((long long)blockIdx.z * nb + blk) * kDinvBlock;
        const E est = Db[kLuNB * kLuNB + (HERM ? 1 : 0)];
        cond = (float)(SWEEP == kSweepL || SWEEP == kSweepLH ? est.re : est.im);
        for (int c = warp; c < kLuNB; c += 4) {                    // (row lane, column c) of the stored inverses
            const E z = Db[c * kLuNB + lane];
            const bool low = lane > c;
            const E o = (SWEEP == kSweepL || SWEEP == kSweepLH) ? (low ? z : lane == c ? Elem<E>::one() : Elem<E>::zero())
                                                                : (low ? Elem<E>::zero() : z);
            if (HERM) D[lane][c] = conj(o);
            else D[c][lane] = o;
        }
    }
    const bool update = ASC ? cur >= 0 : cur < nb;
    const int k0 = cur * kLuNB, nk = min(kLuNB, n - k0);
    E w[8];
    if (update) {
        if (HERM) {   // conj(M[k, r]): columns r of the factor, contiguous in k
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int r = warp + 4 * q;
                W[lane][r] = (lane < nk && r < nr) ? conj(M[(k0 + lane) + (long long)(r0 + r) * n]) : Elem<E>::zero();
            }
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int k = 8 * warp + q;
                w[q] = (lane < nr && k < nk) ? M[(r0 + lane) + (long long)(k0 + k) * n] : Elem<E>::zero();
            }
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");   // X from here on
    E yold[CPC];
#pragma unroll
    for (int c = 0; c < CPC; ++c) yold[c] = (warp == 0 && c < cs && lane < nr) ? Xm[(long long)c * n + r0 + lane] : Elem<E>::zero();
    if (update) {
        for (int e = threadIdx.x; e < CPC * kLuNB; e += 128) {
            const int c = e / kLuNB, k = e - c * kLuNB;
            xs[c][k] = (c < cs && k < nk) ? Xm[(long long)c * n + k0 + k] : Elem<E>::zero();
        }
        __syncthreads();
        E acc[CPC];
#pragma unroll
        for (int c = 0; c < CPC; ++c) acc[c] = Elem<E>::zero();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k = 8 * warp + q;
            if (HERM) w[q] = W[k][lane];
#pragma unroll
            for (int c = 0; c < CPC; ++c) cfma(acc[c], w[q], xs[c][k]);
        }
#pragma unroll
        for (int c = 0; c < CPC; ++c) part[warp][c][lane] = acc[c];
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int c = 0; c < CPC; ++c) {
                yold[c] = yold[c] - ((part[0][c][lane] + part[1][c][lane]) + (part[2][c][lane] + part[3][c][lane]));
                if (t > 0 && c < cs && lane < nr) Xm[(long long)c * n + r0 + lane] = yold[c];
            }
        }
    }
    if (t > 0) return;
    // the next block: times the inverse of its triangle
    if (warp == 0)
#pragma unroll
        for (int c = 0; c < CPC; ++c) xs[c][lane] = yold[c];
    const bool exact = cond <= kInvAlone, refine = cond <= kInvRefined<E>;   // the CTA's
    if (!exact)   // the block's triangle as applied: W[k][r]
        for (int c = warp; c < kLuNB; c += 4) {
            E z = lane < nr && c < nr ? M[(r0 + lane) + (long long)(r0 + c) * n] : Elem<E>::zero();
            const bool low = lane > c, lower = SWEEP == kSweepL || SWEEP == kSweepLH;
            if (lane != c && low != lower) z = Elem<E>::zero();
            if (lane == c && (lower || lane >= nr)) z = Elem<E>::one();
            if (HERM) W[lane][c] = conj(z);
            else W[c][lane] = z;
        }
    __syncthreads();
    // part <- a block (columns k, lane r row r) times xs
    auto times = [&](const E (&B)[kLuNB][kLuNB + 1]) {
        E acc[CPC];
#pragma unroll
        for (int c = 0; c < CPC; ++c) acc[c] = Elem<E>::zero();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k = 8 * warp + q;
            const E w = B[k][lane];
#pragma unroll
            for (int c = 0; c < CPC; ++c) cfma(acc[c], w, xs[c][k]);
        }
#pragma unroll
        for (int c = 0; c < CPC; ++c) part[warp][c][lane] = acc[c];
        __syncthreads();
    };
    auto sum = [&](int c) { return (part[0][c][lane] + part[1][c][lane]) + (part[2][c][lane] + part[3][c][lane]); };
    if (!refine) {   // substitution, a warp per column
        if (warp >= cs) return;
        E v = xs[warp][lane];
        for (int q = 0; q < kLuNB; ++q) {
            const int k = ASC ? q : kLuNB - 1 - q;
            if (lane == k) v = v * D[k][k];
            E vk;
            vk.re = __shfl_sync(0xffffffffu, v.re, k);
            vk.im = __shfl_sync(0xffffffffu, v.im, k);
            if (ASC ? lane > k : lane < k) cfms(v, W[k][lane], vk);
        }
        if (lane < nr) Xm[(long long)warp * n + r0 + lane] = v;
        return;
    }
    times(D);
    if (!exact) {
        E x = Elem<E>::zero();   // warps below CPC: the column's first solution
        if (warp < CPC) xs[warp][lane] = x = sum(warp);
        __syncthreads();
        times(W);
        if (warp == 0) {
#pragma unroll
            for (int c = 0; c < CPC; ++c) xs[c][lane] = yold[c] - sum(c);
        }
        __syncthreads();
        times(D);
        if (warp < cs && lane < nr) Xm[(long long)warp * n + r0 + lane] = x + sum(warp);
        return;
    }
    if (warp < cs && lane < nr) Xm[(long long)warp * n + r0 + lane] = sum(warp);
}

// X <- P X (inverse: P^T X), a CTA per column
template <class E>
__global__ void __launch_bounds__(256) k_permute_rows(int n, const int* perm, E* X, long long xstride, int inverse) {
    extern __shared__ double perm_sm[];
    permute_rows(X + (long long)blockIdx.y * xstride + (long long)blockIdx.x * n, n, 1,
                 perm + (long long)blockIdx.y * n, reinterpret_cast<E*>(perm_sm), inverse != 0);
}

constexpr size_t kLuSmemLimit = 220 * 1024;

bool lu_solve_supported(int n) { return lu_solve_smem_bytes(n, sizeof(cplx)) <= kLuSmemLimit; }
bool lu_solve_supported_f32(int n) { return lu_solve_smem_bytes(n, sizeof(cplxf)) <= kLuSmemLimit; }

cudaError_t lu_perm_from_piv(int n, int nmat, const int* piv, int* perm, cudaStream_t st) {
    if (n < 1 || nmat < 1 || (size_t)n * sizeof(int) > kLuSmemLimit) return cudaErrorInvalidValue;
    if ((size_t)n * sizeof(int) > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_lu_perm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLuSmemLimit);
        if (e != cudaSuccess) return e;
    }
    k_lu_perm<<<nmat, 256, (size_t)n * sizeof(int), st>>>(n, piv, perm);
    return cudaGetLastError();
}

constexpr size_t kPanelClusterSmem = 200 * 1024;
int g_lu_cluster_panels = 1;   // 0: tall panels in global memory (kept for comparison tests)
int g_lu_tensor_cores = 1;     // trailing updates on the tensor cores (complex64 and complex128)

void lu_set_cluster_panels(int on) { g_lu_cluster_panels = on ? 1 : 0; }
void lu_set_tensor_cores(int on) { g_lu_tensor_cores = on ? 1 : 0; }
int lu_get_cluster_panels() { return g_lu_cluster_panels; }
int lu_get_tensor_cores() { return g_lu_tensor_cores; }

cudaError_t launch_cgemm_f32(int m, int n, int k, const cplxf* A, long long lda, long long sa, const cplxf* B,
                             long long ldb, long long sb, cplxf* C, long long ldc, long long sc, int nmat,
                             int use_tc, int* err, cudaStream_t st);

size_t panel_smem(int rows, int nb, size_t esz) { return (size_t)rows * (nb + 1) * esz; }

// CTAs per matrix that a panel of m rows is best split over when nmat matrices share the
// 152 SMs: as long as a CTA keeps enough rows that its share of a column's work is not less
// than the column's cluster barrier (about a microsecond; complex128: 64 rows, 16 columns on
// average, 4 FMAs at two lanes a cycle: 2 us; complex64, 96 rows: order 3000 takes 89 us a panel
// on 16 CTAs, 129 on 8).
template <class E>
int panel_split(int m, int nmat) {
    const int least = std::is_same<E, cplx>::value ? 64 : 96;
    int cs = 1;
    while (cs < 16 && 2LL * cs * nmat <= 152 && m / (2 * cs) >= least) cs *= 2;
    return cs;
}

cudaError_t launch_zgemm_tc(int m, int n, int k, const cplx* A, long long lda, long long sa, const cplx* B, long long ldb,
                            long long sb, cplx* C, long long ldc, long long sc, const int* ek, long long se, int nmat,
                            int* info, cudaStream_t st);

// Cluster launch of the panel factorisation: when the panel is too tall for one CTA, or to
// split it over `want` CTAs.  Returns with *launched = false (nothing launched) when no
// cluster size up to 16 holds the panel or the device cannot co-schedule such a cluster.
template <class E>
cudaError_t launch_panel_cluster(int n, int k0, int nb, int nmat, E* A, long long stride, int* piv, int* info, int want,
                                 cudaStream_t st, bool* launched) {
    *launched = false;
    const int m = n - k0;
    int cs = 2, ci = 0;
    size_t R = 0, smem = 0;
    for (; cs <= 16; cs *= 2, ++ci) {
        R = (m + cs - 1) / cs;
        smem = panel_smem((int)R, nb, sizeof(E));
        if (smem <= kPanelClusterSmem && cs >= want) break;
    }
    if (cs > 16 || (long long)nmat * cs > 0x7fffffffLL) return cudaSuccess;
    static int ok[4] = {-1, -1, -1, -1};     // per cluster size 2, 4, 8, 16: unknown / no / yes
    cudaError_t e = cudaFuncSetAttribute(k_lu_panel_cluster<E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kPanelClusterSmem);
    if (e != cudaSuccess) return e;
    if (cs == 16) {
        e = cudaFuncSetAttribute(k_lu_panel_cluster<E>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return cudaSuccess;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nmat * cs));
    cfg.blockDim = dim3(kLuClusterThreads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (ok[ci] < 0) {
        cfg.dynamicSmemBytes = kPanelClusterSmem;
        int ncl = 0;
        e = cudaOccupancyMaxActiveClusters(&ncl, k_lu_panel_cluster<E>, &cfg);
        if (e != cudaSuccess) cudaGetLastError();
        ok[ci] = (e == cudaSuccess && ncl > 0) ? 1 : 0;
    }
    if (!ok[ci]) return cudaSuccess;
    cfg.dynamicSmemBytes = smem;
    e = cudaLaunchKernelEx(&cfg, k_lu_panel_cluster<E>, n, k0, nb, (int)R, A, stride, piv, info);
    *launched = e == cudaSuccess;
    return e;
}

template <class E>
cudaError_t lu_factor_impl(int n, int nmat, E* A, long long stride, int* piv, int* perm, int* info, cudaStream_t st,
                           long long* launches, int* tc_err) {
    if (n < 1 || nmat < 1 || nmat > 65535 || (size_t)n * sizeof(int) > kLuSmemLimit) return cudaErrorInvalidValue;
    const size_t gemm_smem = 2 * (size_t)kLuNB * kLuTile * sizeof(E);
    cudaError_t e = cudaFuncSetAttribute(k_lu_gemm<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_lu_panel<E, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLuSmemLimit);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(info, 0, (size_t)nmat * sizeof(int), st);
    if (e != cudaSuccess) return e;
    long long nl = 0;
    const int ncb = (n + kLuNB - 1) / kLuNB;
    // one 32-column panel: factor, exchange and solve the columns below cmax, update
    // the trailing columns below cend
    auto panel = [&](int k0, int nb) -> cudaError_t {
        const size_t psm = panel_smem(n - k0, nb, sizeof(E));
        const bool fits = psm <= kLuSmemLimit;
        bool launched = false;
        if (g_lu_cluster_panels)
            for (int want = panel_split<E>(n - k0, nmat); !launched && (want > 1 || !fits); want /= 2) {
                cudaError_t e2 = launch_panel_cluster<E>(n, k0, nb, nmat, A, stride, piv, info, want, st, &launched);
                if (e2 != cudaSuccess) return e2;
                if (want <= 1) break;
            }
        if (!launched && fits) k_lu_panel<E, true><<<nmat, kLuPanelThreads, psm, st>>>(n, k0, nb, A, stride, piv, info);
        else if (!launched) k_lu_panel<E, false><<<nmat, kLuPanelThreads, 0, st>>>(n, k0, nb, A, stride, piv, info);
        ++nl;
        return cudaGetLastError();
    };
    auto panel_step = [&](int k0, int nb, int cmax, int cend) -> cudaError_t {
        if (cudaError_t e2 = panel(k0, nb); e2 != cudaSuccess) return e2;
        if (ncb > 1) {
            k_lu_swap_trsm<E><<<dim3((n + kLuSwapCols - 1) / kLuSwapCols, nmat), kLuSwapCols * 8, 0, st>>>(
                n, k0, nb, A, stride, piv, cmax, nullptr);
            ++nl;
        }
        const int t0 = k0 + nb;
        if (t0 < n && cend > t0) {
            const int rt = (n - t0 + kLuTile - 1) / kLuTile, ct = (cend - t0 + kLuTile - 1) / kLuTile;
            k_lu_gemm<E><<<dim3(rt, ct, nmat), 256, gemm_smem, st>>>(n, k0, nb, A, stride, cend);
            ++nl;
        }
        return cudaGetLastError();
    };
    bool two_level = false;
    if constexpr (std::is_same<E, cplxf>::value) two_level = tc_err && g_lu_tensor_cores && n >= 2 * kLuBlock;
    if (two_level) {
        // complex64 with tensor cores: 128-column blocks.  Inside a block its four
        // panels update only the block's own columns; then the block's exchanges and
        // triangular solve reach the columns right of it once, and the trailing matrix
        // takes one update of depth 128 on the tensor cores (3xTF32), instead of four
        // of depth 32 -- a quarter of the trailing matrix's reads and writes.
        if constexpr (std::is_same<E, cplxf>::value) {
            const size_t blk_smem = (size_t)kLuBlock * (kLuBlock + 1) * sizeof(E);
            e = cudaFuncSetAttribute(k_lu_swap_trsm_block<E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)blk_smem);
            if (e != cudaSuccess) return e;
            for (int K0 = 0; K0 < n; K0 += kLuBlock) {
                const int kb = min(kLuBlock, n - K0), cmax = K0 + kb;
                for (int k0 = K0; k0 < cmax; k0 += kLuNB) {
                    e = panel_step(k0, min(kLuNB, cmax - k0), cmax, cmax);
                    if (e != cudaSuccess) return e;
                }
                const int m = n - cmax;
                if (m > 0) {
                    const size_t sm = (size_t)kb * (kb + 1) * sizeof(E);
                    k_lu_swap_trsm_block<E><<<dim3((m + kLuNB - 1) / kLuNB, nmat), 256, sm, st>>>(n, K0, kb, A, stride,
                                                                                                   piv);
                    ++nl;
                    e = launch_cgemm_f32(m, m, kb, A + cmax + (long long)K0 * n, n, stride, A + K0 + (long long)cmax * n,
                                         n, stride, A + cmax + (long long)cmax * n, n, stride, nmat, 1, tc_err, st);
                    if (e != cudaSuccess) return e;
                    ++nl;
                }
            }
        }
    } else {
        int* ek = nullptr;   // exponents of U's rows, in perm, which is written last
        if (std::is_same<E, cplx>::value && g_lu_tensor_cores && n >= kLuTcMin + kLuNB) {
            ek = perm;
            e = cudaMemsetAsync(ek, 0, (size_t)nmat * n * sizeof(int), st);
            if (e != cudaSuccess) return e;
        }
        for (int k0 = 0; k0 < n; k0 += kLuNB) {
            const int nb = min(kLuNB, n - k0);
            e = panel(k0, nb);
            if (e != cudaSuccess) return e;
            if (ncb > 1) {
                k_lu_swap_trsm<E><<<dim3((n + kLuSwapCols - 1) / kLuSwapCols, nmat), kLuSwapCols * 8, 0, st>>>(
                    n, k0, nb, A, stride, piv, n, n - k0 - nb >= kLuTcMin ? ek : nullptr);
                ++nl;
            }
            const int m = n - k0 - nb;
            if (m > 0) {
                bool done = false;
                if constexpr (std::is_same<E, cplxf>::value) {
                    // complex64: A22 -= L21 U12 on the tensor cores (3xTF32) once the trailing
                    // block spans at least one 128-row tile
                    if (tc_err && g_lu_tensor_cores && m >= 128) {
                        const int t0 = k0 + nb;
                        e = launch_cgemm_f32(m, m, nb, A + t0 + (long long)k0 * n, n, stride, A + k0 + (long long)t0 * n,
                                             n, stride, A + t0 + (long long)t0 * n, n, stride, nmat, 1, tc_err, st);
                        if (e != cudaSuccess) return e;
                        done = true;
                    }
                }
                if constexpr (std::is_same<E, cplx>::value) {
                    // complex128: the same as exact BF16 digit products (zgemm_tc.cu)
                    if (ek && m >= kLuTcMin) {
                        const int t0 = k0 + nb;
                        e = launch_zgemm_tc(m, m, nb, A + t0 + (long long)k0 * n, n, stride, A + k0 + (long long)t0 * n, n,
                                            stride, A + t0 + (long long)t0 * n, n, stride, ek + k0, n, nmat, info, st);
                        if (e != cudaSuccess) return e;
                        done = true;
                    }
                }
                if (!done) {
                    const int tiles = (m + kLuTile - 1) / kLuTile;
                    k_lu_gemm<E><<<dim3(tiles, tiles, nmat), 256, gemm_smem, st>>>(n, k0, nb, A, stride, n);
                }
                ++nl;
            }
        }
    }
    e = lu_perm_from_piv(n, nmat, piv, perm, st);
    ++nl;
    if (launches) *launches += nl;
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

template <class E, int CPC>
cudaError_t lu_solve_steps(int n, int nmat, int trans, const E* LU, long long stride, const int* perm, const E* dinv,
                           int s, E* X, long long xstride, cudaStream_t st) {
    const size_t psm = (size_t)n * sizeof(E);
    if (cudaError_t e = cudaFuncSetAttribute(k_permute_rows<E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kLuSmemLimit);
        e != cudaSuccess)
        return e;
    const int nb = (n + kLuNB - 1) / kLuNB, cg = (s + CPC - 1) / CPC;
    // the first launch of a sweep waits for all before it, the others only where they say so
    cudaError_t e = cudaSuccess;
    auto sweep = [&](auto kernel, bool asc) {
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.blockDim = dim3(128);
        cfg.stream = st;
        cfg.attrs = at;
        for (int q = -1; q < nb - 1 && e == cudaSuccess; ++q) {
            const int cur = asc ? q : nb - 1 - q, tiles = q < 0 ? 1 : nb - 1 - q;
            cfg.gridDim = dim3(tiles, cg, nmat);
            cfg.numAttrs = q < 0 ? 0 : 1;
            e = cudaLaunchKernelEx(&cfg, kernel, n, s, cur, LU, stride, dinv, X, xstride);
        }
    };
    if (trans) {
        sweep(k_solve_step<E, kSweepUH, CPC>, true);
        sweep(k_solve_step<E, kSweepLH, CPC>, false);
        k_permute_rows<E><<<dim3(s, nmat), 256, psm, st>>>(n, perm, X, xstride, 1);
    } else {
        k_permute_rows<E><<<dim3(s, nmat), 256, psm, st>>>(n, perm, X, xstride, 0);
        sweep(k_solve_step<E, kSweepL, CPC>, true);
        sweep(k_solve_step<E, kSweepU, CPC>, false);
    }
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

// Whether a solve takes the launches per block: few columns in all (below four per SM a CTA
// per column group leaves SMs idle, and its time is one CTA's).  Measured, T^-1 X with 12
// columns a matrix, ms, a CTA per column group -> launches per block: order 128, 1 matrix
// 0.177 -> 0.112; 512, 1: 0.766 -> 0.320; 802, 6: 1.54 -> 1.00; 1600, 16: 6.69 -> 4.92; 64 matrices:
// order 256 0.678 -> 0.820, order 512 2.21 -> 2.31.
bool lu_solve_in_steps(int n, int nmat, int s) { return n >= 128 && (long long)nmat * s < 608; }

template <class E>
cudaError_t lu_diag_inv(int n, int nmat, const E* LU, long long stride, E* dinv, cudaStream_t st) {
    k_diag_inv<E><<<dim3((n + kLuNB - 1) / kLuNB, nmat, 4), 256, 0, st>>>(n, LU, stride, dinv);
    k_diag_cond<E><<<dim3((n + kLuNB - 1) / kLuNB, nmat), 128, 0, st>>>(n, LU, stride, dinv);
    return cudaGetLastError();
}

// dinv: the factors' lu_diag_inv (nmat x lu_dinv_elems(n)), or null (a CTA per column group)
template <class E>
cudaError_t lu_solve_impl(int n, int nmat, int trans, const E* LU, long long stride, const int* perm, const E* dinv,
                          int s, E* X, long long xstride, cudaStream_t st) {
    const size_t smem = lu_solve_smem_bytes(n, sizeof(E));
    if (n < 1 || nmat < 1 || nmat > 65535 || s < 1 || smem > kLuSmemLimit) return cudaErrorInvalidValue;
    if (dinv && lu_solve_in_steps(n, nmat, s)) {
        if ((long long)nmat * s <= 32)
            return lu_solve_steps<E, 1>(n, nmat, trans, LU, stride, perm, dinv, s, X, xstride, st);
        return lu_solve_steps<E, 2>(n, nmat, trans, LU, stride, perm, dinv, s, X, xstride, st);
    }
    // columns per CTA: a power of two <= 16 (the register chunk is exactly that wide,
    // so no lane computes for absent columns), the widest that still gives about two
    // CTAs per SM of the 152, which re-reads the factors least
    int cpc = 16;
    while (cpc > 1 && (long long)nmat * ((s + cpc - 1) / cpc) < 304) cpc >>= 1;
    while (cpc > 1 && cpc / 2 >= s) cpc >>= 1;
    const int ng = (s + cpc - 1) / cpc;
    const dim3 grid(ng, nmat);
    cudaError_t e = cudaSuccess;
    switch (cpc) {
#define HB_SOLVE_CASE(CHV)                                                                                       \
    case CHV:                                                                                                    \
        e = cudaFuncSetAttribute(k_lu_solve<E, CHV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLuSmemLimit); \
        if (e != cudaSuccess) return e;                                                                          \
        k_lu_solve<E, CHV><<<grid, kLuSolveThreads, smem, st>>>(n, s, cpc, trans, LU, stride, perm, X, xstride); \
        break;
        HB_SOLVE_CASE(1)
        HB_SOLVE_CASE(2)
        HB_SOLVE_CASE(4)
        HB_SOLVE_CASE(8)
        HB_SOLVE_CASE(16)
#undef HB_SOLVE_CASE
    }
    return cudaGetLastError();
}

cudaError_t lu_factor_batched(int n, int nmat, cplx* A, long long stride, int* piv, int* perm, int* info,
                              cudaStream_t st, long long* launches) {
    return lu_factor_impl<cplx>(n, nmat, A, stride, piv, perm, info, st, launches, nullptr);
}
cudaError_t lu_factor_batched_f32(int n, int nmat, cplxf* A, long long stride, int* piv, int* perm, int* info,
                                  cudaStream_t st, long long* launches, int* tc_err) {
    return lu_factor_impl<cplxf>(n, nmat, A, stride, piv, perm, info, st, launches, tc_err);
}
cudaError_t lu_solve_batched(int n, int nmat, int trans, const cplx* LU, long long stride, const int* perm,
                             const cplx* dinv, int s, cplx* X, long long xstride, cudaStream_t st) {
    return lu_solve_impl<cplx>(n, nmat, trans, LU, stride, perm, dinv, s, X, xstride, st);
}
cudaError_t lu_solve_batched_f32(int n, int nmat, int trans, const cplxf* LU, long long stride, const int* perm,
                                 const cplxf* dinv, int s, cplxf* X, long long xstride, cudaStream_t st) {
    return lu_solve_impl<cplxf>(n, nmat, trans, LU, stride, perm, dinv, s, X, xstride, st);
}
cudaError_t lu_diag_inv_batched(int n, int nmat, const cplx* LU, long long stride, cplx* dinv, cudaStream_t st) {
    return lu_diag_inv<cplx>(n, nmat, LU, stride, dinv, st);
}
cudaError_t lu_diag_inv_batched_f32(int n, int nmat, const cplxf* LU, long long stride, cplxf* dinv, cudaStream_t st) {
    return lu_diag_inv<cplxf>(n, nmat, LU, stride, dinv, st);
}

}  // namespace hbem
