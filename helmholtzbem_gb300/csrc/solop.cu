// Mass projection of T(k) (gen_sol_op.cpp:45-48): T_proj = F^-1 T F^-T with
// F = blockdiag(L, L), L the Cholesky factor of the P1 mass matrix M.  M is
// cyclic tridiagonal, so L is lower bidiagonal plus a dense last row (the fill
// of the wrap-around coupling): every solve is an O(N) recurrence.
//   diag inverse  id[i] = 1/L[i][i]
//   sub           sb[i] = L[i+1][i]          (i < N-1; sb[N-2] is also the last row's)
//   last row      lr[i] = L[N-1][i]          (i < N-1)
#include "hbem_device.cuh"

namespace hbem {

struct CholView {
    int N;
    const double* id;
    const double* sb;
    const double* lr;
};

// forward substitution L z = t on a strided vector, in place.  The entries are loaded
// kRun at a time, the next run before the present one is used: the recurrence is two
// dependent FMAs per entry, a load each as long as ten of them.
constexpr int kRun = 8;
__device__ __forceinline__ void chol_solve_strided(const CholView& L, cplx* x, long long stride) {
    const int N = L.N;
    cplx acc = mk(0.);                        // sum_{i < N-1} lr[i] z[i]
    cplx zprev = mk(0.);
    cplx cur[kRun], nxt[kRun];
#pragma unroll
    for (int q = 0; q < kRun; ++q) cur[q] = q < N ? x[q * stride] : mk(0.);
    for (int i0 = 0; i0 < N - 1; i0 += kRun) {
#pragma unroll
        for (int q = 0; q < kRun; ++q) nxt[q] = i0 + kRun + q < N ? x[(i0 + kRun + q) * stride] : mk(0.);
#pragma unroll
        for (int q = 0; q < kRun; ++q) {
            const int i = i0 + q;
            if (i >= N - 1) break;
            cplx t = cur[q];
            if (i > 0) { t.re -= L.sb[i - 1] * zprev.re; t.im -= L.sb[i - 1] * zprev.im; }
            cplx z = L.id[i] * t;
            x[i * stride] = z;
            axpy(acc, L.lr[i], z);
            zprev = z;
        }
#pragma unroll
        for (int q = 0; q < kRun; ++q) cur[q] = nxt[q];
    }
    const long long last = (long long)(N - 1) * stride;
    x[last] = L.id[N - 1] * (x[last] - acc);
}

// Y = T F^-T: each thread owns one row r of one matrix and one of its two column blocks.
__global__ void k_proj_rows(CholView L, cplx* T, long long mat_stride, int nmat) {
    const int n = 2 * L.N;
    long long gid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    long long tot = 2LL * nmat * n;
    if (gid >= tot) return;
    const int r = (int)(gid % n);
    const long long m = gid / n;
    chol_solve_strided(L, T + (m >> 1) * mat_stride + (m & 1) * (long long)L.N * n + r, n);
}

// T_proj = F^-1 Y: the same along columns.  A column is contiguous in memory, so a warp takes
// 32 columns through shared memory: 32 x 32 tiles in, the recurrence with a lane per column,
// tiles out.
constexpr int kColWarps = 2;
__global__ void __launch_bounds__(32 * kColWarps) k_proj_cols(CholView L, cplx* T, long long mat_stride, int nmat) {
    __shared__ cplx tile[kColWarps][32][33];
    const int n = 2 * L.N, N = L.N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int groups = (n + 31) / 32;                                   // 32-column groups of a matrix
    const long long w = blockIdx.x * (long long)kColWarps + warp;       // (matrix, half of the rows, group)
    if (w >= 2LL * nmat * groups) return;                               // whole warp
    const int g = (int)(w % groups);
    const long long m = w / groups;
    cplx* A = T + (m >> 1) * mat_stride + (m & 1) * N + (long long)g * 32 * n;
    const int cols = min(32, n - g * 32);
    cplx (*t)[33] = tile[warp];                                         // [column][row]
    cplx acc = mk(0.), zprev = mk(0.), cur[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) cur[c] = (c < cols && lane < N) ? A[lane + (long long)c * n] : mk(0.);
    for (int i0 = 0; i0 < N; i0 += 32) {
#pragma unroll
        for (int c = 0; c < 32; ++c) t[c][lane] = cur[c];
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 32; ++c)   // the next tile's loads under this one's recurrence
            cur[c] = (c < cols && i0 + 32 + lane < N) ? A[i0 + 32 + lane + (long long)c * n] : mk(0.);
        const int rows = min(32, N - i0);
        for (int q = 0; q < rows; ++q) {
            const int i = i0 + q;
            cplx v = t[lane][q];
            if (i < N - 1) {
                if (i > 0) { v.re -= L.sb[i - 1] * zprev.re; v.im -= L.sb[i - 1] * zprev.im; }
                zprev = L.id[i] * v;
                axpy(acc, L.lr[i], zprev);
            } else {
                zprev = L.id[i] * (v - acc);
            }
            t[lane][q] = zprev;
        }
        __syncwarp();
        for (int c = 0; c < cols; ++c)
            if (lane < rows) A[i0 + lane + (long long)c * n] = t[c][lane];
        __syncwarp();
    }
}

cudaError_t launch_projection(int N, const double* id, const double* sb, const double* lr, cplx* T, int nmat,
                              cudaStream_t st) {
    CholView L{N, id, sb, lr};
    const long long n = 2LL * N, tot = 2 * nmat * n, warps = 2LL * nmat * ((n + 31) / 32);
    k_proj_rows<<<(unsigned)((tot + 63) / 64), 64, 0, st>>>(L, T, n * n, nmat);
    k_proj_cols<<<(unsigned)((warps + kColWarps - 1) / kColWarps), 32 * kColWarps, 0, st>>>(L, T, n * n, nmat);
    return cudaGetLastError();
}

// T, T' (and T'' when d = 2) at x_q = x_src + h_q (q < nq <= 2) from T, T', T'' at
// x_src (src: three n x n matrices one after another) by their Taylor polynomials,
//   T(x_q) = T + h T' + h^2/2 T'',  T'(x_q) = T' + h T'',  T''(x_q) = T'',
// into dst = [q][0 .. d].  The terms left out are h^3/6 T''', h^2/2 T''' and h T''':
// for |h| <= 1e-6 (T''' of the order of (sqrt(c) r)^2 T' for panel distances r) they
// are below 1e-11 of T' and T, and T'' (which only sets a Newton step's length) is
// good to ~1e-5.
__global__ void k_taylor_near(long long mat, const cplx* src, int nq, double h0, double h1, int d, cplx* dst) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= mat) return;
    const cplx t0 = src[e], t1 = src[mat + e], t2 = src[2 * mat + e];
    for (int q = 0; q < nq; ++q) {
        const double h = q ? h1 : h0;
        cplx* o = dst + (long long)q * (d + 1) * mat;
        o[e] = t0 + h * (t1 + (0.5 * h) * t2);
        o[mat + e] = t1 + h * t2;
        if (d == 2) o[2 * mat + e] = t2;
    }
}

cudaError_t launch_taylor_near(long long mat, const cplx* src, int nq, double h0, double h1, int d, cplx* dst,
                               cudaStream_t st) {
    if (nq < 1 || nq > 2 || d < 1 || d > 2) return cudaErrorInvalidValue;
    k_taylor_near<<<(unsigned)((mat + 255) / 256), 256, 0, st>>>(mat, src, nq, h0, h1, d, dst);
    return cudaGetLastError();
}

}  // namespace hbem
