// Coincident and adjacent panel pairs at real wavenumbers (included by assemble.cu).
//
// Two forms of the same quadrature sum:
//
// * k_singular_nodes, for builders small enough to keep a table: with f(u) = H0(sqrt u) and
//   g(u) = H1(sqrt u) / sqrt u (hankel_u.cuh), u = ks^2 |v|^2,
//       f = a0 + i [2/pi (lambda + log(|v|/s)) a0 + b0],
//       g = a1 + i [2/pi (lambda + log(|v|/s)) a1 + b1 - 2/(pi u)],
//   lambda = log(ks s / 2) + gamma, s the power of two next above D (so that the two logarithms
//   stay of the size of their sum: with s = 1 their rounding showed in W at 4e-15),
//   where a0, b0, a1, b1 are entire functions of u.  On a pair u runs over [0, ks^2 D^2], and
//   for ks D <= 8 their interpolants at 16 Chebyshev nodes of |v|^2 / D^2 are exact to 5e-17
//   (their Chebyshev coefficients fall like J_m(ks D / 2)^2).  So the sum over the pair's
//   n_c^2 (or 2 n_c^2) points is a sum over 16 nodes whose weights -- the points' weights
//   against the nodes' Lagrange polynomials, plain and times log(|v|/s) -- do not depend on the
//   wavenumber: they are made once per builder (k_snode_part, k_snode_join).  Order 11: 16
//   node values instead of 4225 or 8450 points.
// * k_singular_rows, for everything else: the points themselves.  A thread takes pieces of
//   the rows of one outer node; f and g come from the Hankel table, and along a row two
//   moments per kernel value are enough (see k_general).
#pragma once

namespace hbem {

constexpr int kSN = 16;                  // nodes per pair
constexpr double kSNodeX = 8.;           // largest ks D the nodes serve
// per task: [node][moment (S, L, T, W: 4 each)][plain, 2/pi log], then sum W / |v|^2 for L
// and T (8), D^2, s, padding
constexpr int kSNodeStride = kSN * 16 * 2 + 16;

// Panel map on [0, 1] or reversed, with the constants of pan_op01 / pan_swapped taken
// out of the loops (same expressions, same rounding).
struct PMap {
    int line;
    double bx, by, dx, dy, ph, dph, r, rd, sgn, tn;
};

__device__ __forceinline__ PMap make_pmap(const double* P, int kind, bool swapped) {
    PMap m;
    m.line = kind == 0;
    m.sgn = swapped ? -1. : 1.;
    if (kind == 0) {
        const double ex = P[2] - P[0], ey = P[3] - P[1];
        m.bx = swapped ? P[2] : P[0];
        m.by = swapped ? P[3] : P[1];
        m.dx = swapped ? -ex : ex;
        m.dy = swapped ? -ey : ey;
        m.ph = m.dph = m.r = m.rd = 0.;
        m.tn = hypot(ex, ey);
    } else {
        m.bx = P[0];
        m.by = P[1];
        m.dx = m.dy = 0.;
        m.r = P[2];
        m.ph = swapped ? P[4] : P[3];
        m.dph = swapped ? P[3] - P[4] : P[4] - P[3];
        m.rd = swapped ? -(P[2] * m.dph) : P[2] * m.dph;
        m.tn = P[2] * fabs(m.dph);
    }
    return m;
}

// point and forward tangent
__device__ __forceinline__ cplx pmap_at(const PMap& m, double t, cplx& tan) {
    if (m.line) {
        tan = mk(m.sgn * m.dx, m.sgn * m.dy);
        return mk(fma(m.dx, t, m.bx), fma(m.dy, t, m.by));
    }
    double s, c;
    sincos(fma(t, m.dph, m.ph), &s, &c);
    tan = mk(-m.rd * s, m.rd * c);
    return mk(m.bx + m.r * c, m.by + m.r * s);
}

// the maps of a task's panels (adjacent pairs: the common end point at parameter 0 of both)
__device__ __forceinline__ void task_maps(const DevMesh& M, const SingularTask& T, PMap& mi, PMap& mj) {
    const bool adj = T.kind == PK_ADJ;
    mi = make_pmap(M.par + 5 * T.i, M.kind[T.i], adj && !T.swap);
    mj = make_pmap(M.par + 5 * T.j, M.kind[T.j], adj && T.swap);
}

// upper bound of |v|^2 over the pair: the sum of the panels' lengths (one length when coincident)
__device__ __forceinline__ double task_d2(const SingularTask& T, const PMap& mi, const PMap& mj) {
    const double D = (T.kind == PK_ADJ ? mi.tn + mj.tn : mi.tn) * (1. + 1e-9);
    return D * D;
}

// the power of two next above the square root of d2
__device__ __forceinline__ double task_scale(double d2) {
    int e;
    frexp(sqrt(d2), &e);
    return ldexp(1., e);
}

// the blocks of one pair from its moments, by `nthr` threads (16 work items); the first
// shape function is reversed on the panel that an adjacent pair's map reverses
template <int D, bool CURVED>
__device__ __forceinline__ void singular_store(const DevMesh& M, const SingularTask& T, const KConst& K,
                                               const cplx* mom, int tid, int nthr, cplx* out) {
    const bool adj = T.kind == PK_ADJ, rx = adj && !T.swap, ry = adj && T.swap;
    const uint8_t fl = M.flags[tri_index(T.i, T.j)];
    const cplx ti = M.gtan[T.i * M.p], tj = M.gtan[T.j * M.p];
    for (int it = tid; it < 16; it += nthr)
        block_entry<D, CURVED>(K, mom, it >> 2, it & 3, rx, ry, M.gtn[T.i * M.p] * M.gtn[T.j * M.p],
                               (fl & PF_TDT0_ZERO) ? 0. : 2. * (ti.im * tj.im + ti.re * tj.re), out);
}

// ------------------------------------------------------------------ the points themselves

template <int D, bool CURVED>
struct RowDims {
    static constexpr int F = D + 1, SETS = CURVED ? 4 : 3, NA = SETS * F * 4;   // moments of a pair
    static constexpr size_t kSmem = ((size_t)NA * 128 + NA) * sizeof(cplx);
};

// Pieces a row of nc inner nodes is cut into so that `rows` rows fill rounds of 128 threads:
// the threads of a warp take pieces of equal length (a run of points per thread, whose rows
// ended at different steps in every lane, left a warp idle 40 % of its issue slots).  A
// piece costs its points (about 45 FP64 instructions) and one fold (about 50).
__device__ __forceinline__ int row_pieces(int rows, int nc) {
    int best = 1, cost = 0x7fffffff;
    for (int c = 1; c <= 16 && c <= nc; ++c) {
        const int t = (rows * c + 127) / 128 * ((nc + c - 1) / c * 45 + 50);
        if (t < cost) { cost = t; best = c; }
    }
    return best;
}

// Moments of part `sub` of `nparts` equal parts of a pair's rows, reduced over the CTA
// (128 threads) into mom[NA] (shared memory).  acc: NA x 128 entries; sz: the composite nodes z
// (adjacent pairs) or 1 - z (coincident ones).
template <int D, bool CURVED>
__device__ __forceinline__ void singular_moments(const DevMesh& M, const SingularTask& T, const KConst& K, int sub,
                                                 int nparts, const double* sxc, const double* swc, const double* sz,
                                                 cplx* acc, cplx* mom) {
    typedef RowDims<D, CURVED> R;
    constexpr int F = R::F;
    const bool coinc = T.kind == PK_COINC;
    const int nc = M.nc, nrows = (coinc ? 1 : 2) * nc;
    const uint8_t fl = M.flags[tri_index(T.i, T.j)];
    const double ks2 = K.ks.re * K.ks.re;
    PMap mi, mj;
    task_maps(M, T, mi, mj);
    cplx* A = acc + threadIdx.x;
#pragma unroll
    for (int e = 0; e < R::NA; ++e) A[e * 128] = mk(0.);
    const int ra = nrows * sub / nparts, rb = nrows * (sub + 1) / nparts, pieces = row_pieces(rb - ra, nc);
    for (int it = ra * pieces + threadIdx.x; it < rb * pieces; it += 128) {
        const int row = it / pieces, piece = it - row * pieces, K0 = row >= nc ? 1 : 0, a = row - K0 * nc;
        const int z0 = nc * piece / pieces, z1 = nc * (piece + 1) / pieces;
        const double t = sxc[a], wt = t * swc[a];
        // coincident: x = s moves on panel i, y = t; adjacent set 0 likewise, set 1: x = t, y = s
        const bool move_i = coinc || K0 == 0;
        const PMap& mm = move_i ? mi : mj;
        cplx tfix;
        const cplx pfix = pmap_at(move_i ? mj : mi, t, tfix);
        const bool ua = !(fl & (K0 ? PF_DL1_ZERO : PF_DL0_ZERO));
        const bool ub = !(fl & (coinc ? PF_DL1_ZERO : K0 ? PF_DLT1_ZERO : PF_DLT0_ZERO));
        const bool uw = CURVED && !(fl & (K0 ? PF_TDT1_ZERO : PF_TDT0_ZERO));
        cplx S[F][2], L[F][2], B[F][2], Wc[CURVED ? F : 1][2];
#pragma unroll
        for (int q = 0; q < F; ++q) {
            S[q][0] = S[q][1] = L[q][0] = L[q][1] = B[q][0] = B[q][1] = mk(0.);
            if (CURVED) Wc[CURVED ? q : 0][0] = Wc[CURVED ? q : 0][1] = mk(0.);
        }
        for (int z = z0; z < z1; ++z) {
            const double wz = swc[z], s = t * sz[z], ws = wz * s;
            cplx tm;
            const cplx v = pmap_at(mm, s, tm) - pfix;          // minus gamma_i - gamma_j when panel j moves
            const double v2 = norm2(v);
            cplx f, g;
            hk_pair(M.hk, ks2 * v2, f, g);
            const cplx vg = D > 0 ? v2 * g : mk(0.), vf = D > 1 ? v2 * f : mk(0.);
            const cplx kf[3] = {f, vg, vf}, kd[3] = {g, f, vg};
#pragma unroll
            for (int q = 0; q < F; ++q) row_add(S[q], wz, ws, kf[q]);
            if (uw) {
                const double d = tm.im * tfix.im + tm.re * tfix.re;
#pragma unroll
                for (int q = 0; q < F; ++q) row_add(Wc[CURVED ? q : 0], wz * d, ws * d, kf[q]);
            }
            // with v as it is here: L collects v x (fixed or moving tangent of panel j), B the
            // tangent of panel i x v; the sign of v goes into the fold
            if (ua) {
                const cplx tj = move_i ? tfix : tm;
                const double d = v.re * tj.im - v.im * tj.re;
#pragma unroll
                for (int q = 0; q < F; ++q) row_add(L[q], wz * d, ws * d, kd[q]);
            }
            if (ub) {
                const cplx ti = move_i ? tm : tfix;
                const double d = v.im * ti.re - v.re * ti.im;
#pragma unroll
                for (int q = 0; q < F; ++q) row_add(B[q], wz * d, ws * d, kd[q]);
            }
        }
        // the row's two moments into the four of the pair (moments 1, x, y, xy)
        const double sg = move_i ? wt : -wt, tin = sg * mi.tn, tjn = sg * mj.tn;
        auto fold = [&](int set, int q, const cplx (&r)[2], double c, bool s_is_x) {
            cplx* m = A + ((set * F + q) * 4) * 128;
            const cplx r0 = c * r[0], r1 = c * r[1];
            m[0] += r0;
            m[(s_is_x ? 1 : 2) * 128] += r1;
            axpy(m[(s_is_x ? 2 : 1) * 128], t, r0);
            axpy(m[3 * 128], t, r1);
        };
#pragma unroll
        for (int q = 0; q < F; ++q) {
            fold(0, q, S[q], wt, K0 == 0);
            if (coinc) fold(0, q, S[q], wt, false);   // V and W are symmetric in s <-> t: the second triangle
            if (uw) {
                fold(CURVED ? 3 : 0, q, Wc[CURVED ? q : 0], 2. * wt, K0 == 0);
                if (coinc) fold(CURVED ? 3 : 0, q, Wc[CURVED ? q : 0], 2. * wt, false);
            }
            if (ua) fold(1, q, L[q], tin, K0 == 0);
            if (ub) fold(coinc ? 1 : 2, q, B[q], tjn, !coinc && K0 == 0);
        }
    }
    __syncthreads();
    // sum over the threads, each output from another thread on (no two on one bank), in a
    // tree of 16 sums of 8 (one chain of 128 additions showed in W_o - W_i at small k)
    if (threadIdx.x < 2 * R::NA) {
        const int o = threadIdx.x >> 1, c = threadIdx.x & 1;
        const double* src = reinterpret_cast<const double*>(acc + o * 128) + c;
        double s16[16];
#pragma unroll
        for (int h = 0; h < 16; ++h) s16[h] = 0.;
        for (int q = 0; q < 128; q += 16) {
#pragma unroll
            for (int h = 0; h < 16; ++h) s16[h] += src[2 * ((q + h + o) & 127)];
        }
#pragma unroll
        for (int st = 8; st > 0; st >>= 1)
#pragma unroll
            for (int h = 0; h < st; ++h) s16[h] += s16[h + st];
        reinterpret_cast<double*>(mom + o)[c] = s16[0];
    }
    __syncthreads();
}

// whether the node table serves this pair at this wavenumber
__device__ __forceinline__ bool nodes_serve(const DevMesh& M, int ti, const KConst& K) {
    if (!M.snode) return false;
    const double d2 = M.snode[(long long)ti * kSNodeStride + kSN * 32 + 8];
    return K.ks.re * K.ks.re * d2 <= kSNodeX * kSNodeX;
}

__device__ __forceinline__ void load_composite(const DevMesh& M, bool coinc, double* sxc, double* swc, double* sz) {
    for (int t = threadIdx.x; t < M.nc; t += blockDim.x) {
        const double x = M.xc[t];
        sxc[t] = x;
        swc[t] = M.wc[t];
        sz[t] = coinc ? 1. - x : x;
    }
}

// One CTA per (pair, job); q > 0: q CTAs per point set (blocks 2 q t .. of pair t, as in
// k_singular_part), their moments into part for k_singular_rows_join.
template <int D, bool CURVED>
__global__ void __launch_bounds__(128, 2) k_singular_rows(DevMesh M, const SingularTask* tasks, const Job* jobs,
                                                          int q, double* part, cplx* loc, long long npair) {
    typedef RowDims<D, CURVED> R;
    extern __shared__ __align__(16) unsigned char ssm[];
    asm volatile("griddepcontrol.launch_dependents;");   // the general pairs' kernel may fill in behind
    cplx* acc = reinterpret_cast<cplx*>(ssm);
    cplx* mom = acc + R::NA * 128;
    double* sxc = reinterpret_cast<double*>(mom + R::NA);
    double* swc = sxc + M.nc;
    double* sz = swc + M.nc;
    const int job = blockIdx.y;
    const int task = q ? blockIdx.x / (2 * q) : blockIdx.x, sub = q ? blockIdx.x - task * 2 * q : 0;
    const SingularTask T = tasks[task];
    const int nparts = q ? (T.kind == PK_COINC ? q : 2 * q) : 1;
    const KConst K = make_kconst(jobs[job]);
    if (sub >= nparts || nodes_serve(M, task, K)) return;   // whole CTA, before any barrier
    load_composite(M, T.kind == PK_COINC, sxc, swc, sz);
    __syncthreads();
    singular_moments<D, CURVED>(M, T, K, sub, nparts, sxc, swc, sz, acc, mom);
    if (q) {
        cplx* dst = reinterpret_cast<cplx*>(part) + ((long long)job * gridDim.x + blockIdx.x) * R::NA;
        for (int e = threadIdx.x; e < R::NA; e += 128) dst[e] = mom[e];
    } else {
        singular_store<D, CURVED>(M, T, K, mom, threadIdx.x, 128,
                                  loc + ((long long)job * npair + tri_index(T.i, T.j)) * (D + 1) * kLocPerD);
    }
}

// one warp per (pair, job): the parts' moments added in order
template <int D, bool CURVED>
__global__ void __launch_bounds__(128) k_singular_rows_join(DevMesh M, const SingularTask* tasks, const Job* jobs,
                                                            int ntasks, int q, const double* part, cplx* loc,
                                                            long long npair) {
    typedef RowDims<D, CURVED> R;
    __shared__ cplx smom[4][R::NA];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, task = blockIdx.x * 4 + warp, job = blockIdx.y;
    if (task >= ntasks) return;   // whole warp
    const KConst K = make_kconst(jobs[job]);
    if (nodes_serve(M, task, K)) return;
    const SingularTask T = tasks[task];
    const int nparts = T.kind == PK_COINC ? q : 2 * q;
    const cplx* src = reinterpret_cast<const cplx*>(part) + ((long long)job * ntasks + task) * 2 * q * R::NA;
    for (int e = lane; e < R::NA; e += 32) {
        cplx s = mk(0.);
        for (int u = 0; u < nparts; ++u) s += src[(long long)u * R::NA + e];
        smom[warp][e] = s;
    }
    __syncwarp();
    singular_store<D, CURVED>(M, T, K, smom[warp], lane, 32,
                              loc + ((long long)job * npair + tri_index(T.i, T.j)) * (D + 1) * kLocPerD);
}

// ------------------------------------------------------------------ the node table

// a0, b0, a1, b1 at u >= 0 (ascending series below u = 4; beyond, from the Hankel table)
__device__ __forceinline__ void entire_parts(const HkEntry* hk, double u, double& a0, double& b0, double& a1,
                                             double& b1) {
    constexpr double k2pi = 0.63661977236758134308;   // 2 / pi
    if (u <= 4.) {
        const double w = -0.25 * u;
        double t = 1., s0 = 1., h0 = 0., s1 = 1., h1 = 1.;   // h1: sum (H_k + H_(k+1)) t_k / (k + 1)
        for (int k = 1; k <= 14; ++k) {
            t *= w * HBEM_SER_IK2[k];
            s0 += t;
            h0 = fma(HBEM_SER_H[k], t, h0);
            const double t1 = t * HBEM_SER_IK1[k];
            s1 += t1;
            h1 = fma(2. * HBEM_SER_H[k] + HBEM_SER_IK1[k], t1, h1);
        }
        a0 = s0;
        b0 = -k2pi * h0;
        a1 = 0.5 * s1;
        b1 = -0.25 * k2pi * h1;
    } else {
        cplx f, g;
        hk_pair(hk, u, f, g);
        const double lg = k2pi * (0.5 * log(0.25 * u) + kEulerGamma);
        a0 = f.re;
        b0 = fma(-lg, f.re, f.im);
        a1 = g.re;
        b1 = fma(-lg, g.re, g.im) + k2pi / u;
    }
}

// One warp: the pair's moments at job K from its nodes, then its blocks.  vals: shared
// scratch of the warp, mom: NA entries.
template <int D, bool CURVED>
__device__ __forceinline__ void singular_node_pair(const DevMesh& M, const SingularTask& T, int ti, const KConst& K,
                                                   double (*vals)[2][kSN], cplx* mom, cplx* out) {
    typedef RowDims<D, CURVED> R;
    constexpr int F = R::F;
    constexpr double k2pi = 0.63661977236758134308;
    const int lane = threadIdx.x & 31;
    const double* N = M.snode + (long long)ti * kSNodeStride;
    const double d2 = N[kSN * 32 + 8], ks2 = K.ks.re * K.ks.re, iks2 = 1. / ks2;
    if (lane < kSN) {
        const double v2 = d2 * (0.5 + 0.5 * cospi((2 * lane + 1) / (2. * kSN)));
        double a0, b0, a1, b1;
        entire_parts(M.hk, ks2 * v2, a0, b0, a1, b1);
        const double lam = k2pi * (log(0.5 * (K.ks.re * N[kSN * 32 + 9])) + kEulerGamma);
        // real part and k-dependent imaginary part (without the log(|v|/s) term) of f, g, v2 g, v2 f
        const double fi = fma(lam, a0, b0), gi = fma(lam, a1, b1);
        vals[0][0][lane] = a0;
        vals[0][1][lane] = fi;
        vals[1][0][lane] = a1;
        vals[1][1][lane] = gi;                       // its -2/(pi u) enters through sum W / |v|^2
        vals[2][0][lane] = v2 * a1;
        vals[2][1][lane] = fma(v2, gi, -k2pi * iks2);
        vals[3][0][lane] = v2 * a0;
        vals[3][1][lane] = v2 * fi;
    }
    __syncwarp();
    for (int o = lane; o < R::NA; o += 32) {
        const int set = o / (4 * F), q = (o / 4) % F, m = o & 3;
        // S, W take {f, v2 g, v2 f}; L, T take {g, f, v2 g}
        const bool dl = set == 1 || set == 2;
        const int fn = dl ? (q == 0 ? 1 : q == 1 ? 0 : 2) : (q == 0 ? 0 : q == 1 ? 2 : 3);
        const double2* om = reinterpret_cast<const double2*>(N) + set * 4 + m;
        double rs[4] = {0., 0., 0., 0.}, bs[4] = {0., 0., 0., 0.}, ls[4] = {0., 0., 0., 0.};   // short chains of roundings
#pragma unroll
        for (int n = 0; n < kSN; ++n) {
            const double2 w = __ldg(om + n * 16);
            const double al = vals[fn][0][n], be = vals[fn][1][n];
            rs[n & 3] = fma(al, w.x, rs[n & 3]);
            bs[n & 3] = fma(be, w.x, bs[n & 3]);
            ls[n & 3] = fma(al, w.y, ls[n & 3]);
        }
        const double re = (rs[0] + rs[1]) + (rs[2] + rs[3]);
        double im = ((bs[0] + bs[1]) + (bs[2] + bs[3])) + ((ls[0] + ls[1]) + (ls[2] + ls[3]));
        if (dl && q == 0) im = fma(-k2pi * iks2, __ldg(N + kSN * 32 + (set - 1) * 4 + m), im);
        mom[o] = mk(re, im);
    }
    __syncwarp();
    singular_store<D, CURVED>(M, T, K, mom, lane, 32, out);
}

template <int D, bool CURVED>
__global__ void __launch_bounds__(128) k_singular_nodes(DevMesh M, const SingularTask* tasks, int ntasks,
                                                        const Job* jobs, cplx* loc, long long npair) {
    __shared__ double vals[4][4][2][kSN];
    __shared__ cplx mom[4][RowDims<D, CURVED>::NA];
    const int warp = threadIdx.x >> 5, task = blockIdx.x * 4 + warp, job = blockIdx.y;
    if (task >= ntasks) return;   // whole warp
    const KConst K = make_kconst(jobs[job]);
    if (!nodes_serve(M, task, K)) return;
    const SingularTask T = tasks[task];
    singular_node_pair<D, CURVED>(M, T, task, K, vals[warp], mom[warp],
                                  loc + ((long long)job * npair + tri_index(T.i, T.j)) * (D + 1) * kLocPerD);
}

// The sets of moments a pair needs (S always; L, T, W unless their geometric factor
// vanishes at all its points; W on curved panels only): bit set of S = 1, L = 2, T = 4, W = 8
template <class Flags>
__device__ __forceinline__ int snode_sets(const DevMesh& M, const SingularTask& T, Flags fl) {
    int sets = 1;
    if (T.kind == PK_COINC) {
        if ((fl & (PF_DL0_ZERO | PF_DL1_ZERO)) != (PF_DL0_ZERO | PF_DL1_ZERO)) sets |= 2;
        if (!M.lines && !(fl & PF_TDT0_ZERO)) sets |= 8;
    } else {
        if ((fl & (PF_DL0_ZERO | PF_DL1_ZERO)) != (PF_DL0_ZERO | PF_DL1_ZERO)) sets |= 2;
        if ((fl & (PF_DLT0_ZERO | PF_DLT1_ZERO)) != (PF_DLT0_ZERO | PF_DLT1_ZERO)) sets |= 4;
        if (!M.lines && (fl & (PF_TDT0_ZERO | PF_TDT1_ZERO)) != (PF_TDT0_ZERO | PF_TDT1_ZERO)) sets |= 8;
    }
    return sets;
}

// The table's weights.  FP64 bound: per point 110 (lines) to 240 (arcs) instructions of
// geometry and 16 Chebyshev polynomials times the 8 weights (four moments, plain and times
// the logarithm) of each set the pair needs, 128 to 512 multiply-adds.  A CTA takes a
// contiguous part of a pair's points, 128 at a time: first a thread per point (polynomials
// and weights into shared memory), then a thread per polynomial and one weight of each set.
constexpr int kSNodeChunk = 128;
constexpr size_t kSNodeSmem = (size_t)(kSN + 32) * kSNodeChunk * sizeof(double);
constexpr int kSNodePart = kSN * 32 + 8;    // doubles a CTA hands on

template <bool ARCS>
__global__ void __launch_bounds__(128) k_snode_part(DevMesh M, const SingularTask* tasks, int nsplit, double* part) {
    extern __shared__ double nsm[];
    double* Tm = nsm;                          // [polynomial][point]
    double* Wg = nsm + kSN * kSNodeChunk;      // [set][plain 4, log 4][point]
    __shared__ double red[4][8];
    const int task = blockIdx.x / nsplit, sub = blockIdx.x - task * nsplit;
    const SingularTask T = tasks[task];
    const int nc = M.nc, tot = nc * nc, tid = threadIdx.x;
    const bool coinc = T.kind == PK_COINC;
    const uint8_t fl = M.flags[tri_index(T.i, T.j)];
    const int sets = snode_sets(M, T, fl), nsets = __popc(sets);
    PMap mi, mj;
    task_maps(M, T, mi, mj);
    if (!ARCS) mi.line = mj.line = 1;
    const double d2 = task_d2(T, mi, mj), two_id2 = 2. / d2, is = 1. / task_scale(d2), is2 = is * is;
    const long long W = (coinc ? 1LL : 2LL) * tot, c0 = W * sub / nsplit, c1 = W * (sub + 1) / nsplit;
    const int m = tid & 15, slot = tid >> 4;   // the thread's polynomial, and its weight of every set
    double s[4] = {0., 0., 0., 0.}, r[8] = {0., 0., 0., 0., 0., 0., 0., 0.};
    for (long long base = c0; base < c1; base += kSNodeChunk) {
        const int cnt = (int)min((long long)kSNodeChunk, c1 - base);
        __syncthreads();
        double lg = 0., y = 0., wS = 0., wL = 0., wB = 0., wW = 0., px = 0., py = 0.;
        bool ub = false;
        if (tid < cnt) {
            const int w = (int)(base + tid), row = w / nc, K0 = row >= nc ? 1 : 0;
            const double t = M.xc[row - K0 * nc], z = M.xc[w - row * nc], wt = t * M.wc[row - K0 * nc] * M.wc[w - row * nc];
            const bool move_i = coinc || K0 == 0;
            const double q = coinc ? t * (1. - z) : t * z;
            cplx tm, tf;
            const cplx pm = pmap_at(move_i ? mi : mj, q, tm), pf = pmap_at(move_i ? mj : mi, t, tf);
            const cplx v = move_i ? pm - pf : pf - pm;
            const cplx ti = move_i ? tm : tf, tj = move_i ? tf : tm;
            const double v2 = norm2(v);
            if (v2 > 0.) {
                px = move_i ? q : t;
                py = move_i ? t : q;
                lg = 0.31830988618379067154 * log(v2 * is2);   // 2/pi log(|v|/s)
                y = fma(v2, two_id2, -1.);
                const double iv2 = 1. / v2;
                wS = wt;
                if (!(fl & (K0 ? PF_DL1_ZERO : PF_DL0_ZERO))) wL = wt * mi.tn * (v.re * tj.im - v.im * tj.re);
                ub = !(fl & (coinc ? PF_DL1_ZERO : K0 ? PF_DLT1_ZERO : PF_DLT0_ZERO));
                if (ub) wB = wt * mj.tn * (v.im * ti.re - v.re * ti.im);
                if (sets & 8)
                    if (!(fl & (K0 ? PF_TDT1_ZERO : PF_TDT0_ZERO))) wW = 2. * wt * (ti.im * tj.im + ti.re * tj.re);
                if (sets & 2) {
                    const double a = wL * iv2, b = coinc ? wB * iv2 : 0.;
                    r[0] += a + b;
                    r[1] += fma(a, px, b * py);
                    r[2] += fma(a, py, b * px);
                    r[3] += (a + b) * (px * py);
                }
                if (sets & 4) {
                    const double b = wB * iv2;
                    r[4] += b;
                    r[5] = fma(b, px, r[5]);
                    r[6] = fma(b, py, r[6]);
                    r[7] = fma(b, px * py, r[7]);
                }
            }
        }
        double p0 = 1., p1 = y;
        Tm[tid] = p0;
        Tm[kSNodeChunk + tid] = p1;
        for (int q = 2; q < kSN; ++q) {
            const double p2 = fma(2. * y, p1, -p0);
            Tm[q * kSNodeChunk + tid] = p2;
            p0 = p1;
            p1 = p2;
        }
        // weights of the four moments 1, x, y, xy; coincident pairs add the second triangle (x and y exchanged)
        auto put = [&](int row, double a, double b) {
            const double xy = px * py, w4[4] = {a + b, fma(a, px, b * py), fma(a, py, b * px), (a + b) * xy};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                Wg[(8 * row + e) * kSNodeChunk + tid] = w4[e];
                Wg[(8 * row + 4 + e) * kSNodeChunk + tid] = lg * w4[e];
            }
        };
        int row = 0;
        put(row++, wS, coinc ? wS : 0.);
        if (sets & 2) put(row++, wL, coinc ? wB : 0.);
        if (sets & 4) put(row++, wB, 0.);
        if (sets & 8) put(row++, wW, coinc ? wW : 0.);
        __syncthreads();
        const double* tp = Tm + m * kSNodeChunk;
        const double* wp = Wg + slot * kSNodeChunk;
        double sc[4] = {0., 0., 0., 0.};   // summed by chunks: shorter chains of roundings
        // the threads start at different points: no two on one bank
#pragma unroll 4
        for (int q = 0; q < kSNodeChunk; ++q) {
            const int c = (q + tid) & (kSNodeChunk - 1);
            const double t = tp[c];
            sc[0] = fma(t, wp[c], sc[0]);
            if (nsets > 1) sc[1] = fma(t, wp[8 * kSNodeChunk + c], sc[1]);
            if (nsets > 2) sc[2] = fma(t, wp[16 * kSNodeChunk + c], sc[2]);
            if (nsets > 3) sc[3] = fma(t, wp[24 * kSNodeChunk + c], sc[3]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] += sc[e];
    }
    double* dst = part + (long long)blockIdx.x * kSNodePart;
    int row = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {   // [polynomial][plain, log][set][moment]
        const bool on = (sets >> e) & 1;
        double x = 0.;
        if (on) {
            x = row == 0 ? s[0] : row == 1 ? s[1] : row == 2 ? s[2] : s[3];
            ++row;
        }
        dst[m * 32 + (slot >> 2) * 16 + 4 * e + (slot & 3)] = x;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        double x = r[e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if ((tid & 31) == 0) red[tid >> 5][e] = x;
    }
    __syncthreads();
    if (tid < 8) dst[kSN * 32 + tid] = red[0][tid] + red[1][tid] + red[2][tid] + red[3][tid];
}

// moments against the Chebyshev polynomials -> weights at the nodes
__global__ void __launch_bounds__(128) k_snode_join(DevMesh M, const SingularTask* tasks, int nsplit,
                                                    const double* part, double* nodes) {
    __shared__ double S[kSNodePart];
    const int task = blockIdx.x;
    for (int e = threadIdx.x; e < kSNodePart; e += blockDim.x) {
        double x = 0.;
        for (int u = 0; u < nsplit; ++u) x += part[((long long)task * nsplit + u) * kSNodePart + e];
        S[e] = x;
    }
    __syncthreads();
    double* dst = nodes + (long long)task * kSNodeStride;
    for (int e = threadIdx.x; e < kSN * 32; e += blockDim.x) {
        const int q = e >> 5, w = e & 31;
        double x = 0.;
        for (int m = kSN - 1; m > 0; --m) x = fma(cospi((2 * q + 1) * m / (2. * kSN)), S[m * 32 + w], x);
        dst[(q * 16 + (w & 15)) * 2 + (w >> 4)] = (S[w] + 2. * x) / kSN;
    }
    if (threadIdx.x < 8) dst[kSN * 32 + threadIdx.x] = S[kSN * 32 + threadIdx.x];
    if (threadIdx.x == 0) {
        const SingularTask T = tasks[task];
        PMap mi, mj;
        task_maps(M, T, mi, mj);
        const double d2 = task_d2(T, mi, mj);
        dst[kSN * 32 + 8] = d2;
        dst[kSN * 32 + 9] = task_scale(d2);
    }
}

}  // namespace hbem
