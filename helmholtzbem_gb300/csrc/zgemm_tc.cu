// Batched complex128 update C -= A B on the 5th-generation tensor cores: the trailing
// update of the complex128 LU (csrc/lu.cu), depth at most 32.
//
// Why: GB300 has two FP64 lanes per SM and cycle, so the FP64 FMA form of this update was 33 of
// the 45 ms of the LU of four matrices of order 1500 and could not be faster; the tensor
// cores have no FP64 of use here either.  Instead the operands become integers and their
// products exact BF16 ones (the scheme of Ootomo, Ozaki and Yokota for integer units, here
// with BF16 digits and FP32 accumulation):
//   * a row of A (a column of B) is scaled by the power of two above its largest entry and
//     rounded to 56-bit integers X (error 2^-56 of the largest entry, where an FP64 entry
//     itself has 2^-53 of its own size), cut into seven balanced base-256 digits, each of at
//     most 128 in size and so exact in BF16;
//   * digits a of A and b of B are multiplied for a + b = s <= 7, the products of one s summed
//     in one FP32 accumulator: at most 7 x 64 terms of at most 2^14, below 2^23, hence exact in
//     any order; what is left out (s >= 8) is below 2^-60 of row times column maximum;
//   * the eight sums of an entry make one 64-bit integer (error 2^-54 of row times column
//     maximum), converted and subtracted from C in FP64: one rounding for the whole depth,
//     where 64 FMAs round 64 times.
// Measured against 64-bit products of random and of LU operands the error is below the FMA
// kernel's (tests/test_gpu_zgemm.py).
//
// Complex product as one real GEMM, as in tc_gemm.cu: A' = [A_r | A_i] (128 x 64),
// B' = [[B_r, B_i], [-B_i, B_r]] (64 x 32 for 16 complex columns), C' = [re | im].
// A CTA takes 128 rows and a run of 16-column tiles: A's digits are cut once (112 KB of
// 128-byte-swizzled K-major shared memory), B's per tile (28 KB, two buffers).  Tensor memory:
// the eight sums of a tile are 256 columns, so two tiles fit, and a tile's products run while
// the sums of the one before are read, joined and subtracted.  That epilogue is what bounds the
// kernel: per real entry eight 32-bit conversions and two FP64 instructions (a conversion and an
// FMA) instead of 128.  The first update of four matrices of order 1500 takes 196 us; with
// tiles of 32 columns in one buffer, C read in the epilogue and a product per digit pair, 362.
#include <algorithm>
#include <cstdint>

#include "hbem_device.cuh"

namespace hbem {

namespace {

constexpr int kZM = 128;                   // rows per CTA
constexpr int kZNc = 16;                   // complex columns per tile
constexpr int kZN = 2 * kZNc;              // MMA N
constexpr int kZK = 32;                    // complex depth
constexpr int kZDig = 7, kZSums = 8;
constexpr int kZThreads = 256;
constexpr uint32_t kZABytes = kZM * 128u, kZBBytes = kZN * 128u;   // a digit of each operand: rows of 64 BF16
constexpr size_t kZSmem = kZDig * (size_t)(kZABytes + 2 * kZBBytes) + 1024;
constexpr long long kZSpinCap = 1LL << 24;
// instruction descriptor, kind::f16: D FP32, A and B BF16, K-major, N >> 3, M >> 4
__device__ constexpr uint32_t z_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kZM >> 4) << 24);
}

__device__ __forceinline__ uint32_t z_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 128-byte swizzle, K-major: 16-byte chunk q (8 BF16) of row r
__device__ __forceinline__ uint32_t z_chunk(int r, int q) {
    return (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u + ((uint32_t)(q ^ (r & 7)) << 4);
}

__device__ __forceinline__ uint64_t z_desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1u << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1u << 46;
    d |= (uint64_t)2u << 61;
    return d;
}

// biased exponent (zero and subnormals: 0)
__device__ __forceinline__ int z_exp(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// x as an integer in units of 2^-55 of the power of two above the row's (column's) largest
// entry, E its biased exponent: |result| <= 2^55
__device__ __forceinline__ long long z_fixed(double x, int E) {
    const long long b = __double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ff), d = min(60, E - e);
    long long v = ((b & 0xfffffffffffffll) | 0x10000000000000ll) << 2;
    v = e ? (v + ((1ll << d) >> 1)) >> d : 0;
    return b < 0 ? -v : v;
}

// takes the lowest balanced base-256 digit off v
__device__ __forceinline__ int z_digit(long long& v) {
    const int d = (int)(signed char)(v & 0xff);
    v = (v - d) >> 8;
    return d;
}

// two small integers as BF16 (exact up to 256), the first in the low half
__device__ __forceinline__ uint32_t z_pack(int a, int b) {
    const float fa = __int_as_float(0x4B400000 + a) - 12582912.f, fb = __int_as_float(0x4B400000 + b) - 12582912.f;
    return __byte_perm(__float_as_uint(fa), __float_as_uint(fb), 0x7632);
}

// 2^(E + F - 1022 - 1022 - 54) for the largest entries' biased exponents; NaN where either is Inf or NaN
__device__ __forceinline__ double z_scale(int E, int F) {
    if (E == 0x7ff || F == 0x7ff) return CUDART_NAN;
    const int e = E + F - 1022 - 1022 - 54 + 1023;
    if (E == 0 || F == 0 || e < 1) return 0.;
    if (e > 2046) return CUDART_INF;
    return __hiloint2double(e << 20, 0);
}

struct ZJob {
    int m, n, k, tiles;           // tiles: 32-column tiles per CTA
    const cplx* A;
    const cplx* B;
    cplx* C;
    long long lda, ldb, ldc, sa, sb, sc;
};

__device__ __forceinline__ bool z_wait(uint32_t mbar, uint32_t parity) {
    uint32_t done = 0;
    for (long long it = 0; it < kZSpinCap && !done; ++it)
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
    return done != 0;
}

__device__ __forceinline__ void z_ld4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

// the sums (exact integers in FP32) of one real entry as one integer in units of 2^16 of the last
// sum's: neighbours fit 32 bits (sum s has at most s + 1 digit pairs of 64 x 2^14)
__device__ __forceinline__ int z_int(float f, bool small) {   // small: |f| <= 2^22
    return small ? __float_as_int(f + 12582912.f) - 0x4B400000 : __float2int_rn(f);
}
__device__ __forceinline__ long long z_join(const uint32_t (&d)[kZSums][4], int jj) {
    int p[4];
#pragma unroll
    for (int s = 0; s < 4; ++s)
        p[s] = z_int(__uint_as_float(d[2 * s][jj]), 2 * s < 3) * 256 + z_int(__uint_as_float(d[2 * s + 1][jj]), 2 * s + 1 < 3);
    const long long hi = (long long)p[0] * 65536 + p[1], lo = (long long)p[2] * 65536 + p[3];
    return hi * 65536 + ((lo + 0x8000) >> 16);
}

__global__ void __launch_bounds__(kZThreads, 1) k_zgemm_tc(ZJob J) {
    extern __shared__ uint8_t z_raw[];
    uint8_t* As = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(z_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* Bs = As + kZDig * kZABytes;
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_ea[2][kZM], s_eb[3][kZNc];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r0 = blockIdx.x * kZM;
    const cplx* A = J.A + (long long)blockIdx.z * J.sa;
    const cplx* B = J.B + (long long)blockIdx.z * J.sb;
    cplx* C = J.C + (long long)blockIdx.z * J.sc;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(z_smem(&tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(z_smem(&mbar[0])), "r"(1));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(z_smem(&mbar[1])), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const int tile0 = blockIdx.y * J.tiles, ntiles = (J.n + kZNc - 1) / kZNc, tile1 = min(ntiles, tile0 + J.tiles);
    // B of the next tile and the entries of C that a tile updates are read ahead, into registers:
    // one CTA fits an SM, so nothing else covers their latency
    cplx b[2];   // thread (column tid >> 4, two depths)
    auto load_b = [&](int t) {
        const int col = t * kZNc + (tid >> 4), k0 = (tid & 15) * 2;
#pragma unroll
        for (int q = 0; q < 2; ++q)
            b[q] = (t < tile1 && col < J.n && k0 + q < J.k) ? B[(k0 + q) + (long long)col * J.ldb] : mk(0.);
    };
    load_b(tile0);
    {   // A: thread (row tid & 127, half of the depth)
        const int r = tid & 127, kh = tid >> 7;
        cplx a[16];
        int E = 0;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int k = 16 * kh + q;
            a[q] = (r0 + r < J.m && k < J.k) ? A[(r0 + r) + (long long)k * J.lda] : mk(0.);
            E = max(E, max(z_exp(a[q].re), z_exp(a[q].im)));
        }
        s_ea[kh][r] = E;
        __syncthreads();
        E = max(s_ea[0][r], s_ea[1][r]);
#pragma unroll
        for (int part = 0; part < 2; ++part)
#pragma unroll
            for (int h = 0; h < 2; ++h) {      // 8 depths: a 16-byte chunk
                long long v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = z_fixed(part ? a[8 * h + q].im : a[8 * h + q].re, E);
                const uint32_t off = z_chunk(r, part * 4 + kh * 2 + h);
#pragma unroll
                for (int dgt = kZDig - 1; dgt >= 0; --dgt) {   // digit 0 is the leading one
                    int d[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) d[q] = dgt ? z_digit(v[q]) : (int)v[q];
                    *reinterpret_cast<uint4*>(As + dgt * kZABytes + off) =
                        make_uint4(z_pack(d[0], d[1]), z_pack(d[2], d[3]), z_pack(d[4], d[5]), z_pack(d[6], d[7]));
                }
            }
    }
    // the loaded tile's digits into buffer u, its columns' exponents into s_eb[e]: columns j (re) and 16 + j (im) of C' take [B_r | -B_i]
    // and [B_i | B_r]
    auto cut_b = [&](int u, int e) {
        const int j = tid >> 4, k0 = (tid & 15) * 2;
        int E = 0;
#pragma unroll
        for (int q = 0; q < 2; ++q) E = max(E, max(z_exp(b[q].re), z_exp(b[q].im)));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) E = max(E, __shfl_xor_sync(0xffffffffu, E, o));
        if ((tid & 15) == 0) s_eb[e][j] = E;
        long long vr[2], vi[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            vr[q] = z_fixed(b[q].re, E);
            vi[q] = z_fixed(b[q].im, E);
        }
        const int ch = k0 >> 3, sub = (k0 & 7) * 2;               // chunk and byte within it
        const uint32_t o00 = z_chunk(j, ch) + sub, o01 = z_chunk(j, 4 + ch) + sub;
        const uint32_t o10 = z_chunk(kZNc + j, ch) + sub, o11 = z_chunk(kZNc + j, 4 + ch) + sub;
#pragma unroll
        for (int dgt = kZDig - 1; dgt >= 0; --dgt) {
            int dr[2], di[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                dr[q] = dgt ? z_digit(vr[q]) : (int)vr[q];
                di[q] = dgt ? z_digit(vi[q]) : (int)vi[q];
            }
            uint8_t* S = Bs + (u * kZDig + dgt) * kZBBytes;
            const uint32_t re = z_pack(dr[0], dr[1]);
            *reinterpret_cast<uint32_t*>(S + o00) = re;
            *reinterpret_cast<uint32_t*>(S + o01) = z_pack(-di[0], -di[1]);
            *reinterpret_cast<uint32_t*>(S + o10) = z_pack(di[0], di[1]);
            *reinterpret_cast<uint32_t*>(S + o11) = re;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tensor core reads what was written
    };
    // one thread: the digit products of buffer u into its half of the tensor memory.  Digit a of A
    // times digits 0 .. of B is one product: B's digits lie one behind the other, 32 rows each, and
    // so do the sums a + b.  29 products of up to 224 columns, where digit by digit 136 products of
    // 32 columns took 75 ns each whatever their width.
    auto products = [&](int u) {
        const uint32_t taddr = tmem_slot + u * kZSums * kZN;
        const uint64_t ad = z_desc(z_smem(As)), bd = z_desc(z_smem(Bs) + u * kZDig * kZBBytes);
        auto mma = [&](int a, int b0, int nb, int kk, uint32_t acc) {
            asm volatile(
                "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(taddr + (a + b0) * kZN),
                "l"(ad + (a * kZABytes + kk * 32) / 16), "l"(bd + (b0 * kZBBytes + kk * 32) / 16),
                "r"(z_idesc(nb * kZN)), "r"(acc));
        };
#pragma unroll
        for (int a = 0; a < kZDig; ++a) {
            const int nb = min(kZDig, kZSums - a);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                if (a == 1 && kk == 0) {   // the last sum begins here
                    mma(a, nb - 1, 1, kk, 0u);
                    mma(a, 0, nb - 1, kk, 1u);
                } else
                    mma(a, 0, nb, kk, a > 0 || kk > 0 ? 1u : 0u);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(z_smem(&mbar[u]))
                     : "memory");
    };
    const int ra = (warp & 3) * 32 + lane, row = r0 + ra, half = warp >> 2;   // half: which 8 columns of a tile
    bool fail = false;   // a wait ran out (warp-uniform)
    cut_b(0, 0);
    load_b(tile0 + 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0 && tile0 < tile1) products(0);
    for (int t = tile0; t < tile1; ++t) {
        const int u = (t - tile0) & 1, c0 = t * kZNc;
        cplx cc[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int col = c0 + half * 8 + q;
            cc[q] = row < J.m && col < J.n ? C[row + (long long)col * J.ldc] : mk(0.);
        }
        // the next tile's digits go where those of the tile before this one were, whose products
        // this thread has waited for; its exponents do not, slower warps may still read them (three
        // rounds: the barrier below has every warp past the tile before that one)
        if (t + 1 < tile1) cut_b(u ^ 1, (t + 1 - tile0) % 3);
        load_b(t + 2);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (__syncthreads_or(fail)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (tid == 0 && t + 1 < tile1) products(u ^ 1);
        __syncwarp();
        fail = __any_sync(0xffffffffu, !z_wait(z_smem(&mbar[u]), (uint32_t)(((t - tile0) >> 1) & 1)));
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int Er = max(s_ea[0][ra], s_ea[1][ra]);
        const uint32_t lane_base = tmem_slot + u * kZSums * kZN + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
        for (int jq = 0; jq < 2; ++jq) {
            const int j0 = half * 8 + 4 * jq;
            uint32_t re[kZSums][4], im[kZSums][4];
            if (!fail) {
#pragma unroll
                for (int s = 0; s < kZSums; ++s) {
                    z_ld4(lane_base + s * kZN + j0, re[s]);
                    z_ld4(lane_base + s * kZN + kZNc + j0, im[s]);
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            }
            if (row < J.m) {
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const int col = c0 + j0 + jj;
                    if (col >= J.n) continue;
                    const double sc = fail ? CUDART_NAN : z_scale(Er, s_eb[(t - tile0) % 3][j0 + jj]);   // a wait that ran out shows
                    const cplx c = cc[4 * jq + jj];
                    C[row + (long long)col * J.ldc] =
                        mk(fma(-sc, (double)z_join(re, jj), c.re), fma(-sc, (double)z_join(im, jj), c.im));
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (__syncthreads_or(fail)) {   // another bounded chance for the products before the memory is given back
        for (int u = 0; u < 2; ++u)
            for (uint32_t par = 0; par < 2; ++par) z_wait(z_smem(&mbar[u]), par);
        __syncthreads();
    }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot), "r"(512u));
}

}  // namespace

// C_b -= A_b B_b for nmat matrices: m x n, depth k <= 32, column-major
cudaError_t launch_zgemm_tc(int m, int n, int k, const cplx* A, long long lda, long long sa, const cplx* B, long long ldb,
                            long long sb, cplx* C, long long ldc, long long sc, int nmat, cudaStream_t st) {
    if (m <= 0 || n <= 0 || k <= 0) return cudaSuccess;
    if (k > kZK || nmat < 1 || nmat > 65535) return cudaErrorInvalidValue;
    if (cudaError_t e = cudaFuncSetAttribute(k_zgemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kZSmem);
        e != cudaSuccess)
        return e;
    const int rt = (m + kZM - 1) / kZM, ct = (n + kZNc - 1) / kZNc;
    // tiles per CTA: one CTA per SM at a time, so as many as spread all the tiles over the 152
    const long long total = (long long)rt * ct * nmat;
    const int tiles = (int)std::max<long long>(1, std::min<long long>(ct, (total + 151) / 152));
    ZJob J{m, n, k, tiles, A, B, C, lda, ldb, ldc, sa, sb, sc};
    const dim3 grid(rt, (ct + tiles - 1) / tiles, nmat);
    k_zgemm_tc<<<grid, kZThreads, kZSmem, st>>>(J);
    return cudaGetLastError();
}

}  // namespace hbem
