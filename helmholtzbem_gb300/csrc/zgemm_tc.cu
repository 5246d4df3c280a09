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
// B' = [[B_r, B_i], [-B_i, B_r]] (64 x 64 for 32 complex columns), C' = [re | im].
// A CTA takes 128 rows and a run of 32-column tiles: A's digits are cut once (112 KB of
// 128-byte-swizzled K-major shared memory), B's per tile (56 KB).  Tensor memory: the eight
// sums, 64 columns each, all 512.  Per tile 34 digit products of four K = 16 steps; the FP64
// pipe does two instructions per real entry (a conversion and an FMA) instead of 128.
#include <algorithm>
#include <cstdint>

#include "hbem_device.cuh"

namespace hbem {

namespace {

constexpr int kZM = 128;                   // rows per CTA
constexpr int kZNc = 32;                   // complex columns per tile
constexpr int kZN = 2 * kZNc;              // MMA N
constexpr int kZK = 32;                    // complex depth
constexpr int kZDig = 7, kZSums = 8;
constexpr int kZThreads = 256;
constexpr uint32_t kZABytes = kZM * 128u, kZBBytes = kZN * 128u;   // a digit of each operand: rows of 64 BF16
constexpr size_t kZSmem = kZDig * (size_t)(kZABytes + kZBBytes) + 1024;
constexpr long long kZSpinCap = 1LL << 24;
// instruction descriptor, kind::f16: D FP32, A and B BF16, K-major, N >> 3, M >> 4
constexpr uint32_t kZIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kZN >> 3) << 17) |
                             ((uint32_t)(kZM >> 4) << 24);

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

__global__ void __launch_bounds__(kZThreads, 1) k_zgemm_tc(ZJob J) {
    extern __shared__ uint8_t z_raw[];
    uint8_t* As = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(z_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* Bs = As + kZDig * kZABytes;
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail, s_ea[2][kZM], s_eb[kZNc];
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
        s_fail = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(z_smem(&mbar)), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
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
    const uint32_t mbar_addr = z_smem(&mbar);
    const int tile0 = blockIdx.y * J.tiles, ntiles = (J.n + kZNc - 1) / kZNc, tile1 = min(ntiles, tile0 + J.tiles);
    for (int t = tile0; t < tile1; ++t) {
        const int c0 = t * kZNc;
        {   // B: thread (column tid >> 3, four depths); columns j (re) and 32 + j (im) of C' take
            // [B_r | -B_i] and [B_i | B_r]
            const int j = tid >> 3, k0 = (tid & 7) * 4;
            cplx b[4];
            int E = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                b[q] = (c0 + j < J.n && k0 + q < J.k) ? B[(k0 + q) + (long long)(c0 + j) * J.ldb] : mk(0.);
                E = max(E, max(z_exp(b[q].re), z_exp(b[q].im)));
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) E = max(E, __shfl_xor_sync(0xffffffffu, E, o));
            if ((tid & 7) == 0) s_eb[j] = E;
            long long vr[4], vi[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                vr[q] = z_fixed(b[q].re, E);
                vi[q] = z_fixed(b[q].im, E);
            }
            const int ch = k0 >> 3, sub = (k0 & 4) << 1;          // chunk and byte of its half
            const uint32_t o00 = z_chunk(j, ch) + sub, o01 = z_chunk(j, 4 + ch) + sub;
            const uint32_t o10 = z_chunk(kZNc + j, ch) + sub, o11 = z_chunk(kZNc + j, 4 + ch) + sub;
#pragma unroll
            for (int dgt = kZDig - 1; dgt >= 0; --dgt) {
                int dr[4], di[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    dr[q] = dgt ? z_digit(vr[q]) : (int)vr[q];
                    di[q] = dgt ? z_digit(vi[q]) : (int)vi[q];
                }
                uint8_t* S = Bs + dgt * kZBBytes;
                const uint2 re = make_uint2(z_pack(dr[0], dr[1]), z_pack(dr[2], dr[3]));
                const uint2 im = make_uint2(z_pack(di[0], di[1]), z_pack(di[2], di[3]));
                const uint2 ng = make_uint2(z_pack(-di[0], -di[1]), z_pack(-di[2], -di[3]));
                *reinterpret_cast<uint2*>(S + o00) = re;
                *reinterpret_cast<uint2*>(S + o01) = ng;
                *reinterpret_cast<uint2*>(S + o10) = im;
                *reinterpret_cast<uint2*>(S + o11) = re;
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tensor core reads what was written
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem_slot;
        if (tid == 0) {
            for (int s = 0; s < kZSums; ++s) {
                uint32_t acc = 0u;
                for (int a = max(0, s - kZDig + 1); a <= min(s, kZDig - 1); ++a)
                    for (int kk = 0; kk < 4; ++kk) {
                        const uint64_t ad = z_desc(z_smem(As) + a * kZABytes + kk * 32u);
                        const uint64_t bd = z_desc(z_smem(Bs) + (s - a) * kZBBytes + kk * 32u);
                        asm volatile(
                            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(taddr + s * kZN),
                            "l"(ad), "l"(bd), "r"(kZIdesc), "r"(acc));
                        acc = 1u;
                    }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar_addr)
                         : "memory");
        }
        // the entries to update, while the products run
        const int row = r0 + (warp & 3) * 32 + lane, half = warp >> 2;
        if (!z_wait(mbar_addr, (uint32_t)((t - tile0) & 1))) s_fail = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const bool bad = __syncthreads_or(s_fail);
        const int Er = max(s_ea[0][(warp & 3) * 32 + lane], s_ea[1][(warp & 3) * 32 + lane]);
        const uint32_t lane_base = taddr + ((uint32_t)((warp & 3) * 32) << 16);
        for (int j0 = half * 16; j0 < half * 16 + 16; j0 += 4) {
            uint32_t re[kZSums][4], im[kZSums][4];
            if (!bad) {
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
                    // sums 0..3 and 4..7 as integers of weight 2^32 and 1, together in units of 2^16
                    auto join = [&](const uint32_t (&d)[kZSums][4]) {
                        long long hi = 0, lo = 0;
#pragma unroll
                        for (int s = 0; s < 4; ++s) {
                            hi = (hi << 8) + (long long)__float2int_rn(__uint_as_float(d[s][jj]));
                            lo = (lo << 8) + (long long)__float2int_rn(__uint_as_float(d[4 + s][jj]));
                        }
                        return (hi << 16) + ((lo + 0x8000) >> 16);
                    };
                    const double sc = bad ? CUDART_NAN : z_scale(Er, s_eb[j0 + jj]);   // a wait that ran out shows
                    cplx* p = C + row + (long long)col * J.ldc;
                    const cplx c = *p;
                    *p = mk(fma(-sc, (double)join(re), c.re), fma(-sc, (double)join(im), c.im));
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();   // B's digits, the sums and s_eb are free
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (bad) {   // another bounded chance for the products before the memory is given back
            z_wait(mbar_addr, (uint32_t)((t - tile0) & 1));
            break;
        }
    }
    __syncthreads();
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
