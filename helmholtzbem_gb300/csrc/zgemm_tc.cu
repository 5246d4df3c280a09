// Batched complex128 update C -= A B on the 5th-generation tensor cores: the trailing
// update of the complex128 LU (csrc/lu.cu), depth at most 32.
//
// Why: GB300 has two FP64 lanes per SM and cycle, so the FP64 FMA form of this update was 33 of
// the 45 ms of the LU of four matrices of order 1500 and could not be faster; the tensor
// cores have no FP64 of use here either.  Instead the operands become integers and their
// products exact BF16 ones (the scheme of Ootomo, Ozaki and Yokota for integer units, here
// with BF16 digits and FP32 accumulation):
//   * where B's rows differ in size by 2^5 or more, column k of A is multiplied and row k of B divided
//     by the power of two of that row's largest entry over all columns (integer additions on
//     exponents): with rows of different size, partial pivoting leaves A growing and B falling along
//     the depth, and the large entries of the one then meet the small ones of the other (random
//     matrices' rows differ by up to 2^2, those of T(k), orders 192 to 800, mostly by 2^1 to 2^4);
//   * a row of A (a column of B) so scaled is rounded to 56-bit integers X in units of the power
//     of two above its largest entry (error 2^-56 of that entry, where an FP64 entry itself has
//     2^-53 of its own size), cut into seven balanced base-256 digits, each of at most 128 in
//     size and so exact in BF16;
//   * digits a of A and b of B are multiplied for a + b = s <= 7, the products of one s summed
//     in one FP32 accumulator: at most 7 x 64 terms of at most 2^14, below 2^23, hence exact in
//     any order; what is left out (s >= 8) is below 2^-60 of row times column maximum;
//   * the eight sums of an entry make one 64-bit integer (error 2^-54 of row times column
//     maximum), converted and subtracted from C in FP64: one rounding for the whole depth,
//     where 64 FMAs round 64 times.
// The error is relative to (row maximum x column maximum), an FMA's to the terms themselves, so
// the first must not exceed the second by much.  Every row and column carries masks of the depths
// at which it is within 0, 3, 6 and 9 powers of two of its maximum; an entry for which no depth has
// the two distances adding up to 9 is formed by FMAs from A and B instead (z_direct).  So an
// entry's error stays below 2^-38 of its sum |a||b| at worst, whatever the matrix's scaling; over the
// rows of random, graded and T(k) operands it is the FMA kernel's (0.9 to 2.2 times).  Of the
// entries of T(k), orders 300 to 800, at most 2e-4 go the direct way, in 2e-3 of the warps (masks
// of 0 and 6 or less alone: up to 3e-2), of random operands none.
//
// Complex product as one real GEMM, as in tc_gemm.cu: A' = [A_r | A_i] (128 x 64),
// B' = [[B_r, B_i], [-B_i, B_r]] (64 x 32 for 16 complex columns), C' = [re | im].
// A CTA takes 128 rows and a run of 16-column tiles: A's digits are cut once (112 KB of
// 128-byte-swizzled K-major shared memory), B's per tile (28 KB, two buffers).  Tensor memory:
// the eight sums of a tile are 256 columns, so two tiles fit, and a tile's products run while
// the sums of the one before are read, joined and subtracted: per real entry eight 32-bit
// conversions and two FP64 instructions (a conversion and an FMA) instead of 128.  What bounds the
// kernel is that work and the cutting of the next digits, dependent instructions of eight warps (FP64
// pipe 39 % active, tensor pipe 22 %, issue slots 30 %).  The first update of four matrices of order 1500 takes 174 us (with
// the masks of every column loaded and tested by every thread 189, by warp reductions of half
// warps 215; without masks 171); with tiles of 32 columns in one buffer, C read in the epilogue and
// a product per digit pair, 362.
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
constexpr int kZSpinCap = 1 << 18;         // tries, each suspended for a while: about a second; a tile's products take microseconds
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

// Exponents here are biased ones plus a depth's shift s, as plain integers; of zeros kZNone, of
// Inf and NaN kZBad.  Subnormals have the exponent of the smallest normal number.
constexpr int kZNone = -(1 << 20), kZBad = 1 << 20;
constexpr int kZNear = 3, kZLevels = 4;   // the masks' step and number
constexpr int kZEven = 5;                 // rows of B within fewer powers of two are not scaled

__device__ __forceinline__ int z_exp(cplx z, int s) {
    const int m = max(__double2hiint(z.re) & 0x7fffffff, __double2hiint(z.im) & 0x7fffffff), e = m >> 20;
    return (m | __double2loint(z.re) | __double2loint(z.im)) == 0 ? kZNone : e == 0x7ff ? kZBad : max(e, 1) + s;
}

// The shifts of the depths, lane k that of depth k; a whole warp.  ek: the biased exponents of the
// largest entries of B's k rows (0: nothing known).
__device__ __forceinline__ int z_shift(const int* ek, int k) {
    const int lane = threadIdx.x & 31, e = lane < k ? ek[lane] : 0;
    const bool in = e > 0 && e < 0x7ff;
    const int hi = __reduce_max_sync(0xffffffffu, in ? e : 0), lo = __reduce_min_sync(0xffffffffu, in ? e : 0x7ff);
    return in && hi - lo >= kZEven ? e - 1023 : 0;
}

// x times 2^s as an integer in units of 2^-55 of the power of two above the row's (column's)
// largest entry, E its exponent: |result| <= 2^55
__device__ __forceinline__ long long z_fixed(double x, int s, int E) {
    const long long b = __double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ff), d = max(0, min(60, E - max(e, 1) - s));
    long long v = ((b & 0xfffffffffffffll) | (e ? 0x10000000000000ll : 0)) << 2;
    v = (v + ((1ll << d) >> 1)) >> d;
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

struct ZJob {
    int m, n, k, tiles;           // tiles: tiles of kZNc columns per CTA
    const cplx* A;
    const cplx* B;
    cplx* C;
    long long lda, ldb, ldc, sa, sb, sc;
    const int* ek;                // per matrix k exponents of B's rows (z_shift)
    long long se;
    int* info;                    // per matrix: -1 where a wait ran out
};

// An entry of C by FMAs from its row of A and column of B, as k_lu_gemm forms it
__device__ __forceinline__ cplx z_direct(const cplx* a, long long lda, const cplx* b, int k, cplx c) {
#pragma unroll 1
    for (int q = 0; q < k; ++q) cfms(c, a[q * lda], b[q]);
    return c;
}

__device__ __forceinline__ bool z_wait(uint32_t mbar, uint32_t parity) {
    uint32_t done = 0;
    for (int it = 0; it < kZSpinCap && !done; ++it)
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
    // depths near the maximum, a bit each (all: nothing but zeros): bit k / 2 for an even depth k, 16 + k / 2 for an odd one
    __shared__ uint4 s_ma[2][kZM], s_mb[3][kZNc];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r0 = blockIdx.x * kZM;
    const cplx* A = J.A + (long long)blockIdx.z * J.sa;
    const cplx* B = J.B + (long long)blockIdx.z * J.sb;
    cplx* C = J.C + (long long)blockIdx.z * J.sc;
    const int shift = z_shift(J.ek + (long long)blockIdx.z * J.se, J.k);
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
    int bs[2];   // and the shifts of those
#pragma unroll
    for (int q = 0; q < 2; ++q) bs[q] = -__shfl_sync(0xffffffffu, shift, (tid & 15) * 2 + q);
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
        int as[16], E = kZNone;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int k = 16 * kh + q;
            a[q] = (r0 + r < J.m && k < J.k) ? A[(r0 + r) + (long long)k * J.lda] : mk(0.);
            as[q] = __shfl_sync(0xffffffffu, shift, k);
            E = max(E, z_exp(a[q], as[q]));
        }
        s_ea[kh][r] = E;
        __syncthreads();
        E = max(s_ea[0][r], s_ea[1][r]);
        unsigned near[kZLevels] = {};
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int d = E - z_exp(a[q], as[q]);
#pragma unroll
            for (int l = 0; l < kZLevels; ++l) near[l] |= (d <= kZNear * l ? 1u : 0u) << ((q & 1) * 16 + (q >> 1));
        }
        s_ma[kh][r] = make_uint4(near[0] << 8 * kh, near[1] << 8 * kh, near[2] << 8 * kh, near[3] << 8 * kh);
#pragma unroll
        for (int part = 0; part < 2; ++part)
#pragma unroll
            for (int h = 0; h < 2; ++h) {      // 8 depths: a 16-byte chunk
                long long v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = z_fixed(part ? a[8 * h + q].im : a[8 * h + q].re, as[8 * h + q], E);
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
    // the loaded tile's digits into buffer u, its columns' exponents and masks into s_eb[e], s_mb[e]:
    // columns j (re) and 16 + j (im) of C' take [B_r | -B_i] and [B_i | B_r]
    auto cut_b = [&](int u, int e) {
        const int j = tid >> 4, k0 = (tid & 15) * 2;
        const int e0 = z_exp(b[0], bs[0]), e1 = z_exp(b[1], bs[1]);
        int E = max(e0, e1);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) E = max(E, __shfl_xor_sync(0xffffffffu, E, o));
        unsigned near[kZLevels];
#pragma unroll
        for (int l = 0; l < kZLevels; ++l) {
            const unsigned even = __ballot_sync(0xffffffffu, E - e0 <= kZNear * l), odd = __ballot_sync(0xffffffffu, E - e1 <= kZNear * l);
            near[l] = __byte_perm(even, odd, lane < 16 ? 0x5410 : 0x7632);
        }
        if ((tid & 15) == 0) {
            s_eb[e][j] = E;
            s_mb[e][j] = make_uint4(near[3], near[2], near[1], near[0]);   // beside the row's levels
        }
        long long vr[2], vi[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            vr[q] = z_fixed(b[q].re, bs[q], E);
            vi[q] = z_fixed(b[q].im, bs[q], E);
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
    // so do the sums a + b: 29 products of up to 224 columns (digit by digit, 136 products of 32
    // columns, the first update of four matrices of order 1500 took 317 us where it then took 196).
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
    int issued = tile0 < tile1 ? 1 : 0;   // tiles, buffers in turn
    const int Er = max(s_ea[0][ra], s_ea[1][ra]);
    const uint4 m0 = s_ma[0][ra], m1 = s_ma[1][ra], mr = make_uint4(m0.x | m1.x, m0.y | m1.y, m0.z | m1.z, m0.w | m1.w);
    for (int t = tile0; t < tile1; ++t) {
        const int u = (t - tile0) & 1, c0 = t * kZNc;
        cplx cc[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int col = c0 + half * 8 + q;
            cc[q] = row < J.m && col < J.n ? C[row + (long long)col * J.ldc] : mk(0.);
        }
        // bits of the thread's columns: to write from the products; left to z_direct (no depth serves
        // the entry, or its scale has no FP64 number).  Neither: a row or column of zeros.  First all
        // eight at once, by the depths that serve each of them: 8 loads and tests less.
        unsigned write = 0u, odd = 0u;
        {
            const int slot = (t - tile0) % 3;
            const uint4 mb = s_mb[slot][half * 8 + (lane & 7)];
            const int eb = s_eb[slot][half * 8 + (lane & 7)];
            const unsigned meet = (mr.x & __reduce_and_sync(0xffffffffu, mb.x)) | (mr.y & __reduce_and_sync(0xffffffffu, mb.y)) |
                                  (mr.z & __reduce_and_sync(0xffffffffu, mb.z)) | (mr.w & __reduce_and_sync(0xffffffffu, mb.w));
            const int lo = Er - 1076 + __reduce_min_sync(0xffffffffu, eb), hi = Er - 1076 + __reduce_max_sync(0xffffffffu, eb);
            if (meet && lo >= 0 && hi < 2046 && c0 + half * 8 + 8 <= J.n) {
                write = row < J.m ? 0xffu : 0u;
            } else {
#pragma unroll 1
                for (int q = 0; q < 8; ++q) {
                    const int j = half * 8 + q, es = Er + s_eb[slot][j] - 1075;
                    const uint4 m = s_mb[slot][j];
                    const bool one = ((mr.x & m.x) | (mr.y & m.y) | (mr.z & m.z) | (mr.w & m.w)) != 0u;
                    if (row < J.m && c0 + j < J.n && es > kZNone / 2) (one && (unsigned)(es - 1) < 2046u ? write : odd) |= 1u << q;
                }
            }
        }
        // the next tile's digits go where those of the tile before this one were, whose products
        // this thread has waited for; its exponents do not, slower warps may still read them (three
        // rounds: the barrier below has every warp past the tile before that one)
        if (t + 1 < tile1) cut_b(u ^ 1, (t + 1 - tile0) % 3);
        load_b(t + 2);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (__syncthreads_or(fail)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (t + 1 < tile1) {
            if (tid == 0) products(u ^ 1);
            ++issued;
        }
        __syncwarp();
        fail = __any_sync(0xffffffffu, !z_wait(z_smem(&mbar[u]), (uint32_t)(((t - tile0) >> 1) & 1)));
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
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
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                const int es = Er + s_eb[(t - tile0) % 3][j0 + jj] - 1075;
                const double nsc = __hiloint2double(fail ? 0x7ff80000 : (es << 20) | 0x80000000, 0);   // a wait that ran out shows
                const cplx c = cc[4 * jq + jj];
                const cplx o = mk(fma(nsc, (double)z_join(re, jj), c.re), fma(nsc, (double)z_join(im, jj), c.im));
                if ((write >> (4 * jq + jj)) & 1u) C[row + (long long)(c0 + j0 + jj) * J.ldc] = o;
            }
        }
        for (; odd; odd &= odd - 1) {
            const long long col = c0 + half * 8 + __ffs(odd) - 1;
            C[row + col * J.ldc] = z_direct(A + row, J.lda, B + col * J.ldb, J.k, C[row + col * J.ldc]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (__syncthreads_or(fail)) {   // another bounded chance for the products before the memory is given back
        if (tid == 0) atomicExch(J.info + blockIdx.z, -1);
        for (int u = 0; u < 2; ++u)
            if (const int count = (issued + 1 - u) >> 1) z_wait(z_smem(&mbar[u]), (uint32_t)((count - 1) & 1));
        __syncthreads();
    }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot), "r"(512u));
}

}  // namespace

// C_b -= A_b B_b for nmat matrices: m x n, depth k <= 32, column-major.  ek + b se: the biased
// exponents of the largest entries of B_b's k rows.  info[b]: set to -1 where a tensor-core wait ran out.
cudaError_t launch_zgemm_tc(int m, int n, int k, const cplx* A, long long lda, long long sa, const cplx* B, long long ldb,
                            long long sb, cplx* C, long long ldc, long long sc, const int* ek, long long se, int nmat,
                            int* info, cudaStream_t st) {
    if (m <= 0 || n <= 0 || k <= 0) return cudaSuccess;
    if (k > kZK || nmat < 1 || nmat > 65535) return cudaErrorInvalidValue;
    if (cudaError_t e = cudaFuncSetAttribute(k_zgemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kZSmem);
        e != cudaSuccess)
        return e;
    const int rt = (m + kZM - 1) / kZM, ct = (n + kZNc - 1) / kZNc;
    // tiles per CTA: one CTA per SM at a time, so as many as spread all the tiles over the 152
    const long long total = (long long)rt * ct * nmat;
    const int tiles = (int)std::max<long long>(1, std::min<long long>(ct, (total + 151) / 152));
    ZJob J{m, n, k, tiles, A, B, C, lda, ldb, ldc, sa, sb, sc, ek, se, info};
    const dim3 grid(rt, (ct + tiles - 1) / tiles, nmat);
    k_zgemm_tc<<<grid, kZThreads, kZSmem, st>>>(J);
    return cudaGetLastError();
}

}  // namespace hbem
