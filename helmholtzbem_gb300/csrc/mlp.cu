// The learned resonance proposal's network: a multilayer perceptron
//   n_in -> width (GELU) -> ... -> width (GELU) -> n_out
// trained and evaluated on the GPU in BF16 with FP32 accumulation (weights kept in
// FP32 for the optimiser, BF16 copies for the products).
//
// Every product is one kernel: C (FP32, M x N, row-major) = A (BF16, M x K, row-major)
// x B (BF16, N x K, row-major)^T on the 5th-generation tensor cores (tcgen05.mma
// kind::f16 with BF16 operands, FP32 accumulator in tensor memory), K in chunks of 64
// staged in 128-byte-swizzled K-major shared memory.  Forward Y = X W^T; backward
// dX = dY W (B operand W^T), dW = dY^T X (the kernels that form activations and their
// gradients write the K-major transposes too), the dW of all layers in one launch.
// Shapes are padded on the host: rows and columns to multiples of 128, K to 64.
// A gradient (batch 256, width 512, 5 layers) is a chain of about twenty launches of a
// few microseconds, so what counts is how many there are and how much of a launch is
// waiting: 813 us a call with its parameters' gradient on the host, 314 now.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <random>
#include <string>
#include <vector>

#include "../../include/hbem.h"

namespace hbem {

int set_error(int code, const char* msg);
void count_launches(long long n);

namespace {

constexpr int kGM = 128, kGK = 64;
constexpr int kGThreads = 256;
constexpr uint32_t kGTileBytes = 128u * 128u;       // 128 rows x 128 bytes (64 BF16)
constexpr long long kGSpinCap = 1LL << 24;
constexpr int kGMaxJobs = 65;                       // layers of the deepest network

// instruction descriptor, kind::f16: D FP32 (bits 4-5 = 1), A and B BF16 (bits 7-9,
// 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at 24-28
__device__ constexpr uint32_t g_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kGM >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor for a 128-byte-swizzled K-major operand: start
// address >> 4, leading byte offset 1 (unused), stride byte offset 1024 >> 4 between
// 8-row groups, version 1, swizzle mode 128 B
__device__ __forceinline__ uint64_t sw128(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1u << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1u << 46;
    d |= (uint64_t)2u << 61;
    return d;
}

// byte offset of 16-byte chunk c (0..7) of row r in a 128-row swizzled tile
__device__ __forceinline__ uint32_t chunk_off(int r, int c) {
    return (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u + ((uint32_t)(c ^ (r & 7)) << 4);
}

struct GemmJob {
    int M, N, K;                 // multiples of 128, 128, 64
    const __nv_bfloat16* A;      // M x K, leading dimension lda (multiple of 8)
    const __nv_bfloat16* B;      // N x K, leading dimension ldb
    float* C;                    // M x N, leading dimension ldc
    long long lda, ldb, ldc;
    int* err;
};

struct GemmJobs {
    GemmJob j[kGMaxJobs];
};

template <int GN, int ST>
constexpr size_t g_smem() { return ST * (size_t)(kGTileBytes + GN * 128u) + 1024; }

__device__ __forceinline__ bool g_wait(uint32_t mbar, uint32_t parity) {
    uint32_t done = 0;
    for (long long it = 0; it < kGSpinCap && !done; ++it)
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
    return done != 0;
}

// A 128 x GN tile of job blockIdx.z; ST stages of K chunks in flight.  The network's products
// are small (256 x 512 x 512): their time is the latency of the chunks, one after the other
// when each was loaded, multiplied and waited for (12 us); with all in flight and narrow tiles
// over more SMs it is 6.7.  The sums of an entry are formed in the same order whatever GN is.
template <int GN, int ST>
__global__ void __launch_bounds__(kGThreads) k_gemm_bf16_tc(const __grid_constant__ GemmJobs JS) {
    const GemmJob& J = JS.j[blockIdx.z];
    const int r0 = blockIdx.x * kGM, c0 = blockIdx.y * GN;
    if (r0 >= J.M || c0 >= J.N) return;
    extern __shared__ uint8_t g_smem_raw[];
    uint8_t* As = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(g_smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* Bs = As + ST * kGTileBytes;
    __shared__ __align__(8) uint64_t mbar[ST];
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nk = J.K / kGK;
    auto load = [&](int kc) {   // chunk kc: rows of eight 16-byte pieces
        const int st = kc % ST;
#pragma unroll
        for (int q = 0; q < kGM * 8 / kGThreads; ++q) {
            const int e = tid + q * kGThreads, r = e >> 3, c = e & 7;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(As) + st * kGTileBytes + chunk_off(r, c)),
                         "l"(J.A + (long long)(r0 + r) * J.lda + kc * kGK + 8 * c)
                         : "memory");
        }
#pragma unroll
        for (int q = 0; q < GN * 8 / kGThreads; ++q) {
            const int e = tid + q * kGThreads, r = e >> 3, c = e & 7;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(Bs) + st * GN * 128u + chunk_off(r, c)),
                         "l"(J.B + (long long)(c0 + r) * J.ldb + kc * kGK + 8 * c)
                         : "memory");
        }
    };
    for (int kc = 0; kc < ST; ++kc) {
        if (kc < nk) load(kc);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                     "r"((uint32_t)GN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int q = 0; q < ST; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&mbar[q])), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t taddr = tmem_slot;
    bool fail = false;
    for (int kc = 0; kc < nk; ++kc) {
        // groups so far: ST, and one for each chunk before this; chunk kc is in one of all but the last ST - 2
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (__syncthreads_or(fail)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int st = kc % ST;
        if (tid == 0) {
#pragma unroll
            for (int kk = 0; kk < kGK / 16; ++kk) {
                const uint64_t ad = sw128(smem_addr(As) + st * kGTileBytes + (uint32_t)kk * 32u);
                const uint64_t bd = sw128(smem_addr(Bs) + st * GN * 128u + (uint32_t)kk * 32u);
                const uint32_t acc = (kc > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(taddr),
                    "l"(ad), "l"(bd), "r"(g_idesc(GN)), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&mbar[st]))
                         : "memory");
        }
        __syncwarp();
        // the chunk before this one is read by its products: wait (bounded), then overwrite its stage
        if (kc > 0 && kc - 1 + ST < nk) {
            if (!g_wait(smem_addr(&mbar[(kc - 1) % ST]), (uint32_t)(((kc - 1) / ST) & 1))) fail = true;
            else load(kc - 1 + ST);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (!g_wait(smem_addr(&mbar[(nk - 1) % ST]), (uint32_t)(((nk - 1) / ST) & 1))) fail = true;
    asm volatile("cp.async.wait_all;" ::: "memory");
    const bool bad = __syncthreads_or(fail);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!bad) {
        // epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 (rows), half w / 4 of the columns
        const int wq = warp & 3, half = warp >> 2;
        const int row = r0 + wq * 32 + lane;
        const uint32_t lane_base = taddr + ((uint32_t)(wq * 32) << 16);
        for (int j0 = half * GN / 2; j0 < (half + 1) * GN / 2; j0 += 16) {
            uint32_t v[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15])
                : "r"(lane_base + (uint32_t)j0));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float* out = J.C + (long long)row * J.ldc + c0 + j0;
#pragma unroll
            for (int jj = 0; jj < 16; jj += 4)
                *reinterpret_cast<float4*>(out + jj) = make_float4(__uint_as_float(v[jj]), __uint_as_float(v[jj + 1]),
                                                                   __uint_as_float(v[jj + 2]),
                                                                   __uint_as_float(v[jj + 3]));
        }
    } else if (tid == 0) {
        atomicExch(J.err, 1);
        for (int q = 0; q < ST; ++q) g_wait(smem_addr(&mbar[q]), 0u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"((uint32_t)GN));
    }
}

// FP32 FMA reference of the same product (one thread per output), for tests
__global__ void k_gemm_bf16_simt(GemmJob J) {
    const int i = blockIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= J.M || j >= J.N) return;
    float acc = 0.f;
    for (int k = 0; k < J.K; ++k)
        acc = fmaf(__bfloat162float(J.A[(long long)i * J.lda + k]), __bfloat162float(J.B[(long long)j * J.ldb + k]), acc);
    J.C[(long long)i * J.ldc + j] = acc;
}

// ------------------------------------------------------------------ elementwise kernels

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// The kernels around the products work on 32 x 32 tiles (block 32 x 8; grid row tiles x column
// tiles, a batch may have more than the 65,535 that y takes) of a padded rows x cols matrix, so that
// they can write the transpose that a later product reads.

// Z = C + bias (pre-activation, kept for the backward pass); H = act(Z) in BF16, HT its
// transpose (each where not null)
// (rows x cols of the padded layout, cols_used real columns, the rest zero)
__global__ void __launch_bounds__(256) k_bias_act(int rows, int cols, int cols_used, int rows_used, const float* C,
                                                  const float* bias, int act, float* Z, __nv_bfloat16* H,
                                                  __nv_bfloat16* HT) {
    __shared__ __nv_bfloat16 t[32][33];
    const int c = blockIdx.y * 32 + threadIdx.x, r0 = blockIdx.x * 32;
    const float bc = c < cols_used ? bias[c] : 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = r0 + threadIdx.y + 8 * q;
        const long long e = (long long)r * cols + c;
        float z = 0.f;
        if (c < cols_used && r < rows_used) z = C[e] + bc;
        if (Z) Z[e] = z;
        const __nv_bfloat16 h = __float2bfloat16(act ? gelu(z) : z);
        if (H) H[e] = h;
        t[threadIdx.y + 8 * q][threadIdx.x] = h;
    }
    if (!HT) return;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int tc = threadIdx.y + 8 * q;
        HT[(long long)(blockIdx.y * 32 + tc) * rows + r0 + threadIdx.x] = t[threadIdx.x][tc];
    }
}

// A layer's gradient dZ at the tile: BF16 copies Gb (where not null) and, transposed, GT, and the
// tile's column sums (the bias gradient's parts) to part[row tile][cols].
__device__ __forceinline__ void grad_tile(int rows, int cols, const float (&g)[4], __nv_bfloat16* Gb, __nv_bfloat16* GT,
                                          float* part) {
    __shared__ __nv_bfloat16 t[32][33];
    __shared__ float cs[8][33];
    const int c = blockIdx.y * 32 + threadIdx.x, r0 = blockIdx.x * 32;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const __nv_bfloat16 h = __float2bfloat16(g[q]);
        if (Gb) Gb[(long long)(r0 + threadIdx.y + 8 * q) * cols + c] = h;
        t[threadIdx.y + 8 * q][threadIdx.x] = h;
    }
    cs[threadIdx.y][threadIdx.x] = (g[0] + g[1]) + (g[2] + g[3]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int tc = threadIdx.y + 8 * q;
        GT[(long long)(blockIdx.y * 32 + tc) * rows + r0 + threadIdx.x] = t[threadIdx.x][tc];
    }
    if (threadIdx.y == 0) {
        float s = 0.f;
#pragma unroll
        for (int y = 0; y < 8; ++y) s += cs[y][threadIdx.x];
        part[(long long)blockIdx.x * cols + c] = s;
    }
}

// loss += sum of squared errors over the used rows / columns / count; dZ = 2 (Y - T) / count
__global__ void __launch_bounds__(256) k_mse(int rows, int cols, int rows_used, int cols_used, const float* Y,
                                             const float* T, float inv_count, __nv_bfloat16* Gb, __nv_bfloat16* GT,
                                             float* part, float* loss) {
    const int c = blockIdx.y * 32 + threadIdx.x;
    float g[4], s = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = blockIdx.x * 32 + threadIdx.y + 8 * q;
        float d = 0.f;
        if (r < rows_used && c < cols_used) d = Y[(long long)r * cols + c] - T[(long long)r * cols_used + c];
        g[q] = 2.f * d * inv_count;
        s = fmaf(d, d, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0 && s != 0.f) atomicAdd(loss, s * inv_count);
    grad_tile(rows, cols, g, Gb, GT, part);
}

// dZ = dH * GELU'(Z)
__global__ void __launch_bounds__(256) k_act_bwd(int rows, int cols, const float* Z, const float* dH, __nv_bfloat16* Gb,
                                                 __nv_bfloat16* GT, float* part) {
    const int c = blockIdx.y * 32 + threadIdx.x;
    float g[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const long long e = (long long)(blockIdx.x * 32 + threadIdx.y + 8 * q) * cols + c;
        g[q] = dH[e] * gelu_grad(Z[e]);
    }
    grad_tile(rows, cols, g, Gb, GT, part);
}

// The bias gradients of all layers from their tiles' column sums; grid (columns, layers)
struct SumJobs {
    int parts, cols[kGMaxJobs];
    const float* part[kGMaxJobs];
    float* out[kGMaxJobs];
};
__global__ void __launch_bounds__(128) k_colsum(const __grid_constant__ SumJobs J) {
    const int l = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= J.cols[l]) return;
    float s = 0.f;
#pragma unroll 8
    for (int q = 0; q < J.parts; ++q) s += J.part[l][(long long)q * J.cols[l] + c];
    J.out[l][c] = s;
}

// A layer's parameters between their padded arrays and their place in one vector: W (o x i,
// row-major), then b.  TO: the arrays' real entries to the vector, else from it.
template <bool TO>
__global__ void __launch_bounds__(256) k_pack(int o, int i, int ip, float* W, float* b, float* v) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x, nw = (long long)o * i;
    if (e >= nw + o) return;
    float* a = e < nw ? W + e / i * ip + e % i : b + (e - nw);
    if (TO) v[e] = *a;
    else *a = v[e];
}

// out (cols x rows) = in (rows x cols)^T, BF16
__global__ void k_transpose_bf16(int rows, int cols, const __nv_bfloat16* in, __nv_bfloat16* out) {
    __shared__ __nv_bfloat16 t[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int r = by + j, c = bx + threadIdx.x;
        if (r < rows && c < cols) t[j][threadIdx.x] = in[(long long)r * cols + c];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int c = bx + j, r = by + threadIdx.x;
        if (r < rows && c < cols) out[(long long)c * rows + r] = t[threadIdx.x][j];
    }
}

__global__ void k_to_bf16(long long n, const float* in, __nv_bfloat16* out) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e < n) out[e] = __float2bfloat16(in[e]);
}

// Adam on the FP32 master copy (bias-corrected step), BF16 copy refreshed
__global__ void k_adam(long long n, float* p, const float* g, float* m, float* v, float lr, float b1, float b2,
                       float eps, float c1, float c2, __nv_bfloat16* pb) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= n) return;
    const float gi = g[e];
    const float mi = b1 * m[e] + (1.f - b1) * gi, vi = b2 * v[e] + (1.f - b2) * gi * gi;
    m[e] = mi;
    v[e] = vi;
    const float q = p[e] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[e] = q;
    if (pb) pb[e] = __float2bfloat16(q);
}

// ------------------------------------------------------------------ host side

int round_up(int x, int m) { return (x + m - 1) / m * m; }

#define ML_CK(x)                                                                                       \
    do {                                                                                               \
        cudaError_t e_ = (x);                                                                          \
        if (e_ != cudaSuccess) return set_error(HBEM_ERR_CUDA, (std::string(#x) + ": " + cudaGetErrorString(e_)).c_str()); \
    } while (0)

template <class T>
struct DVec {
    T* p = nullptr;
    size_t n = 0;
    cudaError_t ensure(size_t count) {
        if (count <= n) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        cudaError_t e = cudaMalloc(&p, std::max<size_t>(1, count) * sizeof(T));
        if (e == cudaSuccess) n = count;
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
};

bool g_mlp_tensor_cores = true;

}  // namespace

namespace {

template <int GN, int ST>
cudaError_t launch_gemm(const GemmJobs& JS, int count, int mt, int nt, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(k_gemm_bf16_tc<GN, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)g_smem<GN, ST>());
    if (e != cudaSuccess) return e;
    k_gemm_bf16_tc<GN, ST><<<dim3(mt, nt, count), kGThreads, g_smem<GN, ST>(), st>>>(JS);
    return cudaGetLastError();
}

// count independent products.  Where the 32-column tiles still are one to an SM (152) they spread
// the work over four times the SMs that 128-column ones do, with eight chunks of K in flight; past
// that they read A more often for nothing: 1280 x 1280 x 512 (100 wide tiles) 36.9 us a call with
// narrow tiles, 29.1 with wide.  Wide tiles: three chunks, so that two CTAs fit an SM.
cudaError_t gemm_bf16_jobs(const GemmJobs& JS, int count, bool tc, cudaStream_t st) {
    long long tiles = 0;
    int mt = 0, n = 0;
    for (int q = 0; q < count; ++q) {
        const GemmJob& J = JS.j[q];
        if (J.M % kGM || J.N % 128 || J.K % kGK || J.lda % 8 || J.ldb % 8 || J.ldc % 4 || J.M <= 0 || J.N <= 0 || J.K <= 0)
            return cudaErrorInvalidValue;
        tiles += (long long)(J.M / kGM) * (J.N / 128);
        mt = std::max(mt, J.M / kGM);
        n = std::max(n, J.N);
    }
    if (!tc) {
        for (int q = 0; q < count; ++q)
            k_gemm_bf16_simt<<<dim3((JS.j[q].N + 127) / 128, JS.j[q].M), 128, 0, st>>>(JS.j[q]);
        return cudaGetLastError();
    }
    return 4 * tiles <= 152 ? launch_gemm<32, 8>(JS, count, mt, n / 32, st) : launch_gemm<128, 3>(JS, count, mt, n / 128, st);
}

}  // namespace

cudaError_t gemm_bf16(int M, int N, int K, const __nv_bfloat16* A, long long lda, const __nv_bfloat16* B,
                      long long ldb, float* C, long long ldc, int* err, bool tc, cudaStream_t st) {
    GemmJobs JS;
    JS.j[0] = GemmJob{M, N, K, A, B, C, lda, ldb, ldc, err};
    return gemm_bf16_jobs(JS, 1, tc, st);
}

void mlp_set_tensor_cores(int on) { g_mlp_tensor_cores = on != 0; }
int mlp_get_tensor_cores() { return g_mlp_tensor_cores ? 1 : 0; }

}  // namespace hbem

using namespace hbem;

// A layer: W (out x in, row-major, padded to out_p x in_p), b (out)
struct hbem_mlp_s {
    int n_in = 0, width = 0, depth = 0, n_out = 0, nlayers = 0, device = 0;
    std::vector<int> din, dout, din_p, dout_p;           // per layer, real and padded
    std::vector<DVec<float>> W, b, gW, gb, mW, vW, mb, vb;
    std::vector<DVec<__nv_bfloat16>> Wb, WTb;             // BF16 copies: W and W^T (in_p x out_p)
    std::vector<DVec<float>> Z;                           // pre-activations (batch_p x out_p)
    std::vector<DVec<__nv_bfloat16>> H;                   // activations, layer inputs (batch_p x in_p)
    std::vector<DVec<__nv_bfloat16>> HT, GT;              // transposes of H (layers >= 1) and of the gradients dZ
    std::vector<DVec<float>> part;                        // column sums of dZ by tiles of 32 rows
    DVec<float> C, Y, T, flat;                            // flat: all parameters or gradients as one vector
    DVec<__nv_bfloat16> Gb;
    DVec<int> err;                                        // [0] a product's wait ran out, [1] the loss (float)
    float* loss() { return reinterpret_cast<float*>(err.p + 1); }
    long long step = 0;
    ~hbem_mlp_s() {
        for (auto* v : {&W, &b, &gW, &gb, &mW, &vW, &mb, &vb, &Z, &part})
            for (auto& d : *v) d.release();
        for (auto* v : {&Wb, &WTb, &H, &HT, &GT})
            for (auto& d : *v) d.release();
        C.release(); Y.release(); T.release(); flat.release(); Gb.release(); err.release();
    }
};

namespace {

long long nblk(long long n, int t = 256) { return (n + t - 1) / t; }

int refresh_bf16(hbem_mlp m, int l) {
    const long long n = (long long)m->dout_p[l] * m->din_p[l];
    k_to_bf16<<<(unsigned)nblk(n), 256>>>(n, m->W[l].p, m->Wb[l].p);
    k_transpose_bf16<<<dim3((m->din_p[l] + 31) / 32, (m->dout_p[l] + 31) / 32), dim3(32, 8)>>>(
        m->dout_p[l], m->din_p[l], m->Wb[l].p, m->WTb[l].p);
    count_launches(2);
    ML_CK(cudaGetLastError());
    return HBEM_OK;
}

// forward over a padded batch already in m->H[0]; output FP32 in m->Y (batch_p x out_p);
// transposes: the layers' transposed inputs for the backward pass too
int forward(hbem_mlp m, int batch, int batch_p, bool transposes) {
    for (int l = 0; l < m->nlayers; ++l) {
        const bool last = l == m->nlayers - 1;
        ML_CK(m->Z[l].ensure((size_t)batch_p * m->dout_p[l]));
        ML_CK(gemm_bf16(batch_p, m->dout_p[l], m->din_p[l], m->H[l].p, m->din_p[l], m->Wb[l].p, m->din_p[l], m->C.p,
                        m->dout_p[l], m->err.p, g_mlp_tensor_cores, 0));
        const dim3 grid(batch_p / 32, m->dout_p[l] / 32), block(32, 8);
        if (!last) {
            ML_CK(m->H[l + 1].ensure((size_t)batch_p * m->din_p[l + 1]));
            if (transposes) ML_CK(m->HT[l + 1].ensure((size_t)batch_p * m->din_p[l + 1]));
            k_bias_act<<<grid, block>>>(batch_p, m->dout_p[l], m->dout[l], batch, m->C.p, m->b[l].p, 1, m->Z[l].p,
                                        m->H[l + 1].p, transposes ? m->HT[l + 1].p : nullptr);
        } else {
            k_bias_act<<<grid, block>>>(batch_p, m->dout_p[l], m->dout[l], batch, m->C.p, m->b[l].p, 0, m->Y.p, nullptr,
                                        nullptr);
        }
        count_launches(2);
        ML_CK(cudaGetLastError());
    }
    return HBEM_OK;
}

// the batch in BF16, padded, to m->H[0]; behind it, for a backward pass, its transpose
int load_batch(hbem_mlp m, const float* X_host, int batch, int batch_p, bool transposes) {
    const int w0 = std::max(m->din_p[0], 1);
    const size_t n = (size_t)batch_p * w0;
    std::vector<__nv_bfloat16> xb((transposes ? 2 : 1) * n, __float2bfloat16(0.f));
    for (int r = 0; r < batch; ++r)
        for (int c = 0; c < m->n_in; ++c) {
            const __nv_bfloat16 v = __float2bfloat16(X_host[(size_t)r * m->n_in + c]);
            xb[(size_t)r * w0 + c] = v;
            if (transposes) xb[n + (size_t)c * batch_p + r] = v;
        }
    ML_CK(m->H[0].ensure(xb.size()));
    ML_CK(cudaMemcpy(m->H[0].p, xb.data(), xb.size() * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice));
    const int wmax = *std::max_element(m->dout_p.begin(), m->dout_p.end());
    ML_CK(m->C.ensure((size_t)batch_p * std::max(wmax, *std::max_element(m->din_p.begin(), m->din_p.end()))));
    ML_CK(m->Y.ensure((size_t)batch_p * m->dout_p.back()));
    return HBEM_OK;
}

// loss + backward after forward: gradients in gW, gb (launched, not waited for)
int backward(hbem_mlp m, const float* T_host, int batch, int batch_p) {
    const int L = m->nlayers, rt = batch_p / 32;
    const int wmax = *std::max_element(m->dout_p.begin(), m->dout_p.end());
    const dim3 block(32, 8);
    ML_CK(m->T.ensure((size_t)batch * m->n_out));
    ML_CK(cudaMemcpy(m->T.p, T_host, (size_t)batch * m->n_out * sizeof(float), cudaMemcpyHostToDevice));
    ML_CK(m->Gb.ensure((size_t)batch_p * wmax));
    for (int l = 0; l < L; ++l) {
        ML_CK(m->GT[l].ensure((size_t)batch_p * m->dout_p[l]));
        ML_CK(m->part[l].ensure((size_t)rt * m->dout_p[l]));
    }
    ML_CK(cudaMemsetAsync(m->loss(), 0, sizeof(float), 0));
    const int no = m->dout_p[L - 1];
    k_mse<<<dim3(rt, no / 32), block>>>(batch_p, no, batch, m->n_out, m->Y.p, m->T.p,
                                        1.f / (float)((long long)batch * m->n_out), m->Gb.p, m->GT[L - 1].p,
                                        m->part[L - 1].p, m->loss());
    count_launches(1);
    for (int l = L - 1; l > 0; --l) {
        const int op = m->dout_p[l], ip = m->din_p[l];
        // dH = dZ W: A = dZ (batch_p x op), B = W^T (ip x op)
        ML_CK(gemm_bf16(batch_p, ip, op, m->Gb.p, op, m->WTb[l].p, op, m->C.p, ip, m->err.p, g_mlp_tensor_cores, 0));
        // dZ_(l-1) = dH * GELU'(Z_(l-1)) (the padded columns stay zero: Z there is zero, dH too)
        k_act_bwd<<<dim3(rt, ip / 32), block>>>(batch_p, ip, m->Z[l - 1].p, m->C.p, l > 1 ? m->Gb.p : nullptr,
                                                m->GT[l - 1].p, m->part[l - 1].p);
        count_launches(2);
        ML_CK(cudaGetLastError());
    }
    // dW = dZ^T H of every layer: A = dZ^T (op x batch_p), B = H^T (ip x batch_p)
    GemmJobs JS;
    SumJobs SJ;
    SJ.parts = rt;
    for (int l = 0; l < L; ++l) {
        const __nv_bfloat16* ht = l ? m->HT[l].p : m->H[0].p + (size_t)batch_p * m->din_p[0];
        JS.j[l] = GemmJob{m->dout_p[l], m->din_p[l], batch_p, m->GT[l].p, ht, m->gW[l].p, batch_p, batch_p, m->din_p[l], m->err.p};
        SJ.cols[l] = m->dout_p[l];
        SJ.part[l] = m->part[l].p;
        SJ.out[l] = m->gb[l].p;
    }
    ML_CK(gemm_bf16_jobs(JS, L, g_mlp_tensor_cores, 0));
    k_colsum<<<dim3((unsigned)nblk(wmax, 128), L), 128>>>(SJ);
    count_launches(2);
    ML_CK(cudaGetLastError());
    return HBEM_OK;
}

}  // namespace

extern "C" {

int hbem_mlp_create(int n_in, int width, int depth, int n_out, unsigned long long seed, hbem_mlp* out) {
    if (n_in < 1 || width < 1 || depth < 1 || n_out < 1 || !out || n_in > 4096 || width > 8192 || depth > 64 ||
        n_out > 8192)
        return set_error(HBEM_ERR_INVALID, "mlp_create: bad argument");
    hbem_mlp m = new hbem_mlp_s;
    m->n_in = n_in;
    m->width = width;
    m->depth = depth;
    m->n_out = n_out;
    m->nlayers = depth + 1;
    cudaGetDevice(&m->device);
    for (int l = 0; l < m->nlayers; ++l) {
        const int i = l == 0 ? n_in : width, o = l == depth ? n_out : width;
        m->din.push_back(i);
        m->dout.push_back(o);
        m->din_p.push_back(round_up(i, 128));    // a layer's input is the previous output (padded to 128)
        m->dout_p.push_back(round_up(o, 128));
    }
    const int L = m->nlayers;
    m->W.resize(L); m->b.resize(L); m->gW.resize(L); m->gb.resize(L);
    m->mW.resize(L); m->vW.resize(L); m->mb.resize(L); m->vb.resize(L);
    m->Wb.resize(L); m->WTb.resize(L); m->Z.resize(L); m->H.resize(L + 1);
    m->HT.resize(L); m->GT.resize(L); m->part.resize(L);
    std::mt19937_64 gen(seed);
    for (int l = 0; l < L; ++l) {
        const size_t nw = (size_t)m->dout_p[l] * m->din_p[l];
        // He-style initialisation, zero padding
        std::normal_distribution<float> nd(0.f, std::sqrt(2.f / (float)m->din[l]));
        std::vector<float> w(nw, 0.f), z(nw, 0.f), bz(m->dout_p[l], 0.f);
        for (int r = 0; r < m->dout[l]; ++r)
            for (int c = 0; c < m->din[l]; ++c) w[(size_t)r * m->din_p[l] + c] = nd(gen);
        for (auto* d : {&m->W[l], &m->gW[l], &m->mW[l], &m->vW[l]})
            if (d->ensure(nw) != cudaSuccess) { delete m; return set_error(HBEM_ERR_NOMEM, "mlp_create: cudaMalloc"); }
        for (auto* d : {&m->b[l], &m->gb[l], &m->mb[l], &m->vb[l]})
            if (d->ensure(m->dout_p[l]) != cudaSuccess) { delete m; return set_error(HBEM_ERR_NOMEM, "mlp_create: cudaMalloc"); }
        if (m->Wb[l].ensure(nw) != cudaSuccess || m->WTb[l].ensure(nw) != cudaSuccess) {
            delete m;
            return set_error(HBEM_ERR_NOMEM, "mlp_create: cudaMalloc");
        }
        cudaMemcpy(m->W[l].p, w.data(), nw * sizeof(float), cudaMemcpyHostToDevice);
        for (auto* d : {&m->gW[l], &m->mW[l], &m->vW[l]}) cudaMemcpy(d->p, z.data(), nw * sizeof(float), cudaMemcpyHostToDevice);
        for (auto* d : {&m->b[l], &m->gb[l], &m->mb[l], &m->vb[l]})
            cudaMemcpy(d->p, bz.data(), bz.size() * sizeof(float), cudaMemcpyHostToDevice);
        if (int r = refresh_bf16(m, l)) { delete m; return r; }
    }
    if (m->err.ensure(2) != cudaSuccess) { delete m; return set_error(HBEM_ERR_NOMEM, "mlp_create: cudaMalloc"); }
    cudaMemset(m->err.p, 0, 2 * sizeof(int));
    if (cudaDeviceSynchronize() != cudaSuccess) { delete m; return set_error(HBEM_ERR_CUDA, "mlp_create: CUDA error"); }
    *out = m;
    return HBEM_OK;
}

int hbem_mlp_destroy(hbem_mlp m) {
    delete m;
    return HBEM_OK;
}

int hbem_mlp_num_params(hbem_mlp m, long long* count) {
    if (!m || !count) return set_error(HBEM_ERR_INVALID, "mlp: bad argument");
    long long c = 0;
    for (int l = 0; l < m->nlayers; ++l) c += (long long)m->dout[l] * m->din[l] + m->dout[l];
    *count = c;
    return HBEM_OK;
}

// parameters (or gradients) as one vector: per layer W (out x in, row-major) then b.  One copy
// between host and device; the padded arrays are packed and unpacked there (a copy and a host
// loop per layer took 390 us for 870,000 gradients, half of a training step's gradient).
static int params_io(hbem_mlp m, float* host, int which, bool to_host) {
    if (!m || !host) return set_error(HBEM_ERR_INVALID, "mlp: bad argument");
    long long count = 0;
    if (int r = hbem_mlp_num_params(m, &count)) return r;
    ML_CK(m->flat.ensure((size_t)count));
    if (!to_host) ML_CK(cudaMemcpy(m->flat.p, host, (size_t)count * sizeof(float), cudaMemcpyHostToDevice));
    long long off = 0;
    for (int l = 0; l < m->nlayers; ++l) {
        float* W = which ? m->gW[l].p : m->W[l].p;
        float* b = which ? m->gb[l].p : m->b[l].p;
        const long long n = (long long)m->dout[l] * m->din[l] + m->dout[l];
        if (to_host) k_pack<true><<<(unsigned)nblk(n), 256>>>(m->dout[l], m->din[l], m->din_p[l], W, b, m->flat.p + off);
        else k_pack<false><<<(unsigned)nblk(n), 256>>>(m->dout[l], m->din[l], m->din_p[l], W, b, m->flat.p + off);
        count_launches(1);
        ML_CK(cudaGetLastError());
        off += n;
        if (!to_host)
            if (int r = refresh_bf16(m, l)) return r;
    }
    if (to_host) ML_CK(cudaMemcpy(host, m->flat.p, (size_t)count * sizeof(float), cudaMemcpyDeviceToHost));
    else ML_CK(cudaStreamSynchronize(0));
    return HBEM_OK;
}

int hbem_mlp_get_params(hbem_mlp m, float* host) { return params_io(m, host, 0, true); }
int hbem_mlp_set_params(hbem_mlp m, const float* host) { return params_io(m, const_cast<float*>(host), 0, false); }

int hbem_mlp_forward(hbem_mlp m, const float* X_host, int batch, float* Y_host) {
    if (!m || !X_host || !Y_host || batch < 1) return set_error(HBEM_ERR_INVALID, "mlp_forward: bad argument");
    ML_CK(cudaSetDevice(m->device));
    const int bp = round_up(batch, 128);
    if (int r = load_batch(m, X_host, batch, bp, false)) return r;
    if (int r = forward(m, batch, bp, false)) return r;
    const int op = m->dout_p.back();
    std::vector<float> y((size_t)bp * op);
    ML_CK(cudaMemcpy(y.data(), m->Y.p, y.size() * sizeof(float), cudaMemcpyDeviceToHost));
    int e = 0;
    ML_CK(cudaMemcpy(&e, m->err.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) return set_error(HBEM_ERR_NOCONV, "mlp: a tensor-core completion wait timed out");
    for (int r = 0; r < batch; ++r)
        for (int c = 0; c < m->n_out; ++c) Y_host[(size_t)r * m->n_out + c] = y[(size_t)r * op + c];
    return HBEM_OK;
}

int hbem_mlp_gradients(hbem_mlp m, const float* X_host, const float* T_host, int batch, float* loss_host,
                       float* grads_host) {
    if (!m || !X_host || !T_host || !loss_host || batch < 1) return set_error(HBEM_ERR_INVALID, "mlp: bad argument");
    ML_CK(cudaSetDevice(m->device));
    const int bp = round_up(batch, 128);
    if (int r = load_batch(m, X_host, batch, bp, true)) return r;
    if (int r = forward(m, batch, bp, true)) return r;
    if (int r = backward(m, T_host, batch, bp)) return r;
    struct {
        int err;
        float loss;
    } end;
    static_assert(sizeof(end) == 2 * sizeof(int), "as m->err");
    ML_CK(cudaMemcpy(&end, m->err.p, sizeof(end), cudaMemcpyDeviceToHost));
    *loss_host = end.loss;
    if (end.err) return set_error(HBEM_ERR_NOCONV, "mlp: a tensor-core completion wait timed out");
    if (grads_host) return params_io(m, grads_host, 1, true);
    return HBEM_OK;
}

int hbem_mlp_train_step(hbem_mlp m, const float* X_host, const float* T_host, int batch, float lr, float* loss_host) {
    if (int r = hbem_mlp_gradients(m, X_host, T_host, batch, loss_host, nullptr)) return r;
    ++m->step;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
    for (int l = 0; l < m->nlayers; ++l) {
        const long long nw = (long long)m->dout_p[l] * m->din_p[l];
        k_adam<<<(unsigned)nblk(nw), 256>>>(nw, m->W[l].p, m->gW[l].p, m->mW[l].p, m->vW[l].p, lr, b1, b2, eps, c1, c2,
                                           m->Wb[l].p);
        k_adam<<<(unsigned)nblk(m->dout_p[l]), 256>>>(m->dout_p[l], m->b[l].p, m->gb[l].p, m->mb[l].p, m->vb[l].p, lr,
                                                     b1, b2, eps, c1, c2, nullptr);
        k_transpose_bf16<<<dim3((m->din_p[l] + 31) / 32, (m->dout_p[l] + 31) / 32), dim3(32, 8)>>>(
            m->dout_p[l], m->din_p[l], m->Wb[l].p, m->WTb[l].p);
        count_launches(3);
    }
    ML_CK(cudaGetLastError());
    return HBEM_OK;
}

int hbem_bf16_gemm_device(int M, int N, int K, const void* A, long long lda, const void* B, long long ldb, void* C,
                          long long ldc, int tensor_cores) {
    if (!A || !B || !C) return set_error(HBEM_ERR_INVALID, "bf16_gemm: bad argument");
    static thread_local DVec<int> err;
    ML_CK(err.ensure(1));
    ML_CK(cudaMemset(err.p, 0, sizeof(int)));
    cudaError_t e = gemm_bf16(M, N, K, static_cast<const __nv_bfloat16*>(A), lda, static_cast<const __nv_bfloat16*>(B),
                              ldb, static_cast<float*>(C), ldc, err.p, tensor_cores != 0, 0);
    if (e == cudaErrorInvalidValue)
        return set_error(HBEM_ERR_INVALID, "bf16_gemm: M, N must be multiples of 128, K of 64, lda, ldb of 8");
    ML_CK(e);
    count_launches(1);
    int h = 0;
    ML_CK(cudaMemcpy(&h, err.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (h) return set_error(HBEM_ERR_NOCONV, "bf16_gemm: a tensor-core completion wait timed out");
    return HBEM_OK;
}

}  // extern "C"
