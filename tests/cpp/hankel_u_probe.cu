// f(u), g(u) as the real-wavenumber kernels take them (hk_pair) for the doubles in argv[1]:
// four doubles per argument into argv[2].
#include <cstdio>
#include <vector>

#include "../../helmholtzbem_gb300/csrc/hankel_u.cuh"

using namespace hbem;

__global__ void k_probe(const HkEntry* tab, int n, const double* u, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    cplx f, g;
    hk_pair(tab, u[i], f, g);
    out[4 * i] = f.re;
    out[4 * i + 1] = f.im;
    out[4 * i + 2] = g.re;
    out[4 * i + 3] = g.im;
}

int main(int argc, char** argv) {
    FILE* in = argc == 3 ? std::fopen(argv[1], "rb") : nullptr;
    if (!in) return 2;
    std::vector<double> u;
    for (double x; std::fread(&x, sizeof x, 1, in) == 1;) u.push_back(x);
    std::fclose(in);
    const int n = (int)u.size();
    std::vector<double> out(4 * u.size());
    double *du = nullptr, *dout = nullptr;
    cudaError_t e = cudaMalloc(&du, n * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&dout, 4 * n * sizeof(double));
    if (e == cudaSuccess) e = cudaMemcpy(du, u.data(), n * sizeof(double), cudaMemcpyHostToDevice);
    const HkEntry* tab = e == cudaSuccess ? hankel_table(&e) : nullptr;
    if (e == cudaSuccess) {
        k_probe<<<(n + 127) / 128, 128>>>(tab, n, du, dout);
        e = cudaMemcpy(out.data(), dout, 4 * n * sizeof(double), cudaMemcpyDeviceToHost);
    }
    if (e != cudaSuccess) {
        std::fprintf(stderr, "%s\n", cudaGetErrorString(e));
        return 1;
    }
    FILE* f = std::fopen(argv[2], "wb");
    if (!f || std::fwrite(out.data(), sizeof(double), out.size(), f) != out.size()) return 3;
    return std::fclose(f);
}
