// The f64 functions of csrc/sb_f64.cuh and csrc/sb_line.cuh as the device evaluates them:
//   f64_functions_check <function> < doubles > doubles
// A value a result; exp2 and pow take pairs (n, f) and (x, p). Floats go in and out as doubles.
#include <cstdio>
#include <cstring>
#include <vector>

#include "sb_device.cuh"
#include "sb_line.cuh"

using namespace sbgpu;

__global__ void evaluate(int f, const double* in, double* out, int n) {
    __shared__ double tab[kF64TableDoubles];
    load_f64_tables(tab, threadIdx.x, blockDim.x);
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = in[f >= 6 ? 2 * i : i], w = f >= 6 ? in[2 * i + 1] : 0.0;
    switch (f) {
        case 0: out[i] = static_cast<double>(f64_to_f32(v)); break;
        case 1: out[i] = static_cast<double>(f64_to_f32_rn(v)); break;
        case 2: out[i] = f32_to_f64_exact(static_cast<float>(v)); break;
        case 3: out[i] = rcp_any(v); break;
        case 4: out[i] = sqrt_any(v); break;
        case 5: out[i] = rsqrt_any(v); break;
        case 6: out[i] = exp2_512_f64(static_cast<int>(v), w, tab); break;
        case 7: out[i] = pow_f64(v, w, tab); break;
    }
}

int main(int argc, char** argv) {
    static const char* names[] = {"to_f32", "to_f32_rn", "to_f64_exact", "rcp", "sqrt", "rsqrt", "exp2", "pow"};
    int f = -1;
    for (int k = 0; argc > 1 && k < 8; ++k)
        if (!std::strcmp(argv[1], names[k])) f = k;
    if (f < 0) return 2;
    std::vector<double> in;
    double v;
    while (std::fread(&v, sizeof v, 1, stdin) == 1) in.push_back(v);
    const int n = static_cast<int>(in.size()) / (f >= 6 ? 2 : 1);
    if (n == 0) return 0;
    double *din = nullptr, *dout = nullptr;
    std::vector<double> out(n);
    if (cudaMalloc(&din, in.size() * sizeof v) != cudaSuccess || cudaMalloc(&dout, n * sizeof v) != cudaSuccess) return 3;
    if (cudaMemcpy(din, in.data(), in.size() * sizeof v, cudaMemcpyHostToDevice) != cudaSuccess) return 3;
    evaluate<<<(n + 255) / 256, 256>>>(f, din, dout, n);
    if (cudaMemcpy(out.data(), dout, n * sizeof v, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    return std::fwrite(out.data(), sizeof v, n, stdout) == out.size() ? 0 : 4;
}
