// Error of the epilogue's silu(gate) * up against 64 bits, in units of 2^-24 of the result, beside that of the same formula with
// an IEEE division.  Prints "<largest> <mean>" of the epilogue's form, the same of the division, and how many results differ.
// Test code only.
#include <cmath>
#include <cstdio>

#include "../../fp6_llm_b200/csrc/fpx_epilogue.cuh"

constexpr int kGates = 1 << 20, kUps = 8;

struct Sums { double largest[2], sum[2]; unsigned long long differ; };

__global__ void evaluate(double* worst, double* total, unsigned long long* differ) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kGates) return;
    const float gate = -30.0f + 60.0f * (float)i / (float)kGates;   // every result is a normal fp32 number
    double largest[2] = {0.0, 0.0}, sum[2] = {0.0, 0.0};
    unsigned long long other = 0;
    for (int u = 0; u < kUps; u++) {
        const float up = (1.0f + 0.137f * (float)u) * (u & 1 ? -3.0f : 1.0f);
        const float form[2] = {fpx::silu_mul(gate, up), __fdiv_rn(gate, 1.0f + __expf(-gate)) * up};
        const double exact = (double)gate / (1.0 + exp(-(double)gate)) * (double)up;
        if (exact == 0.0) continue;
        for (int k = 0; k < 2; k++) {
            const double err = fabs((double)form[k] - exact) / fabs(exact) * 16777216.0;
            largest[k] = fmax(largest[k], err);
            sum[k] += err;
        }
        other += form[0] != form[1];
    }
    for (int k = 0; k < 2; k++) { worst[2 * i + k] = largest[k]; total[2 * i + k] = sum[k]; }
    differ[i] = other;
}

int main() {
    double *worst, *total;
    unsigned long long* differ;
    if (cudaMallocManaged(&worst, 2 * kGates * sizeof(double)) || cudaMallocManaged(&total, 2 * kGates * sizeof(double)) ||
        cudaMallocManaged(&differ, kGates * sizeof(*differ))) return 1;
    evaluate<<<kGates / 256, 256>>>(worst, total, differ);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    Sums s = {};
    for (int i = 0; i < kGates; i++) {
        for (int k = 0; k < 2; k++) {
            s.largest[k] = fmax(s.largest[k], worst[2 * i + k]);
            s.sum[k] += total[2 * i + k];
        }
        s.differ += differ[i];
    }
    for (int k = 0; k < 2; k++) printf("%.6f %.6f ", s.largest[k], s.sum[k] / ((double)kGates * kUps));
    printf("%llu\n", s.differ);
    return 0;
}
