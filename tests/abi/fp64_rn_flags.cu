// The branch-free FP64 forms where their tests for extreme operands decide: roots of every operand in
// range, mantissas of all ones (which `ordinary` refuses) among them, and how many of them are flagged;
// and `plain`, which must accept no operand whose reciprocal is not CUDA's, and few fewer than
// `ordinary`.  Prints: roots that differ without a flag, flagged roots, operands that `plain` accepts
// and `ordinary` does not, reciprocals of plain operands that differ, ordinary operands with random
// mantissas that `plain` refuses.
#include <cstdio>

#include "fp64_rn.cuh"

namespace {
constexpr int kBlocks = 296, kThreads = 256, kPerThread = 1000;

__device__ unsigned long long next(unsigned long long& s) {  // splitmix64
    s += 0x9E3779B97F4A7C15ull;
    unsigned long long z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void check(unsigned long long* bad) {
    using namespace lica::rn;
    unsigned long long s = (blockIdx.x * (unsigned long long)kThreads + threadIdx.x) * 1000033ull + 11;
    unsigned long long n[5] = {0, 0, 0, 0, 0};
    for (int i = 0; i < kPerThread; ++i) {
        const int kind = i & 3;
        unsigned long long m = next(s) & 0xfffffffffffffull;
        if (kind == 0) m = 0xfffffffffffffull - (next(s) & 3);   // all ones, and up to three units less
        if (kind == 1) m |= 0xffffffffull;                       // a low word of all ones
        const unsigned long long e = 1023 - 399 + next(s) % 798;
        const double x = __longlong_as_double((long long)(m | (e << 52)));
        if (!in_range(x)) continue;
        bool ok = true;
        const double r = root(x, ok);
        n[0] += ok && __double_as_longlong(r) != __double_as_longlong(sqrt(x));
        n[1] += !ok;
        const double b = (next(s) & 1) ? -x : x;
        n[2] += plain(b) && !ordinary(b);
        n[3] += plain(b) && __double_as_longlong(recip(b)) != __double_as_longlong(1.0 / b);
        n[4] += kind >= 2 && ordinary(b) && !plain(b);
    }
    for (int k = 0; k < 5; ++k) atomicAdd(bad + k, n[k]);
}
}  // namespace

int main() {
    unsigned long long *d = nullptr, h[5] = {1, 1, 1, 1, 1};
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 2;
    check<<<kBlocks, kThreads>>>(d);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("%llu %llu %llu %llu %llu\n", h[0], h[1], h[2], h[3], h[4]);
    return 0;
}
