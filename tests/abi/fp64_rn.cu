// Compares the branch-free FP64 reciprocal, quotient and square root with CUDA's operators, bit for
// bit, on seeded operands over the range they are specified for, mantissas near zero and near all
// ones among them.  Prints the number of reciprocals, quotients and unflagged roots that differ.
#include <cstdio>

#include "fp64_rn.cuh"

namespace {
constexpr int kBlocks = 296, kThreads = 256, kPerThread = 2000;

__device__ unsigned long long next(unsigned long long& s) {  // splitmix64
    s += 0x9E3779B97F4A7C15ull;
    unsigned long long z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ double operand(unsigned long long& s, int kind) {
    unsigned long long m = next(s) & 0xfffffffffffffull;
    if (kind == 0) m |= 0xfffffffffff00ull;  // just below a power of two
    if (kind == 1) m &= 0xff;                // just above one
    const unsigned long long e = 1023 - 390 + next(s) % 780;
    return __longlong_as_double((long long)(m | (e << 52)));
}

__global__ void check(unsigned long long* bad) {
    unsigned long long s = (blockIdx.x * (unsigned long long)kThreads + threadIdx.x) * 1000003ull + 7;
    unsigned long long n[3] = {0, 0, 0};
    for (int i = 0; i < kPerThread; ++i) {
        const double x = operand(s, i & 3), a = operand(s, 2);
        const double b = (next(s) & 1) ? -x : x;
        if (!lica::rn::ordinary(b)) continue;
        const double y = lica::rn::recip(b), q = lica::rn::quot(a, b, y);
        bool ok = true;
        const double r = lica::rn::root(x, ok);
        n[0] += __double_as_longlong(y) != __double_as_longlong(1.0 / b);
        n[1] += __double_as_longlong(q) != __double_as_longlong(a / b);
        n[2] += ok && __double_as_longlong(r) != __double_as_longlong(sqrt(x));
    }
    for (int k = 0; k < 3; ++k) atomicAdd(bad + k, n[k]);
}
}  // namespace

int main() {
    unsigned long long *d = nullptr, h[3] = {1, 1, 1};
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 2;
    check<<<kBlocks, kThreads>>>(d);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("%llu %llu %llu\n", h[0], h[1], h[2]);
    return 0;
}
