// stretch.cu -- sampled stretch limits on the device.
//
// getstretch (simulator.cu:802-822) sums twelve values of rand() per particle
// after srand(1973) (simulator.cu:852): 12 n steps of one serial generator, which
// take the host 12 ms at 1M particles.  The generator (glibc_rand.h) is linear
// modulo 2^32, h[i] = h[i-31] + h[i-3], so word i + s is a fixed combination of
// the words i .. i+30, with the coefficients of x^s modulo x^31 - x^28 - 1.  Every
// thread jumps to its own kRun particles with the polynomial of its place in the
// block and the block's first words, and runs the generator from there: the same
// words, and the same sums in the same order.  Latency-bound, 48 us for bodies of
// 4k to 24k particles (150 with the FP64 division and 16 particles per thread);
// make_ready of 1M particles takes 35.6 ms instead of 46.6.
#include <cstdint>
#include <vector>

#include "glibc_rand.h"
#include "pd_device.cuh"
#include "pd_kernels.h"

namespace pdgb {

namespace {

constexpr int kWords = 31;                 // state
constexpr int kReach = 2 * kWords - 1;     // words that the combinations of a block read
constexpr int kDraws = 12;                 // values per particle
constexpr int kRun = 8;                    // particles per thread
constexpr int kStretchThreads = 256;
constexpr int kPerBlock = kRun * kStretchThreads;

struct Poly {
    uint32_t c[kWords];
};

// a b modulo x^31 - x^28 - 1, coefficients modulo 2^32
Poly multiply(const Poly& a, const Poly& b)
{
    uint32_t w[kReach] = {};
    for (int i = 0; i < kWords; ++i)
        for (int j = 0; j < kWords; ++j) w[i + j] += a.c[i] * b.c[j];
    for (int d = kReach - 1; d >= kWords; --d) {
        w[d - 3] += w[d];
        w[d - kWords] += w[d];
    }
    Poly r;
    for (int i = 0; i < kWords; ++i) r.c[i] = w[i];
    return r;
}

Poly power_of_x(unsigned e)
{
    Poly r{}, x{};
    r.c[0] = 1;
    x.c[1] = 1;
    for (; e; e >>= 1) {
        if (e & 1) r = multiply(r, x);
        x = multiply(x, x);
    }
    return r;
}

// a / (2^31 - 1), correctly rounded: the product with the rounded reciprocal and one
// correction by the exact remainder (Markstein, IBM J. Res. Dev. 34, 1990);
// equal to the division for every a in 0 .. 2^31 - 1 (all of them compared on
// the CPU).  The division's own chain is 573 cycles.
__device__ __forceinline__ double by_rand_max(double a)
{
    constexpr double b = 2147483647.0, y = 1.0 / b;
    const double q = dmul(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

// jump: coefficient k of thread t's polynomial at [k * kStretchThreads + t]
__global__ void __launch_bounds__(kStretchThreads)
    k_stretch(const uint32_t* __restrict__ jump, const uint32_t* __restrict__ first, int n, double s0,
              double* __restrict__ out)
{
    __shared__ uint32_t base[kReach];
    __shared__ uint32_t ring[kWords][kStretchThreads];
    const int t = threadIdx.x;
    if (t < kReach) base[t] = first[(size_t)blockIdx.x * kReach + t];
    __syncthreads();
    uint32_t w[kWords];
#pragma unroll
    for (int j = 0; j < kWords; ++j) w[j] = 0u;
    for (int k = 0; k < kWords; ++k) {
        const uint32_t c = __ldg(jump + k * kStretchThreads + t);
#pragma unroll
        for (int j = 0; j < kWords; ++j) w[j] += c * base[k + j];
    }
#pragma unroll
    for (int j = 0; j < kWords; ++j) ring[j][t] = w[j];
    const long long p0 = (long long)blockIdx.x * kPerBlock + (long long)t * kRun;
    int at = 0;
    for (int q = 0; q < kRun && p0 + q < n; ++q) {
        double sum = 0.0;
#pragma unroll
        for (int d = 0; d < kDraws; ++d) {
            const int near = at < 3 ? at + kWords - 3 : at - 3;
            const uint32_t v = ring[at][t] + ring[near][t];
            ring[at][t] = v;
            at = at == kWords - 1 ? 0 : at + 1;
            sum = dadd(sum, by_rand_max((double)(int)(v >> 1)));
        }
        sum = dsub(sum, 6.0);
        out[p0 + q] = dmul(dadd(dmul(sum, 0.01), 1.0), s0);
    }
}

}  // namespace

cudaError_t sample_stretch_limits(float s0, int n, double* out, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const int blocks = (n + kPerBlock - 1) / kPerBlock;
    std::vector<uint32_t> h((size_t)kWords * kStretchThreads + (size_t)blocks * kReach);
    const Poly step = power_of_x(kDraws * kRun), block = power_of_x(kDraws * kPerBlock);
    Poly p = power_of_x(0);
    for (int t = 0; t < kStretchThreads; ++t) {
        for (int k = 0; k < kWords; ++k) h[(size_t)k * kStretchThreads + t] = p.c[k];
        p = multiply(p, step);
    }
    // the last 31 words before the first value, and each block's
    GlibcRand gen(1973);
    uint32_t w[kReach];
    for (int k = 0; k < kWords; ++k) w[k] = gen.at(gen.i - kWords + k);
    for (int b = 0; b < blocks; ++b) {
        for (int k = kWords; k < kReach; ++k) w[k] = w[k - kWords] + w[k - 3];
        for (int k = 0; k < kReach; ++k) h[(size_t)kWords * kStretchThreads + (size_t)b * kReach + k] = w[k];
        uint32_t next[kWords];
        for (int j = 0; j < kWords; ++j) {
            next[j] = 0u;
            for (int k = 0; k < kWords; ++k) next[j] += block.c[k] * w[k + j];
        }
        for (int j = 0; j < kWords; ++j) w[j] = next[j];
    }
    uint32_t* d = nullptr;
    cudaError_t e = cudaMalloc((void**)&d, sizeof(uint32_t) * h.size());
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(d, h.data(), sizeof(uint32_t) * h.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        k_stretch<<<blocks, kStretchThreads, 0, st>>>(d, d + (size_t)kWords * kStretchThreads, n, (double)s0, out);
        e = cudaGetLastError();
    }
    const cudaError_t f = cudaFree(d);   // (waits for the kernel)
    return e != cudaSuccess ? e : f;
}

}  // namespace pdgb
