// Device loops over the arguments of the fast routines of hw_device.cuh that
// stand for a general one: each counts the arguments where the bits differ.
#include "../hw_b200/csrc/hw_device.cuh"

using namespace hwk;

namespace {

__device__ bool Same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// hw_expf_fast and both components of hw_expf2_fast against hw_expf, every
// float of the bit patterns [first, last].
__global__ void ExpKernel(uint32_t first, uint32_t last, float negZero, unsigned long long* bad)
{
    unsigned long long n = 0;
    for (uint64_t b = (uint64_t)first + blockIdx.x * blockDim.x + threadIdx.x; b <= last; b += (uint64_t)gridDim.x * blockDim.x)
    {
        const float x = __uint_as_float((uint32_t)b), want = hw_expf(x);
        const float2 two = hw_expf2_fast(f2(x, x), f2(negZero));
        n += !Same(hw_expf_fast(x), want) | !Same(two.x, want) | !Same(two.y, want);
    }
    if (n) atomicAdd(bad, n);
}

__global__ void LogKernel(uint32_t first, uint32_t last, unsigned long long* bad)
{
    unsigned long long n = 0;
    for (uint64_t b = (uint64_t)first + blockIdx.x * blockDim.x + threadIdx.x; b <= last; b += (uint64_t)gridDim.x * blockDim.x)
    {
        const float x = __uint_as_float((uint32_t)b);
        n += !Same(hw_logf_normal(x), hw_logf(x));
    }
    if (n) atomicAdd(bad, n);
}

// The pulse fields' v / .1f.
__global__ void TenthKernel(uint32_t first, uint32_t last, unsigned long long* bad)
{
    unsigned long long n = 0;
    for (uint64_t b = (uint64_t)first + blockIdx.x * blockDim.x + threadIdx.x; b <= last; b += (uint64_t)gridDim.x * blockDim.x)
    {
        const float x = __uint_as_float((uint32_t)b);
        n += !Same(DivRcp(x, .1f, 10.0f), x / .1f);
    }
    if (n) atomicAdd(bad, n);
}

// Quotients as the histogram forms them: (value - lower) / binSize with bin
// sizes in (2^-40, 2^40) and lower bounds of 0 or magnitudes in (2^-40, 2^40).
__global__ void BinKernel(uint32_t count, unsigned long long* bad)
{
    unsigned long long n = 0;
    for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x)
    {
        uint64_t h = (i + 1) * 0x9e3779b97f4a7c15ull;      // splitmix64
        auto next = [&]() {
            h += 0x9e3779b97f4a7c15ull;
            uint64_t v = (h ^ (h >> 30)) * 0xbf58476d1ce4e5b9ull;
            v = (v ^ (v >> 27)) * 0x94d049bb133111ebull;
            return v ^ (v >> 31);
        };
        const uint64_t r = next(), s = next();
        const float binSize = __uint_as_float(((uint32_t)(88 + r % 79) << 23) | (uint32_t)((r >> 32) & 0x7fffff));
        const float mag = __uint_as_float(((uint32_t)(88 + s % 79) << 23) | (uint32_t)((s >> 32) & 0x7fffff));
        const float lower = (s >> 60) == 0 ? 0.0f : (s >> 59) & 1 ? -mag : mag;
        const float d = I16ToFloat((int16_t)(r >> 48)) - lower;
        n += !Same(DivRcp(d, binSize, 1.0f / binSize), d / binSize);
    }
    if (n) atomicAdd(bad, n);
}

}   // namespace

// counts[0..3]: differing arguments of the four sweeps; returns the CUDA status.
extern "C" int fast_math_sweep(unsigned long long* counts)
{
    unsigned long long* bad = nullptr;
    cudaError_t e = cudaMalloc((void**)&bad, 4 * sizeof(*bad));
    if (e == cudaSuccess) e = cudaMemset(bad, 0, 4 * sizeof(*bad));
    if (e != cudaSuccess) return (int)e;
    const int blocks = 148 * 8, threads = 256;
    ExpKernel<<<blocks, threads>>>(0u, 0x428c0000u, -0.0f, bad);                 // [0, 70]
    ExpKernel<<<blocks, threads>>>(0x80000000u, 0xff800000u, -0.0f, bad);        // [-inf, -0]
    LogKernel<<<blocks, threads>>>(0x00800000u, 0x7f7fffffu, bad + 1);           // positive normal
    TenthKernel<<<blocks, threads>>>(0x30000000u, 0x45cccd00u, bad + 2);         // [2^-31, 6553.6]
    TenthKernel<<<1, 32>>>(0u, 0u, bad + 2);
    BinKernel<<<blocks, threads>>>(1u << 30, bad + 3);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(counts, bad, 4 * sizeof(*bad), cudaMemcpyDeviceToHost);
    cudaFree(bad);
    return (int)e;
}
