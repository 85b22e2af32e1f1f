// Device-side check of r_mod (ctd_arith.cuh): reads moduli, prints 2^64 mod each.
#include <cinttypes>
#include <cstdio>
#include <vector>

#include "../cutrialdive_gb300/csrc/ctd_arith.cuh"

__global__ void remainders(const uint64_t *p, uint64_t *r, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        r[i] = ctd::r_mod(p[i]);
}

int main()
{
    std::vector<uint64_t> p;
    for (unsigned long long x; std::scanf("%llu", &x) == 1;)
        p.push_back(x);
    const uint32_t n = (uint32_t)p.size();
    uint64_t *d = nullptr;
    if (!n || cudaMalloc(&d, 2 * n * sizeof(uint64_t)) != cudaSuccess)
        return 1;
    cudaMemcpy(d, p.data(), n * sizeof(uint64_t), cudaMemcpyHostToDevice);
    remainders<<<(n + 255) / 256, 256>>>(d, d + n, n);
    if (cudaMemcpy(p.data(), d + n, n * sizeof(uint64_t), cudaMemcpyDeviceToHost) != cudaSuccess)
        return 1;
    for (uint64_t r : p)
        std::printf("%" PRIu64 "\n", r);
    return 0;
}
