// Test program: rcp_exact (gbh_df.cuh) against CUDA's IEEE reciprocal. The
// listed significands b (53 bits) are factors of 2^106 + d for odd |d| < 4000
// with an odd cofactor: 1/b lies |d| 2^-106 from the middle between two
// doubles, closer than one Newton step from a seed of 2^-44 can tell. Prints
// mismatches over them and over random divisors, and how many of the listed
// ones rcp_rn gets wrong.
#include <cstdio>
#include <cstdint>

#include <cuda_runtime.h>

#include "gbh_df.cuh"

using namespace gbh;

__constant__ uint64_t hard[] = {
    0x1fffffffffffffull, 0x113deff6b41e35ull, 0x161c2909f39d4bull, 0x1ef43974550f69ull, 0x1ffffffffffffdull,
    0x1ffffffffffffbull, 0x180c93418865f3ull, 0x1700e376062ff1ull, 0x11976638062c3bull, 0x1333333333332full,
    0x1ffffffffffff9ull, 0x16637886414bf5ull, 0x1dbd322fc7846dull, 0x1483dd28a8316bull, 0x1c26fd6f539f95ull,
    0x1ffffffffffff7ull, 0x1c0264cb705aa5ull, 0x13d0b472b17883ull, 0x1139cd2c153191ull, 0x111f8ea9cee249ull,
    0x1c69b03bcac893ull, 0x1af6d7d37db0d7ull, 0x120b0ebf324b0dull, 0x1ffffffffffff5ull, 0x1ffffff8000001ull,
    0x1334adfe7a8ddbull, 0x1455036bcb0d11ull, 0x1f3829c8f1083dull, 0x1949e500b130afull, 0x1ab3b42708104full,
    0x1825540e9a11a3ull, 0x1cc06693a79a71ull, 0x17466b6b56eabdull, 0x1dd3c23027bb6full, 0x175585181cadc5ull,
    0x1f0b6c12c616adull};
constexpr int NHARD = sizeof(hard) / sizeof(hard[0]);

__global__ void k_check(unsigned long long *bad, int rounds)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t s = 0x9e3779b97f4a7c15ull * (uint64_t)(id + 1);
    auto differs = [](double a, double b) { return __double_as_longlong(a) != __double_as_longlong(b); };
    if (id < 2 * NHARD) {
        const double b = (id < NHARD ? 1.0 : -0x1p-37) * (double)hard[id % NHARD];
        if (differs(rcp_exact(b), __drcp_rn(b))) atomicAdd(&bad[0], 1ull);
        if (differs(rcp_rn(b), __drcp_rn(b))) atomicAdd(&bad[2], 1ull);
    }
    unsigned long long n = 0;
    for (int i = 0; i < rounds; ++i) {
        s ^= s << 13;
        s ^= s >> 7;
        s ^= s << 17;
        const double b = __longlong_as_double((long long)((s & 0x800fffffffffffffull) | (uint64_t)(963 + s % 121) << 52));
        n += differs(rcp_exact(b), __drcp_rn(b));
    }
    if (n) atomicAdd(&bad[1], n);
}

int main()
{
    unsigned long long *bad, h[3];
    if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, sizeof(h));
    k_check<<<152 * 4, 128>>>(bad, 400);
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    printf("hard %llu\nrandom %llu\nrcp_rn %llu\n", h[0], h[1], h[2]);
    return 0;
}
