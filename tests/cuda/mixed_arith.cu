// Test program: the mixed form's reciprocal and double-float to double
// conversion (gbh_df.cuh) against the FP64 operations they stand for. Prints
// "name count" lines: worst difference in units in the last place (step),
// differing results (convert), and the worst errors of 1/b in units of 2^-53
// (of the FP64 step: step64; of rcp_step: step_int).
#include <cstdio>
#include <cstdint>

#include <cuda_runtime.h>

#include "gbh_df.cuh"

using namespace gbh;

__device__ uint64_t rnd(uint64_t &s)
{
    s += 0x9e3779b97f4a7c15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

enum { STEP, CONVERT, STEP64, STEP_INT, N };

__global__ void k_check(unsigned long long *bad, int rounds, uint64_t seed)
{
    uint64_t s = seed + 0x1234567ull * (blockIdx.x * blockDim.x + threadIdx.x);
    unsigned long long b[N] = {};
    for (int i = 0; i < rounds; ++i) {
        // divisors: significands at random, of few bits, just above a power of two and some way below one
        const uint64_t r = rnd(s);
        uint64_t m = rnd(s) & 0xfffffffffffffull;
        if ((r & 7) == 1) m = 0xffffffffff000ull - (m & 0xffffff000ull);
        if ((r & 7) == 2) m &= 0xff;
        if ((r & 7) == 3) m &= 0xffffff0000000ull;
        const int e = (int)((r >> 8) % 121) - 60;
        const double x = __longlong_as_double((long long)((r >> 63) << 63 | (uint64_t)(1023 + e) << 52 | m));
        const double m1 = __longlong_as_double((long long)(1023ull << 52 | m));
        const double r0 = (double)rcp_approx(__double2float_rz(m1));
        const double want = ldexp(fma(r0, fma(-m1, r0, 1.0), r0), -e) * (x < 0 ? -1.0 : 1.0), got = rcp_step(x);
        const long long d = __double_as_longlong(got) - __double_as_longlong(want);
        const unsigned long long ad = (unsigned long long)(d < 0 ? -d : d);
        if (ad > b[STEP]) b[STEP] = ad;
        // 1/b to well beyond FP64: q + fma(-b, q, 1) / b
        const double q = 1.0 / x, rest = fma(-x, q, 1.0) / x;
        const double e64 = fabs(((want - q) - rest) * x) * 0x1p53, ei = fabs(((got - q) - rest) * x) * 0x1p53;
        if (e64 > (double)b[STEP64]) b[STEP64] = (unsigned long long)ceil(e64);
        if (ei > (double)b[STEP_INT]) b[STEP_INT] = (unsigned long long)ceil(ei);
        // conversions: rounded pairs, truncated pairs, ties, powers of two, far-off and denormal parts
        const uint64_t k = rnd(s);
        float hi = __uint_as_float((uint32_t)(k >> 63) << 31 | (uint32_t)(27 + (k >> 8) % 200) << 23 | ((uint32_t)k & 0x7fffffu));
        if (k >> 60 == 1) hi = __uint_as_float(__float_as_uint(hi) & 0xff800000u);
        if (k >> 60 == 2) hi = __uint_as_float(__float_as_uint(hi) | 0x7fffffu);
        const uint64_t kl = rnd(s);
        const float unit = ldexpf(1.0f, (int)(__float_as_uint(hi) >> 23 & 0xffu) - 127 - 23);
        float lo = 0.5f * unit * (float)((int32_t)(kl & 0xffffffu) - 0x800000) * 0x1p-23f;   // up to half a unit
        switch (kl >> 61) {
        case 1: lo = __uint_as_float((__float_as_uint(hi) & 0x80000000u) |
                                     (__float_as_uint(unit * ((float)(kl & 0xffffffu) * 0x1p-24f)) & 0x7fffffffu)); break;
        case 2: lo = ldexpf(lo, -(int)(kl >> 40 & 31)); break;
        case 3: lo = unit * 0x1p-29f * (float)((int)(kl & 0xff) - 128) * 0.5f; break;        // ties
        case 4: lo = unit * 0x1p-30f * (float)((int)(kl & 0xff) - 128) * 0.5f; break;
        case 5: lo = ldexpf(lo, -60); break;
        default: break;
        }
        if (hi < 0.0f ? lo > 0.0f : lo < 0.0f)   // taken off a power of two: half a unit below it
            if ((__float_as_uint(hi) & 0x7fffffu) == 0u) lo *= 0.5f;
        const double a = df2d(df_make(hi, lo)), c = (double)hi + (double)lo;
        b[CONVERT] += __double_as_longlong(a) != __double_as_longlong(c);
    }
    for (int j = 0; j < N; ++j)
        if (j == CONVERT) atomicAdd(&bad[j], b[j]);
        else atomicMax(&bad[j], b[j]);
}

int main()
{
    unsigned long long *bad, h[N];
    if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, sizeof(h));
    k_check<<<152 * 4, 128>>>(bad, 400, 42);
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    const char *name[N] = {"step", "convert", "step64", "step_int"};
    for (int j = 0; j < N; ++j) printf("%s %llu\n", name[j], h[j]);
    return 0;
}
