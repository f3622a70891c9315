// Test program: the kernels' integer- and FP32-assisted FP64 arithmetic
// (gbh_df.cuh, gbh_devfn.cuh) against CUDA's IEEE operations. Prints
// "name count" lines: mismatches (bits) or, for the approximations, the worst
// error in units of 2^-53.
#include <cstdio>
#include <cstdint>

#include <cuda_runtime.h>

#include "gbh_devfn.cuh"

using namespace gbh;

__device__ uint64_t rnd(uint64_t &s)
{
    s += 0x9e3779b97f4a7c15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// significands next to powers of two, of few bits and at random; exponents within +-range
__device__ double pick(uint64_t &s, int range)
{
    const uint64_t r = rnd(s);
    uint64_t m = rnd(s) & 0xfffffffffffffull;
    if ((r & 7) == 1) m = 0xfffffffffffffull - (m & 0xff);
    if ((r & 7) == 2) m &= 0xff;
    if ((r & 7) == 3) m &= 0xffffff0000000ull;
    const uint64_t e = 1023 + (int64_t)((r >> 8) % (2 * range + 1)) - range;
    return __longlong_as_double((long long)((r >> 63) << 63 | e << 52 | m));
}

__device__ bool differ(double a, double b)
{
    return a != a ? b == b : __double_as_longlong(a) != __double_as_longlong(b);
}

enum { DIV, RCP, SPECIAL, KEY, ROW, SEED, STEP, DF, VOLT, N };

__global__ void k_check(unsigned long long *bad, int rounds, uint64_t seed, const double *special, int nspecial)
{
    uint64_t s = seed + 0x1234567ull * (blockIdx.x * blockDim.x + threadIdx.x);
    unsigned long long b[N] = {};
    for (int i = 0; i < rounds; ++i) {
        const double x = pick(s, 60), y = pick(s, 60);
        b[DIV] += differ(div_rn(x, y), __ddiv_rn(x, y));
        b[RCP] += differ(rcp_rn(y), __drcp_rn(y));
        // every pair of special operands, and specials against ordinary ones
        const double p = special[rnd(s) % nspecial], q = special[rnd(s) % nspecial];
        b[SPECIAL] += differ(div_rn(p, q), __ddiv_rn(p, q)) + differ(div_rn(p, y), __ddiv_rn(p, y)) +
                      differ(div_rn(x, q), __ddiv_rn(x, q)) + differ(rcp_rn(q), __drcp_rn(q));
        b[KEY] += (dkey(p) < dkey(q)) != (p < q) && p == p && q == q;
        b[KEY] += (dkey(x) < dkey(y)) != (x < y);
        // table rows: positions inside, outside and on the edges of a table of `divs` rows
        const int divs = 1 + (int)(rnd(s) % 5000);
        const uint64_t k = rnd(s);
        double f = (double)(int64_t)(k % 0x3fffffffffffffull) * 0x1p-54 * 1.2 * divs - 0.1 * divs;
        if ((k >> 60) == 1) f = (double)(int)(rnd(s) % (divs + 1));
        if ((k >> 60) == 2) f = nextafter((double)(int)(rnd(s) % (divs + 1)), (k & 1) ? 1e9 : -1e9);
        if ((k >> 60) == 3) f = x;
        VCursor c;
        const double d = divs;
        double g = f, ref = f;
        locate_row(c, g, divs, (unsigned)__double2hiint(d));
        if (ref < 0.0) ref = 0.0;
        else if (ref > divs) ref = divs;
        const int row = (int)ref;
        b[ROW] += c.row != row || c.rowd != (double)row || g - c.rowd != ref - (double)row;
        // approximations, relative error in units of 2^-53
        // (the seed: against the same Newton step in FP64 from the same float)
        const double ay = fabs(y), m1 = __hiloint2double((__double2hiint(ay) & 0xfffff) | 0x3ff00000, __double2loint(ay));
        const double r0 = (double)rcp_approx(__double2float_rz(m1)), r1 = fma(r0, fma(-m1, r0, 1.0), r0);
        const double e = fabs(rcp_seed(m1) / r1 - 1.0) * 0x1p53 + (rcp_seed(y) * m1 / ay * (y < 0 ? -1 : 1) < 0 ? 1e9 : 0);
        if (e > (double)b[SEED]) b[SEED] = (unsigned long long)ceil(e);
        const double es = fabs(rcp_step(m1) / r1 - 1.0) * 0x1p53 + (rcp_step(y) * m1 / ay * (y < 0 ? -1 : 1) < 0 ? 1e9 : 0);
        if (es > (double)b[STEP]) b[STEP] = (unsigned long long)ceil(es);
        const double v = pick(s, 100);
        float hi = (float)v, lo = (float)(v - (double)hi);
        if (i & 1) {   // a significand that ends in hi, lo far below or taken off a power of two
            lo = (rnd(s) & 1) ? -hi * 0x1p-25f : hi * 0x1p-40f;
        }
        const double exact = (double)hi + (double)lo;
        const double er = fabs((df2d(df_make(hi, lo)) - exact) / exact) * 0x1p53;
        const df w = d2df_volt(v), u = d2df(v);
        b[VOLT] += fabs(v) > 0x1p-70 && (w.hi != u.hi || w.lo != u.lo);
        b[SPECIAL] += isfinite(p) ? 0 : !(fabs((double)d2df_volt(p).hi) > 1e38);
        if (er > (double)b[DF]) b[DF] = (unsigned long long)ceil(er);
    }
    for (int j = 0; j < N; ++j)
        if (j == SEED || j == STEP || j == DF) atomicMax(&bad[j], b[j]);
        else atomicAdd(&bad[j], b[j]);
}

int main()
{
    const double inf = 1.0 / 0.0, nan = inf - inf;
    const double sp[] = {0.0, -0.0, 1.0, -1.0, inf, -inf, nan, 0x1p-1074, -0x1p-1022, 0x1.fffffffffffffp1023,
                         0x1p-460, 0x1p460, 0x1p450, 0x1p-450, 0x1p451, 0x1.fffffffffffffp0, 3.0, -0x1p-1050};
    unsigned long long *bad, h[N];
    double *dsp;
    if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess || cudaMalloc(&dsp, sizeof(sp)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, sizeof(h));
    cudaMemcpy(dsp, sp, sizeof(sp), cudaMemcpyHostToDevice);
    const int blocks = 152 * 4, threads = 128, rounds = 400;
    k_check<<<blocks, threads>>>(bad, rounds, 42, dsp, (int)(sizeof(sp) / sizeof(sp[0])));
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    const char *name[N] = {"div", "rcp", "special", "key", "row", "seed", "step", "df", "volt"};
    for (int j = 0; j < N; ++j) printf("%s %llu\n", name[j], h[j]);
    return 0;
}
