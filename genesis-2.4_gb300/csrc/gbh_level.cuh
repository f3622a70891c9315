// gbh_level.cuh -- level elimination: the device side of the kernels that
// gbh_jit.cu generates for trees whose dendrites are passive
// (TileType::level).
//
// The stack kernels give each neuron one lane, which walks its rows one
// after another: a step lasts as long as the longest neuron's chain (about
// 900 clocks a row), however few neurons there are. Rows below the first
// compartment with channels (TileType::nstatic) keep their diagonal D', its
// reciprocal and their coupling factor T from step to step, so what is left
// of them is one right-hand side each way, and rows at the same depth do not
// depend on each other. Here a block owns a group of neurons of one tile; its
// sweeping warps take all their static rows depth by depth, whatever neuron
// they belong to: forward from the deepest, a row pulls its children's
// R T in ascending row order, backward from the top, a row reads its parent's
// solution. One more warp (one neuron per lane) meanwhile runs the channel
// program and the pools of the rows above the static ones, finishes their
// elimination once the static rows below them are done, and starts on the
// next step's channels while the sweeping warps substitute back. The
// operations per row and their order are the sequential sweep's
// (hines_solve.c:223-296), so FP64 results keep the reference's bits.
//
// Rows are stored in level order (depth, then parent), so a level's loads are
// contiguous and a row's children sit side by side. R and the solution stay
// in shared memory for all steps of a launch; per row and step the kernel
// reads K, T, C, 1/D' and (FP64) D' and two indices, 48 bytes (40 mixed),
// against 78 from the stack kernels, several levels ahead of their use.
#pragma once
#include "gbh_devfn.cuh"

namespace gbh {

// A block's share of a tile: lanes [lane0, lane0 + nlanes), their static rows
// at elements [eoff, eoff + n) of the level-ordered arrays, in nch chunks of
// at most blockDim - 32 rows (first row, rows | LV_FIRST | LV_LAST).
struct LevelGroup {
    int tile, lane0, nlanes, n, nch, choff;
    int kidoff;      // the top rows' first static children: topkid[kidoff + s * 32 + lane]
    int pad;
    int64_t eoff;
};

// First and last chunk of a level: the forward sweep (descending) ends a
// level at its first chunk, the backward one (ascending) at its last.
constexpr int LV_FIRST = 1 << 30, LV_LAST = 1 << 29, LV_COUNT = (1 << 29) - 1;
// Children of a row: index of the first one, and their number above this bit.
constexpr int LV_KID_BITS = 20;

struct LevelView {
    const LevelGroup *groups;
    const int2 *chunks;
    const int *map;      // row * 32 + lane within the tile
    const int *kid;      // static children: first | number << LV_KID_BITS
    const int *par;      // parent's solution: top row * 32 + lane of the group, or ntop * 32 + its element
    const int *topkid;
    double2 *kt;         // rhs term K, coupling factor T = A / D'
    double2 *cy;         // backward coefficient C, 1 / D'
    double *d;           // D' (FP64 form)
    double *pd;          // B T: what the row takes from its parent's diagonal
    unsigned *gen;       // per group: the fields' generation its factors were kept at (DevView::sgen)
};

// Shared doubles of a group: the top rows' solutions, R / solutions, the
// contributions R T and, under Crank-Nicolson, Vm; then its chunks.
__host__ __device__ inline size_t level_smem(int ntop, int n, int nch, bool crank)
{
    return sizeof(double) * ((size_t)ntop * LANES + (size_t)n * (crank ? 3 : 2)) + sizeof(int2) * (size_t)nch;
}

// Named barriers of a block: 1 the sweeping warps, 2 the static rows are
// eliminated, 3 the top rows are solved.
enum LevelBar { LB_SWEEP = 1, LB_FORWARD = 2, LB_TOP = 3 };

#ifdef __CUDACC__
// What the sweeping warps of a block do in a launch. sm: level_smem bytes.
template <bool MIXED, bool CRANK, int NTOP>
__device__ __forceinline__ void level_sweep(const DevView &v, const LevelView &L, const LevelGroup &g, const Tile &tl,
                                            const TileType &ty, double *sm, int nsteps, bool full, bool refresh)
{
    const int tid = threadIdx.x, nt = blockDim.x - LANES, nth = blockDim.x;
    double *U = sm;                       // top rows' solutions, then the static rows' R / solution
    double *X = U + NTOP * LANES;
    double *PR = X + g.n;
    double *O = CRANK ? PR + g.n : X;     // Vm
    int2 *ch = reinterpret_cast<int2 *>(PR + g.n * (CRANK ? 2 : 1));
    const int nch = g.nch;
    const int *map = L.map + g.eoff, *kid = L.kid + g.eoff, *par = L.par + g.eoff;
    double2 *kt = L.kt + g.eoff, *cy = L.cy + g.eoff;
    double *dd = L.d + g.eoff, *pd = L.pd + g.eoff;
    double *V = v.V + tl.vm * LANES;
    for (int c = tid; c < nch; c += nt) ch[c] = L.chunks[g.choff + c];
    for (int e = tid; e < g.n; e += nt) O[e] = V[map[e]];
    bar_named(LB_SWEEP, nt);
    // a row's rhs term from its fields, as its channel program forms it
    const int *pf = v.prog + ty.pf_off;
    const double *P = v.P + tl.fld * LANES;
    auto kterm = [&](int m) {
        const int *ps = pf + 6 * (m / LANES);
        const int l = m % LANES;
        if (MIXED)
            return df2d(df_mul(df_add(ld_df(&P[ps[2] * LANES + l]), ld_df(&P[ps[3] * LANES + l])),
                               ld_df(&P[ps[4] * LANES + l])));
        return (P[ps[2] * LANES + l] + P[ps[3] * LANES + l]) * P[ps[4] * LANES + l];
    };
    if (full) {
        // the factors from the fields: the diagonals' elimination, level by
        // level; PR holds B T meanwhile
        const double *A = v.A + tl.topo * LANES, *B = v.B + tl.topo * LANES;
        for (int c = nch - 1; c >= 0; --c) {
            const int2 m = ch[c];
            if (tid < (m.y & LV_COUNT)) {
                const int e = m.x + tid, r = map[e], l = r % LANES;
                const int *ps = pf + 6 * (r / LANES);
                double D;
                if (MIXED) D = df2d(ld_df(&P[ps[5] * LANES + l]));
                else D = 0.0 * P[ps[4] * LANES + l] + P[ps[5] * LANES + l];
                const int k0 = kid[e] & ((1 << LV_KID_BITS) - 1), nk = (unsigned)kid[e] >> LV_KID_BITS;
                for (int k = 0; k < nk; ++k) D -= PR[k0 + k];
                const double y = MIXED ? rcp_newton(D) : 1.0 / D;   // FP64: correctly rounded
                const double T = MIXED ? A[r] * y : A[r] / D;
                const double b = B[r] * T;
                PR[e] = b;
                pd[e] = b;
                kt[e] = make_double2(kterm(r), T);
                cy[e].y = y;
                if (!MIXED) dd[e] = D;
            }
            if (m.y & LV_FIRST) bar_named(LB_SWEEP, nt);
        }
    } else if (refresh) {   // inputs on the rhs fields: their terms once per launch
        for (int e = tid; e < g.n; e += nt) kt[e].x = kterm(map[e]);
    }
    __threadfence_block();
    bar_named(LB_SWEEP, nt);
    // Row data is loaded PF chunks ahead, across the barriers between levels:
    // the loads (L2: some 300 clocks) would otherwise follow each barrier.
    constexpr int PF = 4;
    struct Fw { double2 kt; int kid; } fw[PF];
    struct Bw { double2 cy; double d; int par; } bw[PF];
    auto ldf = [&](Fw &q, int c) {
        if (c < 0) return;
        const int2 m = ch[c];
        if (tid < (m.y & LV_COUNT)) {
            q.kt = kt[m.x + tid];
            q.kid = __ldg(&kid[m.x + tid]);
        }
    };
    auto ldb = [&](Bw &q, int c) {
        if (c >= nch) return;
        const int2 m = ch[c];
        if (tid < (m.y & LV_COUNT)) {
            q.cy = cy[m.x + tid];
            if (!MIXED) q.d = dd[m.x + tid];
            q.par = __ldg(&par[m.x + tid]);
        }
    };
#pragma unroll
    for (int u = 0; u < PF; ++u) ldf(fw[u], nch - 1 - u);
    for (int it = 0; it < nsteps; ++it) {
        for (int c0 = nch - 1; c0 >= 0; c0 -= PF) {
#pragma unroll
            for (int u = 0; u < PF; ++u) {
                const int c = c0 - u;
                if (c < 0) break;
                const int2 m = ch[c];
                if (tid < (m.y & LV_COUNT)) {
                    const int e = m.x + tid;
                    const int k0 = fw[u].kid & ((1 << LV_KID_BITS) - 1), nk = (unsigned)fw[u].kid >> LV_KID_BITS;
                    double R = O[e] + fw[u].kt.x;
                    for (int k = 0; k < nk; ++k) R -= PR[k0 + k];
                    X[e] = R;
                    PR[e] = R * fw[u].kt.y;
                }
                ldf(fw[u], c - PF);
                if ((m.y & LV_FIRST) && c > 0) bar_named(LB_SWEEP, nt);
            }
        }
#pragma unroll
        for (int u = 0; u < PF; ++u) ldb(bw[u], u);
        bar_named(LB_FORWARD, nth);
        bar_named(LB_TOP, nth);
        for (int c0 = 0; c0 < nch; c0 += PF) {
#pragma unroll
            for (int u = 0; u < PF; ++u) {
                const int c = c0 + u;
                if (c >= nch) break;
                const int2 m = ch[c];
                if (tid < (m.y & LV_COUNT)) {
                    const int e = m.x + tid;
                    const double xp = U[bw[u].par], y = bw[u].cy.y;
                    double r;
                    if (MIXED) {
                        r = fma(-bw[u].cy.x, xp, X[e]) * y;
                    } else {
                        // RN(r / D') from the correctly rounded y = 1/D' by
                        // Markstein's correction, the division's bits
                        r = X[e] - bw[u].cy.x * xp;
                        const double q = r * y;
                        r = fma(fma(-bw[u].d, q, r), y, q);
                    }
                    X[e] = r;
                    if (CRANK) O[e] = MIXED ? fma(2.0, r, -O[e]) : r + r - O[e];
                }
                ldb(bw[u], c + PF);
                if (m.y & LV_LAST) bar_named(LB_SWEEP, nt);
            }
        }
        if (it + 1 < nsteps) {
#pragma unroll
            for (int u = 0; u < PF; ++u) ldf(fw[u], nch - 1 - u);
        }
    }
    for (int e = tid; e < g.n; e += nt) V[map[e]] = O[e];
}

// The static children of top row s of this lane: their contributions off
// (R, D), in ascending row order.
__device__ __forceinline__ void level_top_kids(const LevelView &L, const LevelGroup &g, const double *PR, int s,
                                               int lane, double &R, double &D)
{
    const int kk = L.topkid[g.kidoff + s * LANES + lane];
    const int k0 = kk & ((1 << LV_KID_BITS) - 1), nk = (unsigned)kk >> LV_KID_BITS;
    for (int k = 0; k < nk; ++k) {
        D -= L.pd[g.eoff + k0 + k];
        R -= PR[k0 + k];
    }
}
#endif

}  // namespace gbh
