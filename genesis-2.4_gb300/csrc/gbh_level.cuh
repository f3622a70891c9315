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
// contiguous and a row's children sit side by side. R, the solution and the
// rows' constants stay in shared memory for all steps of a launch (64 bytes a
// row in FP64, 56 mixed; 8 more under Crank-Nicolson); a neuron of more rows
// than fit keeps its constants in global memory.
#pragma once
#include "gbh_devfn.cuh"

namespace gbh {

// A block's share of a tile: lanes [lane0, lane0 + nlanes), their n static
// rows at elements eoff of the level-ordered arrays (LV_SPARE more behind
// them), in nch chunks of at most blockDim - 32 rows (first row, rows |
// CHUNK_FIRST | CHUNK_LAST; LV_GUARD empty ones before and behind them).
struct LevelGroup {
    int tile, lane0, nlanes, n, nch, choff;
    int kidoff;      // the top rows' static children: topkid[kidoff + s * 32 + lane]
    int many;        // some row has three children or more
    int64_t eoff;
};

// The sweeps read the descriptors two chunks ahead.
constexpr int LV_GUARD = 2;
// Spare elements behind a group's rows: a zero (what a row without children
// subtracts), and one that threads without a row work on, so that the sweeps
// run without branches.
constexpr int LV_SPARE = 2;
// A row's first two children (its spare zero where it has fewer) are packed
// 16 bits each; rows of a group are limited by that.
constexpr int LV_MAX_ROWS = 65000;
// A top row's static children: the first one and, above this bit, their number.
constexpr int LV_KID_BITS = 20;

struct LevelView {
    const LevelGroup *groups;
    const int2 *chunks;
    const int *map;      // row * 32 + lane within the tile
    const int *kid;      // first and second static child
    const int *nkid;     // number of static children, consecutive from the first
    const int *par;      // parent's solution: top row * 32 + lane of the group, or ntop * 32 + its element
    const int *topkid;
    double2 *kt;         // rhs term K, coupling factor T = A / D'
    double2 *cy;         // backward coefficient C (mixed: C / D'), 1 / D'
    const double *c;     // C
    double *d;           // D' (FP64 form)
    double *pd;          // B T: what the row takes from its parent's diagonal
    unsigned *gen;       // per group: the fields' generation its factors were kept at (DevView::sgen)
    const int *tin, *tout;   // per-step inputs and outputs (DevView::tin_*, tout_*): element of a static row, -1 others
    const int2 *io;      // per tile: any input (x) or output (y) of a static row
};

// Shared memory of a group's block, in the order level_smem_of lays it out:
// the constants (resident), the top rows' solutions, R / solutions, the
// contributions R T and, under Crank-Nicolson, Vm; D' (FP64), the chunks and
// the indices.
__host__ __device__ inline size_t level_smem(int ntop, int n, int nch, bool crank, bool mixed, bool resident)
{
    const size_t ns = (size_t)n + LV_SPARE;
    return 8 * ((size_t)ntop * LANES + ns * (crank ? 3 : 2)) + 8 * ((size_t)nch + 2 * LV_GUARD) +
           (resident ? ns * (mixed ? 40 : 48) : 0);
}

// Named barriers of a block: 1 the sweeping warps, 2 the static rows are
// eliminated, 3 the top rows are solved.
enum LevelBar { LB_SWEEP = 1, LB_FORWARD = 2, LB_TOP = 3 };

#ifdef __CUDACC__
// One block's arrays in shared memory.
struct LevelSm {
    double2 *kt, *cy;
    double *U, *X, *PR, *O, *d;
    int2 *ch;
    int *kid, *par;
};
template <bool MIXED, bool CRANK, int NTOP, bool RES>
__device__ __forceinline__ LevelSm level_smem_of(double *sm, const LevelGroup &g)
{
    LevelSm q;
    const int n = g.n + LV_SPARE;
    q.kt = reinterpret_cast<double2 *>(sm);
    q.cy = q.kt + n;
    q.U = sm + (RES ? 4 * n : 0);
    q.X = q.U + NTOP * LANES;
    q.PR = q.X + n;
    q.O = CRANK ? q.PR + n : q.X;
    q.d = q.PR + n * (CRANK ? 2 : 1);
    q.ch = reinterpret_cast<int2 *>(q.d + (RES && !MIXED ? n : 0)) + LV_GUARD;
    q.kid = reinterpret_cast<int *>(q.ch + g.nch + LV_GUARD);
    q.par = q.kid + n;
    return q;
}

// A static row's rhs term from its fields, as its channel program forms it
// (m: row * 32 + lane of the tile).
template <bool MIXED> __device__ __forceinline__ double level_kterm(const double *P, const int *pf, int m)
{
    const int *ps = pf + 6 * (m / LANES);
    const int l = m % LANES;
    if (MIXED)
        return df2d(df_mul(df_add(ld_df(&P[ps[2] * LANES + l]), ld_df(&P[ps[3] * LANES + l])),
                           ld_df(&P[ps[4] * LANES + l])));
    return (P[ps[2] * LANES + l] + P[ps[3] * LANES + l]) * P[ps[4] * LANES + l];
}

// A step's inputs into the fields of a group (lanes [lane0, lane0 + nlanes) of
// the tile) by `nt` threads: of its static rows, whose rhs terms in kt follow,
// or, kt null, of the rows above them.
template <bool MIXED>
__device__ __forceinline__ void level_in(const DevView &v, const LevelView &L, int tile, int lane0, int nlanes,
                                      int64_t eoff, long long step, int tid, int nt, double2 *kt)
{
    const Tile &tl = v.tiles[tile];
    const double *src = v.io_in + (step - v.io_step0) * v.io_nin;
    double *P = v.P + tl.fld * LANES;
    for (int k = v.tin_start[tile] + tid; k < v.tin_start[tile + 1]; k += nt) {
        const int at = v.tin_off[k], off = at & ~(1 << 30), l = off & (LANES - 1), e = L.tin[k];
        if ((e < 0) != (kt == nullptr) || l < lane0 || l >= lane0 + nlanes) continue;
        const double x = src[v.tin_idx[k]];
        if (at & (1 << 30)) {
            const float hi = __double2float_rn(x);
            st_df(&P[off], df_make(hi, __double2float_rn(x - (double)hi)));
        } else {
            P[off] = x;
        }
        if (kt) kt[e].x = level_kterm<MIXED>(P, v.prog + v.types[tl.type].pf_off, L.map[eoff + e]);
    }
}

// A step's outputs of a group: of its static rows from their solutions X, or, X
// null, of the rows above them, whose warp has stored their Vm.
__device__ __forceinline__ void level_out(const DevView &v, const LevelView &L, int tile, int lane0, int nlanes,
                                              long long step, int tid, int nt, const double *X)
{
    double *dst = v.io_out + (step - v.io_step0) * v.io_nout;
    const double *V = v.V + v.tiles[tile].vm * LANES;
    for (int k = v.tout_start[tile] + tid; k < v.tout_start[tile + 1]; k += nt) {
        const int off = v.tout_off[k], l = off & (LANES - 1), e = L.tout[k];
        if ((e < 0) != (X == nullptr) || l < lane0 || l >= lane0 + nlanes) continue;
        dst[v.tout_idx[k]] = X ? X[e] : V[off];
    }
}

// What the sweeping warps of a block do in a launch (sm: level_smem bytes).
// MANY: a row may have more than two static children. IO: per-step inputs and
// outputs, in a kernel of their own: with them the others' steps took up to
// 12 % longer (10 to 20 registers more a thread).
template <bool MIXED, bool CRANK, int NTOP, bool RES, bool IO, bool MANY>
__device__ __forceinline__ void level_steps(const DevView &v, const LevelView &L, const LevelGroup &g,
                                            const LevelSm &q, int nsteps, long long step0)
{
    const int tid = threadIdx.x, nt = blockDim.x - LANES, nth = blockDim.x;
    double *const U = q.U, *const X = q.X, *const PR = q.PR, *const O = q.O;
    const int2 *const ch = q.ch;
    const int nch = g.nch, spare = g.n + 1;   // see LV_SPARE
    const double2 *const kt = RES ? q.kt : L.kt + g.eoff, *const cy = RES ? q.cy : L.cy + g.eoff;
    const double *const dd = RES ? q.d : L.d + g.eoff;
    const int *const kid = RES ? q.kid : L.kid + g.eoff, *const par = RES ? q.par : L.par + g.eoff;
    // mixed: a parent subtracts R T in one multiply-add, T from its child's
    // constants; FP64: the child leaves R T in PR
    const double *const pulled = MIXED ? X : PR;
    auto element = [&](int2 m) { return tid < (m.y & CHUNK_COUNT) ? m.x + tid : spare; };
    auto busy = [&](int2 m) { return (tid & ~(LANES - 1)) < (m.y & CHUNK_COUNT); };   // a warp with rows
    auto sync = [&]() {
        if (nt == LANES) __syncwarp();
        else bar_named(LB_SWEEP, nt);
    };
    // The FP64 unit takes an instruction from a warp every 64 clocks, whatever
    // depends on it, so a level lasts as long as its instructions in a row;
    // what does not wait for the level before is read and formed meanwhile:
    // the next level's constants, its Vm + K forward and, mixed, R / D'
    // backward, and the descriptors two chunks ahead.
    const bool put = IO && v.io_in && L.io[g.tile].x, take = IO && v.io_out && L.io[g.tile].y;
    for (int it = 0; it < nsteps; ++it) {
        if (put) {
            level_in<MIXED>(v, L, g.tile, g.lane0, g.nlanes, g.eoff, step0 + it, tid, nt, RES ? q.kt : L.kt + g.eoff);
            if (!RES) __threadfence_block();
            sync();
        }
        int2 m = ch[nch - 1], mn = ch[nch - 2];
        int e = element(m), k = kid[e];
        double T = kt[e].y, own = O[e] + kt[e].x;
        for (int c = nch - 1; c >= 0; --c) {
            const int2 m2 = ch[c - 2];
            const int en = element(mn);
            int kn;
            double Tn, ownn;
            if (busy(m)) {
                const int i0 = k & 0xffff, i1 = (unsigned)k >> 16;
                const double c0 = pulled[i0], c1 = pulled[i1];
                double t0 = 0.0, t1 = 0.0;
                if (MIXED) {
                    t0 = kt[i0].y;
                    t1 = kt[i1].y;
                }
                const double2 a = kt[en];
                const double on = O[en];
                kn = kid[en];
                double R = MIXED ? fma(-c0, t0, own) : own - c0;
                R = MIXED ? fma(-c1, t1, R) : R - c1;
                if (MANY) {
                    const int nk = e == spare ? 0 : L.nkid[g.eoff + e];
                    for (int j = 2; j < nk; ++j)
                        R = MIXED ? fma(-X[i0 + j], kt[i0 + j].y, R) : R - PR[i0 + j];
                }
                X[e] = R;
                if (!MIXED) PR[e] = R * T;
                ownn = on + a.x;
                Tn = a.y;
            } else {
                const double2 a = kt[en];
                kn = kid[en];
                ownn = O[en] + a.x;
                Tn = a.y;
            }
            if (m.y & CHUNK_FIRST) sync();
            k = kn;
            T = Tn;
            own = ownn;
            e = en;
            m = mn;
            mn = m2;
        }
        m = ch[0];
        mn = ch[1];
        e = element(m);
        double2 a = cy[e];
        double D = MIXED ? 0.0 : dd[e], old = CRANK ? O[e] : 0.0;
        int p = par[e];
        own = MIXED ? X[e] * a.y : X[e];
        bar_named(LB_FORWARD, nth);
        bar_named(LB_TOP, nth);
        for (int c = 0; c < nch; ++c) {
            const int2 m2 = ch[c + 2];
            const int en = element(mn);
            double2 an;
            double Dn = 0.0, on, oldn = 0.0;
            int pn;
            if (busy(m)) {
                const double xp = U[p];
                an = cy[en];
                on = X[en];
                pn = par[en];
                if (!MIXED) Dn = dd[en];
                if (CRANK) oldn = O[en];
                double r;
                if (MIXED) {
                    r = fma(-a.x, xp, own);   // R / D' - (C / D') x
                } else {
                    // RN(r / D') from the correctly rounded y = 1/D' by
                    // Markstein's correction, the division's bits
                    r = own - a.x * xp;
                    const double t = r * a.y;
                    r = fma(fma(-D, t, r), a.y, t);
                }
                X[e] = r;
                if (CRANK) O[e] = MIXED ? fma(2.0, r, -old) : r + r - old;
                if (MIXED) on *= an.y;
            } else {
                an = cy[en];
                on = MIXED ? X[en] * an.y : X[en];
                pn = par[en];
                if (!MIXED) Dn = dd[en];
                if (CRANK) oldn = O[en];
            }
            if (m.y & CHUNK_LAST) sync();
            a = an;
            D = Dn;
            own = on;
            old = oldn;
            p = pn;
            e = en;
            m = mn;
            mn = m2;
        }
        if (take) {   // before the next step's sweep
            level_out(v, L, g.tile, g.lane0, g.nlanes, step0 + it, tid, nt, O);
            sync();
        }
    }
}

template <bool MIXED, bool CRANK, int NTOP, bool RES, bool IO = false>
__device__ __forceinline__ void level_sweep(const DevView &v, const LevelView &L, const LevelGroup &g, const Tile &tl,
                                            const TileType &ty, double *sm, int nsteps, long long step0, bool full,
                                            bool refresh)
{
    const int tid = threadIdx.x, nt = blockDim.x - LANES;
    const LevelSm q = level_smem_of<MIXED, CRANK, NTOP, RES>(sm, g);
    double *const X = q.X, *const PR = q.PR, *const O = q.O;
    const int2 *const ch = q.ch;
    const int nch = g.nch;
    const int *map = L.map + g.eoff, *kid = L.kid + g.eoff, *par = L.par + g.eoff;
    double2 *kt = L.kt + g.eoff, *cy = L.cy + g.eoff;
    double *dd = L.d + g.eoff, *pd = L.pd + g.eoff;
    double *V = v.V + tl.vm * LANES;
    for (int c = tid - LV_GUARD; c < nch + LV_GUARD; c += nt)
        q.ch[c] = c >= 0 && c < nch ? L.chunks[g.choff + c] : make_int2(0, 0);
    for (int e = tid; e < g.n; e += nt) O[e] = V[map[e]];
    if (tid < LV_SPARE) X[g.n + tid] = O[g.n + tid] = PR[g.n + tid] = 0.0;
    bar_named(LB_SWEEP, nt);
    const int *pf = v.prog + ty.pf_off;
    const double *P = v.P + tl.fld * LANES;
    if (full) {
        // the factors from the fields: the diagonals' elimination, level by
        // level; PR holds B T meanwhile
        const double *A = v.A + tl.topo * LANES, *B = v.B + tl.topo * LANES;
        for (int c = nch - 1; c >= 0; --c) {
            const int2 m = ch[c];
            if (tid < (m.y & CHUNK_COUNT)) {
                const int e = m.x + tid, r = map[e], l = r % LANES;
                const int *ps = pf + 6 * (r / LANES);
                double D;
                if (MIXED) D = df2d(ld_df(&P[ps[5] * LANES + l]));
                else D = 0.0 * P[ps[4] * LANES + l] + P[ps[5] * LANES + l];
                const int k0 = kid[e] & 0xffff, nk = L.nkid[g.eoff + e];
                for (int k = 0; k < nk; ++k) D -= PR[k0 + k];
                const double y = MIXED ? rcp_step(D) : 1.0 / D;   // FP64: correctly rounded
                const double T = MIXED ? A[r] * y : A[r] / D;
                const double b = B[r] * T;
                PR[e] = b;
                pd[e] = b;
                kt[e] = make_double2(level_kterm<MIXED>(P, pf, r), T);
                cy[e] = make_double2(MIXED ? L.c[g.eoff + e] * y : L.c[g.eoff + e], y);
                if (!MIXED) dd[e] = D;
            }
            if (m.y & CHUNK_FIRST) bar_named(LB_SWEEP, nt);
        }
    } else if (refresh) {   // inputs on the rhs fields: their terms once per launch
        for (int e = tid; e < g.n; e += nt) kt[e].x = level_kterm<MIXED>(P, pf, map[e]);
    }
    if (full || refresh) {
        __threadfence_block();
        bar_named(LB_SWEEP, nt);
    }
    if (RES)
        for (int e = tid; e < g.n + LV_SPARE; e += nt) {
            q.kt[e] = kt[e];
            q.cy[e] = cy[e];
            if (!MIXED) q.d[e] = dd[e];
            q.kid[e] = kid[e];
            q.par[e] = par[e];
        }
    bar_named(LB_SWEEP, nt);
    if (g.many) level_steps<MIXED, CRANK, NTOP, RES, IO, true>(v, L, g, q, nsteps, step0);
    else level_steps<MIXED, CRANK, NTOP, RES, IO, false>(v, L, g, q, nsteps, step0);
    bar_named(LB_SWEEP, nt);
    for (int e = tid; e < g.n; e += nt) V[map[e]] = O[e];
}

// The static children of top row s of this lane: their contributions off
// (R, D), in ascending row order.
template <bool MIXED, bool RES>
__device__ __forceinline__ void level_top_kids(const LevelView &L, const LevelGroup &g, const LevelSm &q, int s,
                                               int lane, double &R, double &D)
{
    const double2 *kt = RES ? q.kt : L.kt + g.eoff;
    const int kk = L.topkid[g.kidoff + s * LANES + lane];
    const int k0 = kk & ((1 << LV_KID_BITS) - 1), nk = (unsigned)kk >> LV_KID_BITS;
    for (int k = 0; k < nk; ++k) {
        D -= L.pd[g.eoff + k0 + k];
        R = MIXED ? fma(-q.X[k0 + k], kt[k0 + k].y, R) : R - q.PR[k0 + k];
    }
}
#endif

}  // namespace gbh
