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
    double2 *cy;         // backward coefficient C (mixed: C / D'), 1 / D'
    const double *c;     // C
    double *d;           // D' (FP64 form)
    double *pd;          // B T: what the row takes from its parent's diagonal
    unsigned *gen;       // per group: the fields' generation its factors were kept at (DevView::sgen)
};

// Where a block keeps its rows' constants between steps: in shared memory,
// read from L2 once per launch (resident), or streamed from L2 through a ring
// of LV_RING chunks on every sweep.
constexpr int LV_RING = 6;

// Shared memory of a group's block of nt sweeping threads, in the order
// level_smem_of lays it out: the constants (or the ring), the top rows'
// solutions, R / solutions, the contributions R T and, under Crank-Nicolson,
// Vm; D' (FP64), the chunks and the indices.
__host__ __device__ inline size_t level_smem(int ntop, int n, int nch, bool crank, bool mixed, bool resident, int nt)
{
    const size_t row = 16 + 8 + 4;   // two constants, D' or nothing, an index
    const size_t state = 8 * ((size_t)ntop * LANES + (size_t)n * (crank ? 3 : 2)) + 8 * (size_t)nch;
    return state + (resident ? (size_t)n * (2 * row - (mixed ? 16 : 8)) : LV_RING * row * (size_t)nt);
}

// Named barriers of a block: 1 the sweeping warps, 2 the static rows are
// eliminated, 3 the top rows are solved.
enum LevelBar { LB_SWEEP = 1, LB_FORWARD = 2, LB_TOP = 3 };

#ifdef __CUDACC__
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One block's arrays in shared memory.
struct LevelSm {
    double2 *kt, *cy;    // resident: the constants; else kt is the ring's pairs
    double *U, *X, *PR, *O, *d;
    int2 *ch;
    int *kid, *par;
};
template <bool MIXED, bool CRANK, int NTOP, bool RES>
__device__ __forceinline__ LevelSm level_smem_of(double *sm, const LevelGroup &g, int nt)
{
    LevelSm q;
    q.kt = reinterpret_cast<double2 *>(sm);
    q.cy = q.kt + g.n;
    double *p = sm + (RES ? 4 * g.n : 2 * LV_RING * nt);
    q.U = p;
    q.X = p + NTOP * LANES;
    q.PR = q.X + g.n;
    q.O = CRANK ? q.PR + g.n : q.X;
    p = q.PR + g.n * (CRANK ? 2 : 1);
    q.d = p;
    p += RES ? (MIXED ? 0 : g.n) : LV_RING * nt;
    q.ch = reinterpret_cast<int2 *>(p);
    q.kid = reinterpret_cast<int *>(q.ch + g.nch);
    q.par = q.kid + g.n;
    return q;
}

// A row's constants in registers: (K, T) and its children forward, (C, 1/D')
// -- mixed (C/D', 1/D') -- D' and its parent backward.
struct LevelRow {
    double2 a;
    double d;
    int k;
};

// What the sweeping warps of a block do in a launch (sm: level_smem bytes).
template <bool MIXED, bool CRANK, int NTOP, bool RES>
__device__ __forceinline__ void level_sweep(const DevView &v, const LevelView &L, const LevelGroup &g, const Tile &tl,
                                            const TileType &ty, double *sm, int nsteps, bool full, bool refresh)
{
    const int tid = threadIdx.x, nt = blockDim.x - LANES, nth = blockDim.x;
    const LevelSm q = level_smem_of<MIXED, CRANK, NTOP, RES>(sm, g, nt);
    double *const U = q.U, *const X = q.X, *const PR = q.PR, *const O = q.O;
    const int2 *const ch = q.ch;
    const int nch = g.nch;
    const int *map = L.map + g.eoff, *kid = L.kid + g.eoff, *par = L.par + g.eoff;
    double2 *kt = L.kt + g.eoff, *cy = L.cy + g.eoff;
    double *dd = L.d + g.eoff, *pd = L.pd + g.eoff;
    double *V = v.V + tl.vm * LANES;
    for (int c = tid; c < nch; c += nt) q.ch[c] = L.chunks[g.choff + c];
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
                cy[e] = make_double2(MIXED ? L.c[g.eoff + e] * y : L.c[g.eoff + e], y);
                if (!MIXED) dd[e] = D;
            }
            if (m.y & LV_FIRST) bar_named(LB_SWEEP, nt);
        }
    } else if (refresh) {   // inputs on the rhs fields: their terms once per launch
        for (int e = tid; e < g.n; e += nt) kt[e].x = kterm(map[e]);
    }
    if (full || refresh) {
        __threadfence_block();
        bar_named(LB_SWEEP, nt);
    }
    if (RES) {
        for (int e = tid; e < g.n; e += nt) {
            cp_async16(&q.kt[e], &kt[e]);
            cp_async16(&q.cy[e], &cy[e]);
            if (!MIXED) cp_async8(&q.d[e], &dd[e]);
            cp_async4(&q.kid[e], &kid[e]);
            cp_async4(&q.par[e], &par[e]);
        }
        cp_commit();
        cp_wait<0>();
        bar_named(LB_SWEEP, nt);
    }
    // Streamed: the chunks of a step in the order they are used -- forward
    // from the last, backward from the first -- are fetched LV_RING - 1 uses
    // ahead, across levels, sweeps and steps (the loads would otherwise follow
    // each level's barrier: some 600 clocks). Each thread fetches the rows it
    // takes itself, so only its own copies have to be waited for.
    int fpos = 0, fslot = 0, slot = 0;   // next use to fetch, its ring slot, the slot in use
    int *const ring_i = q.kid;
    // mixed, resident: a parent subtracts R T in one multiply-add, T from its
    // child's constants; else the child leaves R T in PR
    constexpr bool FMA = MIXED && RES;
    const double *const pulled = FMA ? X : PR;
    auto fetch = [&]() {
        if (RES) return;
        const bool fwd = fpos < nch;
        const int2 m = ch[fwd ? nch - 1 - fpos : fpos - nch];
        if (tid < (m.y & LV_COUNT)) {
            const int e = m.x + tid, s = fslot * nt + tid;
            cp_async16(&q.kt[s], fwd ? &kt[e] : &cy[e]);
            cp_async4(&ring_i[s], fwd ? &kid[e] : &par[e]);
            if (!MIXED && !fwd) cp_async8(&q.d[s], &dd[e]);
        }
        cp_commit();
        fpos = fpos + 1 == 2 * nch ? 0 : fpos + 1;
        fslot = fslot + 1 == LV_RING ? 0 : fslot + 1;
    };
    auto take = [&](int e, bool fwd, LevelRow &r) {   // (every use takes one ring slot, rows or none)
        if (RES) {
            r.a = fwd ? q.kt[e] : q.cy[e];
            r.k = fwd ? q.kid[e] : q.par[e];
            if (!MIXED && !fwd) r.d = q.d[e];
        } else {
            const int s = slot * nt + tid;
            r.a = q.kt[s];
            r.k = ring_i[s];
            if (!MIXED && !fwd) r.d = q.d[s];
        }
    };
    auto next_slot = [&]() {
        if (RES) return;
        slot = slot + 1 == LV_RING ? 0 : slot + 1;
    };
    if (!RES)
        for (int u = 0; u < LV_RING - 1; ++u) fetch();
    // The FP64 unit takes an instruction from a warp every 64 clocks, whatever
    // depends on it, so a level lasts as long as its instructions in a row:
    // whatever does not wait for the level before is formed ahead of the
    // barrier -- the constants, Vm + K forward and, mixed, R / D' backward.
    for (int it = 0; it < nsteps; ++it) {
        LevelRow row;
        double own = 0.0, old = 0.0;
        int2 m = ch[nch - 1];
        bool mine = tid < (m.y & LV_COUNT);
        if (!RES) cp_wait<LV_RING - 2>();
        if (mine) {
            take(m.x + tid, true, row);
            own = O[m.x + tid] + row.a.x;
        }
        next_slot();
        for (int c = nch - 1; c >= 0; --c) {
            const int2 mn = ch[c > 0 ? c - 1 : 0];
            const bool minen = c > 0 && tid < (mn.y & LV_COUNT);
            const int k0 = row.k & ((1 << LV_KID_BITS) - 1), nk = mine ? (unsigned)row.k >> LV_KID_BITS : 0;
            // the first two children's loads together
            double c0 = 0.0, c1 = 0.0, t0 = 0.0, t1 = 0.0;
            if (nk > 0) {
                c0 = pulled[k0];
                if (FMA) t0 = q.kt[k0].y;
            }
            if (nk > 1) {
                c1 = pulled[k0 + 1];
                if (FMA) t1 = q.kt[k0 + 1].y;
            }
            LevelRow rn;
            double on = 0.0;
            fetch();
            if (!RES) cp_wait<LV_RING - 2>();
            if (minen) {
                take(mn.x + tid, true, rn);
                on = O[mn.x + tid];
            }
            if (c > 0) next_slot();
            if (mine) {
                const int e = m.x + tid;
                double R = own;
                if (FMA) {
                    if (nk > 0) R = fma(-c0, t0, R);
                    if (nk > 1) R = fma(-c1, t1, R);
                    for (int k = 2; k < nk; ++k) R = fma(-X[k0 + k], q.kt[k0 + k].y, R);
                } else {
                    if (nk > 0) R -= c0;
                    if (nk > 1) R -= c1;
                    for (int k = 2; k < nk; ++k) R -= PR[k0 + k];
                    PR[e] = R * row.a.y;
                }
                X[e] = R;
            }
            if (c > 0 && (m.y & LV_FIRST)) bar_named(LB_SWEEP, nt);
            own = on + rn.a.x;
            row = rn;
            m = mn;
            mine = minen;
        }
        m = ch[0];
        mine = tid < (m.y & LV_COUNT);
        if (!RES) cp_wait<LV_RING - 2>();
        if (mine) {
            take(m.x + tid, false, row);
            own = X[m.x + tid];
            if (MIXED) own *= row.a.y;
            if (CRANK) old = O[m.x + tid];
        }
        next_slot();
        bar_named(LB_FORWARD, nth);
        bar_named(LB_TOP, nth);
        for (int c = 0; c < nch; ++c) {
            const int2 mn = ch[c + 1 < nch ? c + 1 : c];
            const bool minen = c + 1 < nch && tid < (mn.y & LV_COUNT);
            double xp = 0.0;
            if (mine) xp = U[row.k];
            LevelRow rn;
            double on = 0.0, oldn = 0.0;
            fetch();
            if (!RES) cp_wait<LV_RING - 2>();
            if (minen) {
                take(mn.x + tid, false, rn);
                on = X[mn.x + tid];
                if (CRANK) oldn = O[mn.x + tid];
            }
            if (c + 1 < nch) next_slot();
            if (mine) {
                const int e = m.x + tid;
                double r;
                if (MIXED) {
                    r = fma(-row.a.x, xp, own);   // R / D' - (C / D') x
                } else {
                    // RN(r / D') from the correctly rounded y = 1/D' by
                    // Markstein's correction, the division's bits
                    r = own - row.a.x * xp;
                    const double t = r * row.a.y;
                    r = fma(fma(-row.d, t, r), row.a.y, t);
                }
                X[e] = r;
                if (CRANK) O[e] = MIXED ? fma(2.0, r, -old) : r + r - old;
            }
            if (c + 1 < nch && (m.y & LV_LAST)) bar_named(LB_SWEEP, nt);
            own = MIXED ? on * rn.a.y : on;
            old = oldn;
            row = rn;
            m = mn;
            mine = minen;
        }
        // (no barrier here: the next forward sweep starts with the deepest
        // level, whose solutions no other row reads, and passes one before it
        // rewrites any row above)
    }
    if (!RES) cp_wait<0>();
    bar_named(LB_SWEEP, nt);
    for (int e = tid; e < g.n; e += nt) V[map[e]] = O[e];
}

// The static children of top row s of this lane: their contributions off
// (R, D), in ascending row order.
template <bool FMA>
__device__ __forceinline__ void level_top_kids(const LevelView &L, const LevelGroup &g, const LevelSm &q, int s,
                                               int lane, double &R, double &D)
{
    const int kk = L.topkid[g.kidoff + s * LANES + lane];
    const int k0 = kk & ((1 << LV_KID_BITS) - 1), nk = (unsigned)kk >> LV_KID_BITS;
    for (int k = 0; k < nk; ++k) {
        D -= L.pd[g.eoff + k0 + k];
        if (FMA) R = fma(-q.X[k0 + k], q.kt[k0 + k].y, R);
        else R -= q.PR[k0 + k];
    }
}
#endif

}  // namespace gbh
