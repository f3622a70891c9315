// gbh_rows.cuh -- row-parallel steps: the device side of the kernels that
// gbh_jit.cu generates for small batches of neurons with channels along their
// dendrites (TileType::rows).
//
// With one neuron per lane a step lasts as long as one neuron's compartments
// one after another, some 4,000 to 8,000 clocks each: 24 tiles of 64
// compartments took 250 us, with 24 warps on a device that holds thousands. Here a
// block owns a group of neurons of a tile and gives each of their compartments
// a thread: compartments whose programs are equal (up to their field rows)
// run side by side, 32 to a warp, and the elimination goes through the rows
// depth by depth, forward from the deepest, a row subtracting its children's
// contributions in ascending row order, backward from the root. The operations
// per row and their order are the sequential sweep's (hines_solve.c:223-296),
// so FP64 results keep the reference's bits. An FP64 instruction costs a warp
// the same for one lane as for 32, so large batches keep the lane mapping; the
// engine times both.
#pragma once
#include "gbh_devfn.cuh"

namespace gbh {

// A block's share of a tile: lanes [lane0, lane0 + nlanes), their n rows at
// elements eoff of the level-ordered arrays, nch chunks of at most blockDim
// rows (first, rows | CHUNK_LAST at the last of a level), nitems runs of up to 32
// rows of one program class.
struct RowGroup {
    int tile, lane0, nlanes, n, nch, choff, nitems, itoff;
    int64_t eoff;
};

struct RowView {
    const RowGroup *groups;
    const int2 *chunks;
    const int4 *items;     // class, first entry of `work`, entries
    const int2 *work;      // by class: element, first field row * 32 + lane
    const int *map;        // row * 32 + lane within the tile
    const int2 *link;      // first child (consecutive, ascending rows) | number of children << 16; parent's
                           // element (the root's: the zero behind the group's rows)
    const int *prev;       // the previous compartment with a voltage lookup, -1 none, -2 the row has none
    const int *pos;        // element of row s of group lane l at s * nlanes + l
    const double *A, *B, *C;
};

// Shared memory of a block of n rows: state, coefficients and links.
__host__ __device__ inline size_t rows_smem(int n, int nch)
{
    return ((size_t)n + 1) * (8 * 9 + 8 + 4 * 2) + 8 * (size_t)nch;
}

#ifdef __CUDACC__
struct RowSm {
    double *V, *R, *D, *Y, *PR, *PD;   // Vm; rhs, then the solution; D', 1/D'; what the parent subtracts
    double *A, *B, *C;
    int2 *ch, *link;
    int *fresh, *in;                   // table rows: of a fresh lookup, carried into the compartment
};
__device__ __forceinline__ RowSm rows_smem_of(double *sm, const RowGroup &g)
{
    RowSm q;
    const int n = g.n + 1;
    q.V = sm;
    q.R = q.V + n;
    q.D = q.R + n;
    q.Y = q.D + n;
    q.PR = q.Y + n;
    q.PD = q.PR + n;
    q.A = q.PD + n;
    q.B = q.A + n;
    q.C = q.B + n;
    q.ch = reinterpret_cast<int2 *>(q.C + n);
    q.link = q.ch + g.nch;
    q.fresh = reinterpret_cast<int *>(q.link + n);
    q.in = q.fresh + n;
    return q;
}

// The group's state and constants, once per launch.
__device__ __forceinline__ void rows_load(const RowView &L, const RowGroup &g, const RowSm &q, const double *Vt)
{
    for (int c = threadIdx.x; c < g.nch; c += blockDim.x) q.ch[c] = L.chunks[g.choff + c];
    for (int e = threadIdx.x; e < g.n; e += blockDim.x) {
        q.V[e] = Vt[L.map[g.eoff + e]];
        q.A[e] = L.A[g.eoff + e];
        q.B[e] = L.B[g.eoff + e];
        q.C[e] = L.C[g.eoff + e];
        q.link[e] = L.link[g.eoff + e];
    }
    if (threadIdx.x == 0) q.R[g.n] = 0.0;   // the root's parent
    __syncthreads();
}

// Table row of a fresh lookup of v.
__device__ __forceinline__ int rows_fresh(double v, double vmin, double inv, int divs, unsigned top)
{
    VCursor c;
    double f = (v - vmin) * inv;
    locate_row(c, f, divs, top);
    return c.row;
}

// The cursor a compartment starts from: at table row `row`, or reset.
__device__ __forceinline__ void rows_cursor(VCursor &c, int row, const double *vals, int ncols)
{
    c.lo = c.hi = 0.0;
    c.row = c.base = 0;
    c.rowd = c.frac = 0.0;
    if (row >= 0) {
        c.row = row;
        c.rowd = (double)row;
        c.lo = vals[row];
        c.hi = vals[row + 1];
        c.base = row * ncols;
    }
}

__device__ __forceinline__ bool rows_hit(const double *vals, int row, double v)
{
    const long long k = dkey(v);
    return !(dkey(vals[row]) > k || k >= dkey(vals[row + 1]));
}

// FP64 form: the reference carries the table bracket of one compartment to the
// next of its neuron (hines_chip.c:174-203). The incoming row of each is the
// fresh row of the previous one, unless a value lies in the previous bracket
// while its own fresh row differs (a rounding edge at a table node): then
// every neuron's chain is replayed in row order.
__device__ __forceinline__ void rows_cursors(const RowView &L, const RowGroup &g, const RowSm &q, const double *vals,
                                             double vmin, double inv, int divs, unsigned top, int S)
{
    const int *prev = L.prev + g.eoff;
    int edge = 0;
    for (int e = threadIdx.x; e < g.n; e += blockDim.x) q.fresh[e] = rows_fresh(q.V[e], vmin, inv, divs, top);
    __syncthreads();
    for (int e = threadIdx.x; e < g.n; e += blockDim.x) {
        const int p = prev[e];
        const int r = p >= 0 ? q.fresh[p] : -1;
        q.in[e] = r;
        if (p >= 0 && r != q.fresh[e] && rows_hit(vals, r, q.V[e])) edge = 1;
    }
    if (__syncthreads_or(edge)) {
        for (int l = threadIdx.x; l < g.nlanes; l += blockDim.x) {
            int state = -1;
            for (int s = 0; s < S; ++s) {
                const int e = L.pos[g.eoff + s * g.nlanes + l];
                if (prev[e] == -2) continue;
                q.in[e] = state;
                if (state < 0 || !rows_hit(vals, state, q.V[e])) state = q.fresh[e];
            }
        }
        __syncthreads();
    }
}

// The elimination of all rows of the group from (R, D): the solution into R,
// Vm of the next step into V. An FP64 instruction takes its scheduler's unit
// for 64 clocks, so a level costs its instructions in a row -- the diagonal's
// and the rhs's children, reciprocal, factor and two products forward, five
// backward -- and whatever does not wait for the level before is read ahead of
// its barrier.
template <bool MIXED, bool CRANK>
__device__ __forceinline__ void rows_eliminate(const DevView &v, const RowGroup &g, const RowSm &q, unsigned &lost)
{
    const int tid = threadIdx.x;
    int2 m = q.ch[g.nch - 1];
    int e = tid < (m.y & CHUNK_COUNT) ? m.x + tid : -1, lk = 0;
    double a = 0.0, b = 0.0, D = 0.0, R = 0.0;
    auto own = [&](int c) {   // the row of chunk c this thread takes
        m = q.ch[c];
        e = tid < (m.y & CHUNK_COUNT) ? m.x + tid : -1;
        if (e >= 0) {
            lk = q.link[e].x;
            a = q.A[e];
            b = q.B[e];
            D = q.D[e];
            R = q.R[e];
        }
    };
    own(g.nch - 1);
    for (int c = g.nch - 1; c >= 0; --c) {
        const int first = m.y & CHUNK_FIRST;
        if (e >= 0) {
            const int k0 = lk & 0xffff, nk = lk >> 16;
            for (int k = k0; k < k0 + nk; ++k) {
                D -= q.PD[k];
                R -= q.PR[k];
            }
            const double y = MIXED ? rcp_step(D) : rcp_rn(D);
            const double T = MIXED ? a * y : div_by(a, D, y);
            q.PD[e] = b * T;
            q.PR[e] = R * T;
            q.R[e] = R;
            if (!MIXED) q.D[e] = D;
            q.Y[e] = y;
        }
        if (c > 0) own(c - 1);
        if (first) __syncthreads();
    }
    int p = 0;
    double cc = 0.0, y = 0.0;
    auto back = [&](int c) {
        m = q.ch[c];
        e = tid < (m.y & CHUNK_COUNT) ? m.x + tid : -1;
        if (e >= 0) {
            p = q.link[e].y;
            cc = q.C[e];
            y = q.Y[e];
            R = q.R[e];
            if (!MIXED) D = q.D[e];
        }
    };
    back(0);
    for (int c = 0; c < g.nch; ++c) {
        const int last = m.y & CHUNK_LAST;
        if (e >= 0) {
            const double xp = q.R[p];
            double r;
            if (MIXED) {
                r = fma(-cc, xp, R) * y;
            } else {
                r = R - cc * xp;
                r = div_by(r, D, y);
            }
            q.R[e] = r;
            if (p == g.n) finite_check(v, r, true);   // the root: a NaN anywhere in the tree reaches it
        }
        if (c + 1 < g.nch) back(c + 1);
        if (last) __syncthreads();
    }
    for (int i = tid; i < g.n; i += blockDim.x) {
        const double r = q.R[i], old = q.V[i];
        if (MIXED) see_row(lost, r);   // (what the mixed form makes of a NaN may not)
        q.V[i] = CRANK ? (MIXED ? fma(2.0, r, -old) : r + r - old) : r;
    }
    __syncthreads();
}
#endif

}  // namespace gbh
