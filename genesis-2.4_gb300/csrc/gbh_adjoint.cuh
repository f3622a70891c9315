// gbh_adjoint.cuh -- reverse-mode (adjoint) kernels of the FP64 form.
//
// Loss L = sum over steps n and target rows j of (Vm_j after step n - trace[n][j])^2.
// The reference has no gradient; this is the differentiated form of its step
// (do_chip_hh4_update, genesis/src/hines/hines_chip.c:157-600, followed by
// do_euler_hsolve / do_crank_hsolve, genesis/src/hines/hines_solve.c:140-296).
//
// FP64 arithmetic on GB300: one warp issues at most ~0.47 lane-DFMA per clock
// whether its lanes are active or not, an SM ~1.6 with four warps or more, so
// a batch of a few thousand neurons (one warp per 32) reaches a quarter of the
// GPU's FP64 rate in any kernel that walks the steps one after another. The
// sweep therefore keeps the sequential kernels lean and moves the rest into
// kernels that are parallel over steps as well as neurons:
//
//   forward   the engine's own step kernel advances work copies of Vm and the
//             gate states; k_adj_copy stores them every K steps (checkpoints)
//             and, when a segment is recomputed, before every step (snapshot);
//   k_adj_linearize, k_adj_eliminate   (parallel over steps) recompute each
//             step of a segment from its snapshot with the step's exact
//             arithmetic and store the local derivatives the reverse needs:
//             1/D', A/D', R' and x of every row, ichan and sumg of every
//             compartment, the gate product of every channel, and per gate
//             d prod/dx, dx'/dVm (table slope, zero where the lookup clamps or
//             without interpolation) and dx'/dx (the trapezoid factor
//             (2-B')/B', zero for instant gates);
//   k_adj_reverse   (sequential over steps, a thread per compartment) the
//             adjoint recurrence of Vm and the gate states:
//               seed      Vm-bar += 2 (Vm after - target) at target rows
//                         (Crank-Nicolson: Vm after = 2x - Vm before);
//               back substitution reversed, rows ascending:
//                         x_s = (R'_s - C_s x_p) / D'_s;
//               forward elimination reversed, rows descending:
//                         t_s = A_s / D'_s, D'_p -= B_s t_s, R'_p -= R'_s t_s;
//               channels  rhs = Vm + ichan*tbyc, diag = sumg*tbyc + diagterm,
//                         G = gmax prod x^p, x' = (x(2-B') + A')/B';
//             it stores the adjoints of R, D and of the back substitution;
//   k_adj_reduce   (parallel over rows) sums the parameter gradients of a
//             segment from those adjoints and the tape, steps descending so
//             the totals do not depend on the checkpoint interval.
// Supported programs: compartments with voltage-table gated channels
// (M_BEGIN, M_NEWVOLT, M_CHAN, M_CHAN_G, M_GATE of kind GK_1V with a nonzero
// power, M_ADDCURR, M_END); the host rejects anything else.
#pragma once
#include <cuda_runtime.h>
#include "gbh_devfn.cuh"
#include "gbh_adjoint.h"

namespace gbh {

__device__ __forceinline__ double *adj_tape(const AdjView &v, int k, int t, int lane)
{
    return v.tape + ((int64_t)k * v.tp_stride + v.tp_off[t]) * LANES + lane;
}

// locate() of the interpolating lookup, also reporting whether the fraction
// moves with v (false where a fresh lookup clamps at either end of the table).
__device__ __forceinline__ bool locate_lin(VCursor &c, double v, const TableGeom &tg, const double *vals)
{
    double f = (v - tg.xmin) * tg.invdx;
    bool lin = true;
    if ((c.lo > v) || (v >= c.hi)) {
        if (f < 0.0) {
            f = 0.0;
            lin = false;
        } else if (f > tg.xdivs) {
            f = tg.xdivs;
            lin = false;
        }
        c.row = (int)f;
        f = f - (double)c.row;
        c.lo = vals[c.row];
        c.hi = vals[c.row + 1];
        c.base = c.row * tg.ncols;
    } else {
        f = f - (double)c.row;
    }
    c.frac = f;
    return lin;
}

// ---------------------------------------------------------------- copies
// grid (tiles, row chunks of ADJ_COPY_ROWS), one warp a row. (One warp walking
// 32 rows took 20 us for 24 tiles of 256 rows, a load's latency a row.)
__global__ void __launch_bounds__(LANES * ADJ_COPY_ROWS)
k_adj_copy(AdjView v, int c, int dir, int to_tape)
{
    const int lane = threadIdx.x;
    const int t = blockIdx.x;
    const Tile tl = v.tiles[t];
    const AdjType at = v.atypes[tl.type];
    const int r = blockIdx.y * ADJ_COPY_ROWS + threadIdx.y;
    if (r >= at.nslots + at.ngates) return;
    double *blk = to_tape ? adj_tape(v, c, t, lane)
                          : v.ckpt + ((int64_t)c * v.ck_stride + v.ck_off[t]) * LANES + lane;
    double *w = r < at.nslots ? v.V + (tl.vm + r) * LANES + lane
                              : v.P + (tl.fld + v.snap_field[at.snap_off + r - at.nslots]) * LANES + lane;
    if (dir == 0) blk[r * LANES] = *w;
    else *w = blk[r * LANES];
}

// Checkpoint c0 + k -> tape step k (blockIdx.z = k): the snapshot rows of a
// segment whose every step was kept by the forward pass.
__global__ void __launch_bounds__(LANES * ADJ_COPY_ROWS)
k_adj_ck_to_tape(AdjView v, int c0)
{
    const int lane = threadIdx.x;
    const int t = blockIdx.x;
    const int k = blockIdx.z;
    const Tile tl = v.tiles[t];
    const AdjType at = v.atypes[tl.type];
    const int r = blockIdx.y * ADJ_COPY_ROWS + threadIdx.y;
    if (r >= at.nslots + at.ngates) return;
    const double *src = v.ckpt + ((int64_t)(c0 + k) * v.ck_stride + v.ck_off[t]) * LANES + lane;
    adj_tape(v, k, t, lane)[r * LANES] = src[r * LANES];
}

// ---------------------------------------------------------------- linearisation
// a / b with y = rcp_exact(b) at hand
__device__ __forceinline__ double div_of(double a, double b, double y)
{
    return mid_range(a) && divisor_ok(b) ? div_by(a, b, y) : div_ieee(a, b);
}

// Channels: grid (tiles, steps), 32 threads; each row's diagonal and right-hand
// side go to the tape's RD and RP rows. Apart from the elimination, whose two
// shared-memory columns (32 KB a warp at 64 rows) leave 7 warps an SM: the
// gates' loads, one behind another, want more in flight (24 tiles of 64 rows x
// 100 steps: 2.40 ms in one kernel, 1.09 + 0.37 ms apart and with one
// reciprocal a divisor; that alone 2.19).
__global__ void __launch_bounds__(32)
k_adj_linearize(AdjView v)
{
    const int lane = threadIdx.x;
    const int t = blockIdx.x;
    const int k = blockIdx.y;
    const Tile tl = v.tiles[t];
    const TileType ty = v.types[tl.type];
    const AdjType at = v.atypes[tl.type];
    const TableGeom tg = v.tgeom[ty.table_set];
    const double *tab = v.tab64 + tg.tab_off;
    const double *xvals = v.xyvals + tg.xv_off;
    const int ncols = tg.ncols;
    const bool interp = ty.interp != 0;
    const int S = at.nslots;
    const AdjRows R = adj_rows(S, at.ngates, at.nchans);
    const double *P = v.P + tl.fld * LANES + lane;
    double *tp = adj_tape(v, k, t, lane);

    VCursor vc;
    if (ncols) { vc.lo = vc.hi = 0.0; } else { vc.lo = -1e20; vc.hi = 1e20; }
    vc.row = vc.base = 0;
    vc.frac = 0.0;
    double dfdv = 0.0;
    double Ek = 0.0, Gk = 0.0;
    int gi = 0, ci = -1, cg0 = 0;
    double gx[ADJ_MAX_GATES];
    int gp[ADJ_MAX_GATES];
    const int *pc = v.prog + ty.prog_off;
    for (int s = 0; s < S; ++s) {
        const double Vm = tp[(R.V + s) * LANES];
        double sumg = 0.0, ichan = 0.0;
        for (;;) {
            const int code = pc[0];
            if (code == M_BEGIN) {
                ichan = P[pc[1] * LANES] + P[pc[2] * LANES];
                pc += 5;
            } else if (code == M_NEWVOLT) {
                if (interp) {
                    dfdv = locate_lin(vc, Vm, tg, xvals) ? tg.invdx : 0.0;
                } else {
                    locate(vc, Vm, tg.xmin, tg.invdx, tg.xdivs, tg.xtop, xvals, ncols, false);
                    dfdv = 0.0;
                }
                pc += 1;
            } else if (code == M_CHAN || code == M_CHAN_G) {
                if (code == M_CHAN) {
                    Ek = P[pc[1] * LANES];
                    Gk = P[pc[2] * LANES];
                    pc += 3;
                } else {
                    Gk = P[pc[1] * LANES];
                    pc += 2;
                }
                ++ci;
                cg0 = gi;
            } else if (code == M_GATE) {
                const int b = vc.base + pc[2];
                double X, Y, sX = 0.0, sY = 0.0;
                if (interp) {
                    const double fr = vc.frac;
                    X = tab[b];
                    sX = tab[b + ncols] - X;
                    X = X + fr * sX;
                    Y = tab[b + 1];
                    sY = tab[b + 1 + ncols] - Y;
                    Y = Y + fr * sY;
                } else {
                    X = tab[b];
                    Y = tab[b + 1];
                }
                const int p = pc[3];
                const double st = tp[(R.ST + gi) * LANES];
                const int pw = abs(p);
                const double rX = rcp_exact(X);
                const double x = div_of(p > 0 ? st * (2.0 - X) + Y : Y, X, rX);
                Gk = gpow<double>(Gk, x, pw);
                const double along = p > 0 ? st + x : x;   // -(dx'/dB') * B'
                tp[(R.DXDV + gi) * LANES] = rX * dfdv * (sY - along * sX);
                tp[(R.DXDST + gi) * LANES] = p > 0 ? (2.0 - X) * rX : 0.0;
                const int j = gi - cg0;
                if (j < ADJ_MAX_GATES) {
                    gx[j] = x;
                    gp[j] = pw;
                } else if (v.status) {
                    atomicOr(v.status, ST_BAD_OP);
                }
                ++gi;
                pc += 5;
            } else if (code == M_ADDCURR) {
                sumg += Gk;
                ichan += Ek * Gk;
                const int ng = min(gi - cg0, ADJ_MAX_GATES);
                double prod = 1.0;
                for (int g = 0; g < ng; ++g) prod = gpow<double>(prod, gx[g], gp[g]);
                tp[(R.PROD + ci) * LANES] = prod;
                for (int g = 0; g < ng; ++g) {
                    double q = (double)gp[g];
                    for (int e = 1; e < gp[g]; ++e) q *= gx[g];
                    for (int h = 0; h < ng; ++h)
                        if (h != g) q = gpow<double>(q, gx[h], gp[h]);
                    tp[(R.Q + cg0 + g) * LANES] = q;
                }
                pc += 2;
            } else if (code == M_END) {
                const double tbyc = P[pc[1] * LANES];
                tp[(R.RP + s) * LANES] = Vm + ichan * tbyc;
                tp[(R.RD + s) * LANES] = sumg * tbyc + P[pc[2] * LANES];
                tp[(R.ICH + s) * LANES] = ichan;
                tp[(R.SG + s) * LANES] = sumg;
                pc += 4;
                break;
            } else {
                if (v.status) atomicOr(v.status, ST_BAD_OP);
                return;
            }
        }
    }
}

// Elimination: grid (tiles, steps), 32 threads. Shared memory: 2 * smax * 32
// doubles.
__global__ void __launch_bounds__(32)
k_adj_eliminate(AdjView v, int smax)
{
    extern __shared__ double sm[];
    const int lane = threadIdx.x;
    const int t = blockIdx.x;
    const int k = blockIdx.y;
    const Tile tl = v.tiles[t];
    const AdjType at = v.atypes[tl.type];
    const int S = at.nslots;
    const AdjRows R = adj_rows(S, at.ngates, at.nchans);
    const int *par = v.parent + tl.topo * LANES + lane;
    const double *Aw = v.A + tl.topo * LANES + lane;
    const double *Bw = v.B + tl.topo * LANES + lane;
    const double *Cw = v.Cb + tl.topo * LANES + lane;
    double *tp = adj_tape(v, k, t, lane);
    double *Dc = sm + lane;
    double *Rc = Dc + (size_t)smax * LANES;
#pragma unroll 4
    for (int s = 0; s < S; ++s) {
        Dc[s * LANES] = tp[(R.RD + s) * LANES];
        Rc[s * LANES] = tp[(R.RP + s) * LANES];
    }
    for (int s = 0; s < S; ++s) {
        const int p = par[s * LANES];
        const double d = Dc[s * LANES];
        const double rd = rcp_exact(d);
        tp[(R.RD + s) * LANES] = rd;
        tp[(R.RP + s) * LANES] = Rc[s * LANES];
        double temp = 0.0;
        if (p >= 0) {
            temp = div_of(Aw[s * LANES], d, rd);
            Dc[p * LANES] -= Bw[s * LANES] * temp;
            Rc[p * LANES] -= Rc[s * LANES] * temp;
        }
        tp[(R.T + s) * LANES] = temp;
    }
    for (int s = S - 1; s >= 0; --s) {
        const int p = par[s * LANES];
        double r = Rc[s * LANES];
        if (p >= 0) r -= Cw[s * LANES] * Rc[p * LANES];
        r = div_of(r, Dc[s * LANES], tp[(R.RD + s) * LANES]);
        Rc[s * LANES] = r;
        tp[(R.X + s) * LANES] = r;
    }
}

// ---------------------------------------------------------------- reverse
// grid (groups), up to 16 warps: a block owns some neurons of a tile and gives
// each of their compartments a thread. The elimination's reverse goes through
// the tree depth by depth (back substitution reversed from the deepest rows
// up, a row pulling its children's contributions in ascending row order;
// forward elimination reversed from the root down), the channels' reverse and
// the next step's seeds take all rows at once. With one neuron per lane and
// the tree walked on one warp a step took 120 us for 24 tiles of 64
// compartments on 24 SMs (3 FP64 instructions up and 8 down per row, 64 rows
// in a row); with a thread per compartment it takes 22 us, bound by the
// levels' barriers and the tape's loads. Shared memory: the adjoints of R and
// D, what a parent takes from its children, the adjoint of Vm, the
// coefficients and links of the group's rows, and the tile type's slot and
// channel plans.
__global__ void __launch_bounds__(ADJ_REV_THREADS)
k_adj_reverse(AdjView v, AdjPlan pl, int hmax, int nk, int step0)
{
    extern __shared__ double sm[];
    const int tid = threadIdx.x, nt = blockDim.x;
    const AdjGroup g = pl.groups[blockIdx.x];
    const int t = g.tile, n = g.n;
    const Tile tl = v.tiles[t];
    const TileType ty = v.types[tl.type];
    const AdjType at = v.atypes[tl.type];
    const int S = at.nslots;
    const bool crank = ty.crank != 0;
    const AdjRows R = adj_rows(S, at.ngates, at.nchans);
    double *Rb = sm, *Db = Rb + n + 1, *CR = Db + n + 1, *Vb = CR + n, *B = Vb + n, *C = B + n;
    int2 *ch = reinterpret_cast<int2 *>(C + n), *link = ch + g.nch;
    int *map = reinterpret_cast<int *>(link + n), *tgt = map + n;
    AdjSlot *slots = reinterpret_cast<AdjSlot *>(tgt + n);
    AdjChan *chans = reinterpret_cast<AdjChan *>(slots + S);
    for (int i = tid; i < g.nch; i += nt) ch[i] = pl.chunks[g.choff + i];
    for (int i = tid; i < n; i += nt) {
        const int m = pl.map[g.eoff + i];
        map[i] = m;
        link[i] = pl.link[g.eoff + i];
        B[i] = v.B[tl.topo * LANES + m];
        C[i] = v.Cb[tl.topo * LANES + m];
        tgt[i] = v.tgt[tl.topo * LANES + m];
        Vb[i] = v.Vbar[tl.vm * LANES + m];
    }
    for (int i = tid; i < S; i += nt) slots[i] = v.slot_plan[at.slot_off + i];
    for (int i = tid; i < at.nchans && i < hmax; i += nt) chans[i] = v.chan_plan[at.chan_off + i];
    if (tid == 0) Rb[n] = Db[n] = 0.0;
    __syncthreads();
    auto tape = [&](int k) { return v.tape + ((int64_t)k * v.tp_stride + v.tp_off[t]) * LANES; };

    // seed of step k at row e: vb is the adjoint of Vm after step k; each
    // row's squared errors are summed on their own, steps descending
    auto seed = [&](int k, int e, double vb) {
        const int j = tgt[e];
        if (j >= 0) {
            const double *tp = tape(k) + map[e];
            const double x = __ldg(tp + R.X * LANES);
            const double vnext = crank ? x + x - __ldg(tp + R.V * LANES) : x;
            const double diff = vnext - __ldg(v.trace + (size_t)(step0 + k) * v.ntargets + j);
            v.loss[tl.topo * LANES + map[e]] += diff * diff;
            vb += 2.0 * diff;
        }
        Rb[e] = crank ? 2.0 * vb : vb;
        Vb[e] = crank ? -vb : 0.0;
    };
    // the tape rows of step k this thread's compartments will read, into L1
    auto ahead = [&](int k) {
        if (k < 0) return;
        const double *tp = tape(k);
        for (int e = tid; e < n; e += nt) {
            const double *q = tp + map[e];
            prefetch_l1(q + R.RD * LANES);
            prefetch_l1(q + R.T * LANES);
            prefetch_l1(q + R.RP * LANES);
            prefetch_l1(q + R.X * LANES);
            const AdjSlot sp = slots[map[e] / LANES];
            const int lane = map[e] % LANES;
            for (int c = sp.ch0; c < sp.ch0 + sp.nch; ++c) {
                const AdjChan h = c < hmax ? chans[c] : v.chan_plan[at.chan_off + c];
                for (int i = h.g0; i < h.g0 + h.ng; ++i) {
                    prefetch_l1(tp + (R.Q + i) * LANES + lane);
                    prefetch_l1(tp + (R.DXDV + i) * LANES + lane);
                    prefetch_l1(tp + (R.DXDST + i) * LANES + lane);
                }
            }
        }
    };
    ahead(nk - 1);
    for (int e = tid; e < n; e += nt) seed(nk - 1, e, Vb[e]);
    __syncthreads();
    for (int k = nk - 1; k >= 0; --k) {
        double *tp = tape(k);
        ahead(k - 1);
        // back substitution reversed, children before their parents
        for (int c = g.nch - 1; c >= 0; --c) {
            const int2 m = ch[c];
            if (tid < (m.y & CHUNK_COUNT)) {
                const int e = m.x + tid, k0 = link[e].x & 0xffff, nkid = link[e].x >> 16;
                double *q = tp + map[e];
                const double rd = __ldg(q + R.RD * LANES), x = __ldg(q + R.X * LANES);
                double r = Rb[e];
                for (int i = k0; i < k0 + nkid; ++i) r -= CR[i];
                const double rb = r * rd;
                Rb[e] = rb;
                CR[e] = C[e] * rb;
                Db[e] = -x * rb;
                q[R.RBBS * LANES] = rb;
            }
            if (m.y & CHUNK_FIRST) __syncthreads();
        }
        // forward elimination reversed, parents before their children
        for (int c = 0; c < g.nch; ++c) {
            const int2 m = ch[c];
            if (tid < (m.y & CHUNK_COUNT)) {
                const int e = m.x + tid, p = link[e].y;
                if (p < n) {
                    const double *q = tp + map[e];
                    const double tt = __ldg(q + R.T * LANES), rd = __ldg(q + R.RD * LANES);
                    const double tb = -B[e] * Db[p] - __ldg(q + R.RP * LANES) * Rb[p];
                    Rb[e] -= tt * Rb[p];
                    Db[e] -= tt * (tb * rd);
                }
            }
            if (m.y & CHUNK_LAST) __syncthreads();
        }
        // channels reversed (adjoint of Vm and of the gate states), then the
        // seed of step k-1
        for (int e = tid; e < n; e += nt) {
            const int mp = map[e], lane = mp % LANES;
            const AdjSlot sp = slots[mp / LANES];
            const double *P = v.P + tl.fld * LANES + lane;
            double *Xb = v.Xbar + v.xb_off[t] * LANES + lane;
            const double rb = Rb[e], db = Db[e];
            tp[R.RBF * LANES + mp] = rb;
            tp[R.DBF * LANES + mp] = db;
            const double tbyc = __ldg(P + sp.f_tbyc * LANES);
            const double Ibar = rb * tbyc, Sbar = db * tbyc;
            double vbn = Vb[e] + rb;
            for (int c = sp.ch0; c < sp.ch0 + sp.nch; ++c) {
                const AdjChan h = c < hmax ? chans[c] : v.chan_plan[at.chan_off + c];
                const double Ek = h.f_ek >= 0 ? __ldg(P + h.f_ek * LANES) : 0.0;
                const double w = (Sbar + Ibar * Ek) * __ldg(P + h.f_gmax * LANES);
#pragma unroll 2
                for (int i = h.g0; i < h.g0 + h.ng; ++i) {
                    const double xhat = Xb[i * LANES] + w * __ldg(tp + (R.Q + i) * LANES + lane);
                    vbn += xhat * __ldg(tp + (R.DXDV + i) * LANES + lane);
                    Xb[i * LANES] = xhat * __ldg(tp + (R.DXDST + i) * LANES + lane);
                }
            }
            if (k > 0) seed(k - 1, e, vbn);
            else Vb[e] = vbn;
        }
        __syncthreads();
    }
    for (int e = tid; e < n; e += nt) v.Vbar[tl.vm * LANES + map[e]] = Vb[e];
}

// ---------------------------------------------------------------- gradient sums
// grid (tiles, smax), 32 threads: one (tile, slot) per block, one lane per
// thread. Sums the segment's steps in descending order onto the totals.
__global__ void __launch_bounds__(32)
k_adj_reduce(AdjView v, int nk)
{
    const int lane = threadIdx.x;
    const int t = blockIdx.x;
    const int s = blockIdx.y;
    const Tile tl = v.tiles[t];
    const AdjType at = v.atypes[tl.type];
    if (s >= at.nslots) return;
    const AdjRows R = adj_rows(at.nslots, at.ngates, at.nchans);
    const AdjSlot sp = v.slot_plan[at.slot_off + s];
    const double *P = v.P + tl.fld * LANES + lane;
    double *Gf = v.Gf + tl.fld * LANES + lane;
    const int64_t topo = (tl.topo + s) * LANES + lane;
    const int p = v.parent[topo];
    const double tbyc = P[sp.f_tbyc * LANES];
    double g_i = Gf[sp.f_emrm * LANES];     // Em/Rm and inject share the adjoint of ichan
    double g_j = Gf[sp.f_inj * LANES];
    double g_t = Gf[sp.f_tbyc * LANES];
    double g_d = Gf[sp.f_diag * LANES];
    double ga = v.GA[topo], gb = v.GB[topo], gc = v.GC[topo];
    const double B = v.B[topo];
    for (int k = nk - 1; k >= 0; --k) {
        const double *tp = adj_tape(v, k, t, lane);
        const double rb = tp[(R.RBF + s) * LANES], db = tp[(R.DBF + s) * LANES];
        const double ib = rb * tbyc;
        g_i += ib;
        g_j += ib;
        g_t += rb * tp[(R.ICH + s) * LANES] + db * tp[(R.SG + s) * LANES];
        g_d += db;
        if (p >= 0) {
            gc -= tp[(R.X + p) * LANES] * tp[(R.RBBS + s) * LANES];
            const double dbp = tp[(R.DBF + p) * LANES], rbp = tp[(R.RBF + p) * LANES];
            gb -= tp[(R.T + s) * LANES] * dbp;
            ga += (-B * dbp - tp[(R.RP + s) * LANES] * rbp) * tp[(R.RD + s) * LANES];
        }
    }
    Gf[sp.f_emrm * LANES] = g_i;
    Gf[sp.f_inj * LANES] = g_j;
    Gf[sp.f_tbyc * LANES] = g_t;
    Gf[sp.f_diag * LANES] = g_d;
    v.GA[topo] = ga;
    v.GB[topo] = gb;
    v.GC[topo] = gc;
    // channels of the slot: Ek and gmax gradients, kept per channel
    for (int c = sp.ch0; c < sp.ch0 + sp.nch; ++c) {
        const AdjChan ch = v.chan_plan[at.chan_off + c];
        const double Ek = ch.f_ek >= 0 ? P[ch.f_ek * LANES] : 0.0;
        const double gmax = P[ch.f_gmax * LANES];
        double *gek = v.Gek + (v.ch_off[t] + c) * LANES + lane;
        double *ggm = v.Ggm + (v.ch_off[t] + c) * LANES + lane;
        double a = *gek, b = *ggm;
        for (int k = nk - 1; k >= 0; --k) {
            const double *tp = adj_tape(v, k, t, lane);
            const double ib = tp[(R.RBF + s) * LANES] * tbyc, sb = tp[(R.DBF + s) * LANES] * tbyc;
            const double prod = tp[(R.PROD + c) * LANES];
            a += ib * gmax * prod;
            b += (sb + ib * Ek) * prod;
        }
        *gek = a;
        *ggm = b;
    }
}

}  // namespace gbh
