// Plain FP64 collocate / integrate: FP64 everywhere, one CTA per pair or per part
// of a pair's planes, grid updates by FP64 atomics.  The GPU form of the
// reference's per-pair loops (grid_collocate_core, grid_base_ref_c.cc:403-508;
// grid_collocate_general, :593-846) and the denominator the tiled path is
// measured against.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "gpw_coef.cuh"
#include "gpw_ff.cuh"
#include "gpw_internal.h"

namespace gpw {

// ---------------------------------------------------------------------------
// pair set-up: packed coefficients c (ortho) or q (general, lattice basis)
__global__ void k_prep(const PairGeom *__restrict__ geoms, const LevelDev *__restrict__ levels,
                       const double *__restrict__ tmat, int tau, const double *__restrict__ pab,
                       double *__restrict__ coef) {
    extern __shared__ double sm[];
    const PairGeom &g = geoms[blockIdx.x];  // read in place (L1), not copied per thread
    CoefWs w;
    w.carve(sm, g.la_max, g.lb_max);
    fill_alpha(w, g);
    fill_local_block(w, g, tau, pab);
    __syncthreads();
    const int nc = ncoef(g.lp);
    if (g.ortho) {
        forward_coef(w, g, coef + g.coef_off);
        return;
    }
    double *c = w.end();  // packed c, before the lattice transform
    forward_coef(w, g, c);
    __syncthreads();
    // q[k][j][i] = sum over same-degree (lz,ly,lx) of T * c; T in lp = kMaxLp packing
    const LevelDev &lv = levels[g.level];
    const double *Tm = tmat + lv.tmat_off;
    const int NT = ncoef(kMaxLp);
    for (int t = threadIdx.x; t < nc; t += blockDim.x) {
        // decode t -> (k, j, i) in lp packing
        int k = 0, j = 0, i = 0;
        {
            int r = t;
            for (k = 0; k <= g.lp; k++) {
                const int cnt = ((g.lp - k + 1) * (g.lp - k + 2)) / 2;
                if (r < cnt) break;
                r -= cnt;
            }
            const int q = g.lp - k;
            for (j = 0; j <= q; j++) {
                if (r <= q - j) break;
                r -= q - j + 1;
            }
            i = r;
        }
        const int n = i + j + k;
        const int row = pidx(kMaxLp, k, j, i);
        double s = 0.0;
        for (int lz = 0; lz <= n; lz++)
            for (int ly = 0; ly <= n - lz; ly++) {
                const int lx = n - lz - ly;
                s += Tm[(int64_t)row * NT + pidx(kMaxLp, lz, ly, lx)] * c[pidx(g.lp, lz, ly, lx)];
            }
        coef[g.coef_off + t] = s;
    }
}

int smem_prep(int A, int B) {
    // workspace + a packed coefficient vector for the general-cell transform
    return 8 * (coef_ws_doubles(A, B) + ncoef(A + B));
}

// ---------------------------------------------------------------------------
// integrate back-transform: moments -> hab.  extra: the moments go to degree lp + extra
// (the backward pass's; those beyond lp are not read).
__global__ void k_backtransform(const PairGeom *__restrict__ geoms, const LevelDev *__restrict__ levels,
                                const double *__restrict__ tmat, int tau,
                                const double *__restrict__ mom, int extra, double *__restrict__ hab) {
    extern __shared__ double sm[];
    const PairGeom &g = geoms[blockIdx.x];  // read in place (L1), not copied per thread
    CoefWs w;
    w.carve(sm, g.la_max, g.lb_max);
    fill_alpha(w, g);
    const int nc = ncoef(g.lp);
    const double *W = mom + (extra ? g.mom_ext_off : g.coef_off);
    int lpw = g.lp + extra;
    double *Wc = w.end();
    if (!g.ortho) {
        // Wc[lz][ly][lx] = sum over same-degree (k,j,i) of T[(k,j,i)][(lz,ly,lx)] * Wq[k][j][i]
        const LevelDev &lv = levels[g.level];
        const double *Tm = tmat + lv.tmat_off;
        const int NT = ncoef(kMaxLp);
        for (int t = threadIdx.x; t < nc; t += blockDim.x) {
            int lz = 0, ly = 0, lx = 0;
            int r = t;
            for (lz = 0; lz <= g.lp; lz++) {
                const int cnt = ((g.lp - lz + 1) * (g.lp - lz + 2)) / 2;
                if (r < cnt) break;
                r -= cnt;
            }
            const int q = g.lp - lz;
            for (ly = 0; ly <= q; ly++) {
                if (r <= q - ly) break;
                r -= q - ly + 1;
            }
            lx = r;
            const int n = lx + ly + lz;
            const int col = pidx(kMaxLp, lz, ly, lx);
            double s = 0.0;
            for (int k = 0; k <= n; k++)
                for (int j = 0; j <= n - k; j++) {
                    const int i = n - k - j;
                    s += Tm[(int64_t)pidx(kMaxLp, k, j, i) * NT + col] * W[pidx(lpw, k, j, i)];
                }
            Wc[t] = s;
        }
        W = Wc;
        lpw = g.lp;
    }
    __syncthreads();
    adjoint_coef(w, g, tau, W, lpw, hab);
}

// ---------------------------------------------------------------------------
// Orthorhombic pairs.  An FP64 multiply-add costs 64 float instructions here
// (two lanes per cycle and SM), so the kernel is laid out to run little else on
// the FP64 pipe: about L of them per cube point.
//
// A CTA (4 warps) takes one item: every nparts-th plane of a pair's cube.  The
// three 1-D tables are built once per CTA; after that the warps work alone, one
// plane at a time, with no CTA barrier:
//   lane = x column (blocks of 32 columns in integrate, of 16 in collocate; the last one
//   of 32, 16 or 8; the warp's other lanes on the following rows), so that
//   collocate  T[ly] = sum_lx Cxy[ly][lx] X[lx][x] once per column, in registers,
//              then rho(y, x) = sum_ly T[ly] Y[ly][y] per point, Y broadcast from
//              shared memory, one FP64 reduction into the grid;
//   integrate  T[ly] += V(y, x) Y[ly][y] per point, lane-local: no shuffles per row.
//              Cxy[ly][lx] = sum_x T[ly][x] X[lx][x] once per plane (spread over the
//              lanes, T through shared memory), then W[lz][ly][lx] += Cxy Z[lz], the
//              packed moments spread over the lanes' registers.
// A row's range comes from the FP32 sphere rule where its error bound allows
// (sphere_jmax_fast, sphere_imax_fast), one folded row per lane.
// The form before it (one CTA per pair, three barriers per plane, a shuffle
// reduction of 11 accumulators per row, launches of similar pairs one after the
// other) took 21.1 ms to integrate and 6.1 ms to collocate 1000 pairs (l <= 2,
// 64^3); this one takes 0.45 and 0.42 ms, 65 % of the FP64 rate (1.10 TFLOP/s in a
// GEMM) counting L multiply-adds per cube point.
constexpr int kOrthoWarps = 4;  // (a power of two)

// the rows jf <= 0 that a cube can have: those whose mirror 1 - jf lies inside as well
GPW_HD int folded_rows(const PairGeom &g) { return 1 - (g.lb[1] > 1 - g.hi[1] ? g.lb[1] : 1 - g.hi[1]); }

// the shared memory of one of the items of pair g (planes in zparts, columns in xparts), in
// bytes; kOrthoStatic of it are the kernel's static shared variables
constexpr int kOrthoStatic = 16;
int smem_ortho_item(const PairGeom &g, int extra, int zparts, int xparts) {
    const int L = g.lp + 1 + extra;
    const int nx = (g.hi[0] - g.lb[0] + xparts) / xparts, ny = g.hi[1] - g.lb[1] + 1, nz = g.hi[2] - g.lb[2] + 1;
    const int np = (nz + zparts - 1) / zparts, nc = ncoef(L - 1);
    return 8 * (nc + L * (nx + ny + np) + kOrthoWarps * (33 * L + nshell(L - 1))) +
           4 * (nx + ny + nc + kOrthoWarps * folded_rows(g)) + kOrthoStatic;
}
// Parts such that an item fits a CTA: planes first, then columns.  extra = 0: one plane
// and a few columns always fit where smem_ortho_fp64 does, since the tables of y then take
// 8 L + 12 bytes a row, less than its 16 L + 8.  (Matters for thousands of columns only.)
bool fit_ortho_item(const PairGeom &g, int extra, int smem_limit, int &zparts, int &xparts) {
    const int planes = 2 - 2 * g.kgmin, nx = g.hi[0] - g.lb[0] + 1;
    while (zparts < planes && smem_ortho_item(g, extra, zparts, xparts) > smem_limit) zparts++;
    while (xparts < nx && smem_ortho_item(g, extra, zparts, xparts) > smem_limit) xparts *= 2;
    return smem_ortho_item(g, extra, zparts, xparts) <= smem_limit;
}

// The cube sizes that the FP64 path accepts: what one CTA held when it kept a
// whole pair (tables, dense coefficients and one plane's rows) in shared memory.
int smem_ortho_fp64(const PairGeom &g) {
    const int L = g.lp + 1;
    const int nx = g.hi[0] - g.lb[0] + 1, ny = g.hi[1] - g.lb[1] + 1, nz = g.hi[2] - g.lb[2] + 1;
    return 8 * (L * L * L + L * (nx + ny + nz) + L * L + ny * L) + 8 * ny;
}

// Integrate's results are the same bits from call to call: every sum has a fixed order.
// Where a warp's planes are added up they are dealt out beforehand, turn t (warp w has
// t = w, w + 4, ...) of an item of np planes, the largest (the middle ones) first and the
// warps in alternating order, so that their shares are about equal; -1: none in this turn.
// (Planes taken from a counter as warps come free, and parts added by atomics: 860 us for
// both directions of 1000 pairs on 64^3, 6.82 ms for 1500 general pairs on 128^3, mixed;
// this order 863 us and 6.72 ms.)
__device__ __forceinline__ int plane_of_turn(int t, int np) {
    const int j = np - 1 - ((t / kOrthoWarps) & 1 ? t ^ (kOrthoWarps - 1) : t);
    return j < 0 ? -1 : (j & 1 ? np - 1 - (j >> 1) : j >> 1);
}

// Moments of divided pairs: a slot per item, stride moments each.
struct PartSums {
    double *sum;
    int *ticket;
    int stride;
};
// An item's moments value(t), t < nc, to its pair's.  Those of a divided pair go to the
// item's slot, and the CTA that comes last adds up the parts, in order.
template <class F>
__device__ __forceinline__ void put_moments(const Fp64Item &it, int nc, const PartSums &ps, double *out, F value) {
    if (it.nparts == 1) {
        for (int t = threadIdx.x; t < nc; t += blockDim.x) out[t] = value(t);
        return;
    }
    __shared__ bool last;
    double *first = ps.sum + (int64_t)(it.slot - it.part) * ps.stride;
    for (int t = threadIdx.x; t < nc; t += blockDim.x) __stcg(first + (int64_t)it.part * ps.stride + t, value(t));
    __threadfence();
    __syncthreads();
    int *ticket = ps.ticket + (it.slot - it.part);
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1) == it.nparts - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int t = threadIdx.x; t < nc; t += blockDim.x) {
        double s = 0.0;
#pragma unroll 8
        for (int p = 0; p < it.nparts; p++) s += __ldcg(first + (int64_t)p * ps.stride + t);
        out[t] = s;
    }
    if (threadIdx.x == 0) *ticket = 0;  // for the next launch
}

// kAcc: the registers of T, L <= kAcc (kNPow, or kNPowB for the backward pass's
// moments to degree lp + 2)
template <bool kAdj, int kAcc>
__global__ void __launch_bounds__(32 * kOrthoWarps)
k_ortho_fp64(const PairGeom *__restrict__ geoms, const Fp64Item *__restrict__ items, int uparts, int uxparts,
             const LevelDev *__restrict__ levels, const int *__restrict__ table, const double *__restrict__ coef,
             double *__restrict__ mom, PartSums ps, GridPtrs grids, int *status, int extra) {
    extern __shared__ double sm[];
    constexpr int kN2 = (kAcc * (kAcc + 1)) / 2, kM2 = (kN2 + 31) / 32;        // (ly, lx) sums per lane
    constexpr int kNC = (kAcc * (kAcc + 1) * (kAcc + 2)) / 6, kMC = (kNC + 31) / 32;  // moments per lane
    const int bid = blockIdx.x;
    const Fp64Item it = items ? items[bid] : Fp64Item{bid / uparts, bid % uparts, uparts, uxparts, -1};
    const PairGeom &g = geoms[it.pair];
    const LevelDev &lv = levels[g.level];
    double *__restrict__ grid = grids.p[g.level];
    const int lp = g.lp + extra, L = lp + 1, nc = ncoef(lp), n2 = nshell(lp);
    int lb0 = g.lb[0], nx = g.hi[0] - lb0 + 1, zpart = it.part, zparts = it.nparts;
    if (it.xparts > 1) {  // a part of the columns only
        const int w = (nx + it.xparts - 1) / it.xparts, xpart = it.part % it.xparts;
        zpart = it.part / it.xparts;
        zparts = it.nparts / it.xparts;
        lb0 += xpart * w;
        nx = max(0, min(w, nx - xpart * w));
    }
    const int lb1 = g.lb[1], kgmin = g.kgmin, ny = g.hi[1] - lb1 + 1, rlb = 1 - folded_rows(g);
    const int tot = 2 - 2 * kgmin;  // planes kgmin .. 1 - kgmin
    const int np = zpart < tot ? (tot - zpart + zparts - 1) / zparts : 0;
    const int kg0 = kgmin + zpart;
    double *C = sm;            // packed coefficients, or the CTA's moments
    double *Xt = C + nc;       // [lx][x]
    double *Yt = Xt + L * nx;  // [ly][y]
    double *Zt = Yt + L * ny;  // [lz][plane of this item]
    double *wsp = Zt + L * np;
    int *xidx = reinterpret_cast<int *>(wsp + kOrthoWarps * (33 * L + n2));
    int *yidx = xidx + nx;
    int *dec = yidx + ny;      // integrate: packed moment -> lz | (ly, lx) << 8
    int *rows_all = dec + nc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *sT = wsp + warp * (33 * L + n2);  // [ly][lane], rows of 33
    double *sC = sT + 33 * L;                 // Cxy, packed (ly, lx)
    int *rows = rows_all + warp * (1 - rlb) - rlb;  // igmin of the folded rows jf = rlb .. 0
    for (int t = tid; t < nx + ny + np; t += 32 * kOrthoWarps) {
        const int d = t < nx ? 0 : (t < nx + ny ? 1 : 2);
        const int gi = d == 0 ? t : (d == 1 ? t - nx : t - nx - ny);
        const int gg = d == 0 ? lb0 + gi : (d == 1 ? lb1 + gi : kg0 + gi * zparts);
        const int n = d == 0 ? nx : (d == 1 ? ny : np);
        double *tab = (d == 0 ? Xt : (d == 1 ? Yt : Zt)) + gi;
        const double u = (double)gg * lv.dh[d][d] - g.off[d];
        double e = exp(-g.zetp * u * u);
        for (int k = 0; k < L; k++) {
            tab[k * n] = e;
            e *= u;
        }
        if (d < 2)
            (d == 0 ? xidx : yidx)[gi] =
                axis_index(lv.periodic[d], g.cc[d], gg, g.lb[d], lv.lb_grid[d], lv.npts[d], lv.ngrid[d]);
    }
    for (int t = tid; t < nc; t += 32 * kOrthoWarps) {
        if (!kAdj) {
            C[t] = coef[g.coef_off + t];
            continue;
        }
        C[t] = 0.0;
        int lz = 0, ly = 0, r = t;
        while (r >= nshell(lp - lz)) r -= nshell(lp - lz++);
        while (r > lp - lz - ly) r -= lp - lz - ly++ + 1;
        dec[t] = lz | ((ly * L - (ly * (ly - 1)) / 2 + r) << 8);
    }
    // this lane's (ly, lx) entries: with n2 <= 16 of them, np2 = 2^lg lanes share one
    int lg = 0;
    if (kAdj)
        while ((n2 << (lg + 1)) <= 32) lg++;
    int oly[kM2], olx[kM2];
#pragma unroll
    for (int m = 0; m < kM2; m++) {
        const int o = (lane >> lg) + 32 * m;
        int ly = 0, r = o;
        while (ly < L && r > lp - ly) r -= lp - ly++ + 1;
        oly[m] = o < n2 ? ly : -1;
        olx[m] = r;
    }
    double W[kAdj ? kMC : 1];
#pragma unroll
    for (int m = 0; m < (kAdj ? kMC : 1); m++) W[m] = 0.0;
    const SphereRule rule(g.radius, lv.dh[0][0], lv.dh[1][1], lv.dh[2][2]);
    const double *Xt0 = Xt - lb0;  // by cube offset
    const int *xidx0 = xidx - lb0;
    const int xlast = lb0 + nx - 1;
    const int *T0 = g.table_off >= 0 ? table + g.table_off : nullptr;
    const int gn0 = lv.ngrid[0], gn1 = lv.ngrid[1];
    __syncthreads();
    // Collocate with fewer planes than warps (a call with one pair): 2^lsub warps share a
    // plane's rows, T computed by each (36 planes of 36 x 36, one pair, L = 2: 9 CTAs of four
    // planes 14.3 us, 36 CTAs of one 9.0 us).
    const int lsub = kAdj || np > 2 ? 0 : 3 - np, sub = warp & ((1 << lsub) - 1);
    for (int turn = warp >> lsub; (kAdj ? turn - warp : turn) < np; turn += kOrthoWarps >> lsub) {
        const int pl = kAdj ? plane_of_turn(turn, np) : turn;
        if (kAdj && pl < 0) continue;
        const int kg = kg0 + pl * zparts, kf = fold(kg);
        const int k = axis_index(lv.periodic[2], g.cc[2], kg, g.lb[2], lv.lb_grid[2], lv.npts[2], lv.ngrid[2]);
        if (k < 0) {
            if (lane == 0) atomicOr(status, kStatOutOfWindow);
            continue;
        }
        // folded rows jgmin .. 0 of the plane and the plane's widest x range
        const int jgmin = T0 ? T0[1 + 2 * (kf - T0[0])] : -sphere_jmax_fast(rule, kf);
        const int *Tr = T0 ? T0 + 1 + 2 * (1 - T0[0]) + T0[2 + 2 * (kf - T0[0])] : nullptr;
        int wide = 1;
        __syncwarp();
        for (int jf = jgmin + lane; jf <= 0; jf += 32) {
            const int ig = Tr ? Tr[jf - jgmin] : -sphere_imax_fast(rule, kf, jf);
            rows[jf] = ig;
            wide = min(wide, ig);
        }
        wide = __reduce_min_sync(0xffffffffu, wide);
        const double *Zk = Zt + pl;
        if (!kAdj) {
#pragma unroll
            for (int m = 0; m < kM2; m++) {
                if (oly[m] < 0) continue;
                const int ly = oly[m], lx = olx[m];
                double s = 0.0;
                int base = 0;  // packed index of (lz, 0, 0)
                for (int lz = 0; lz <= lp - lx - ly; lz++) {
                    const int q = lp - lz;
                    s += C[base + ly * (q + 1) - (ly * (ly - 1)) / 2 + lx] * Zk[lz * np];
                    base += nshell(q);
                }
                sC[lane + 32 * m] = s;
            }
        }
        __syncwarp();
        double cxy[kAdj ? kM2 : 1];
#pragma unroll
        for (int m = 0; m < (kAdj ? kM2 : 1); m++) cxy[m] = 0.0;
        const int nrow = 2 - 2 * jgmin, xbeg = max(wide, lb0), xend = min(1 - wide, xlast);
        for (int c0 = xbeg; c0 <= xend;) {
            const int left = xend - c0 + 1;
            const int lw = kAdj && left > 24 ? 5 : (left > 8 ? 4 : 3);  // log2 of the block's columns
            // (blocks of at most 32, 16, 8 columns: collocate 461, 453, 540 us on the workload
            // above, integrate 485, 488, 536: fewer idle lanes at a row's ends, but T, or the sums
            // over the columns, anew per block.  Done for 32 columns at a time: collocate with
            // blocks of 16 453 -> 421 us, integrate with blocks of 32 only where more than 24
            // columns are left 456 -> 451; 592 -> 574 with two more powers)
            const int grp = lane >> lw, ng = 32 >> lw;          // the lane's row group
            const int ig = c0 + (lane & ((1 << lw) - 1));
            const bool in = ig <= xend;
            const int igf = fold(ig), xi = xidx0[min(ig, xlast)];
            double T[kAcc];
            if (!kAdj) {
                // T of 32 columns at a time, a lane each (an FP64 operation costs a warp the same
                // with half its lanes idle): two blocks of 16 share them
                const int off = (c0 - xbeg) & 31;
                if (off == 0) {
                    const double *xt = Xt0 + min(c0 + lane, xlast);
                    const double *c = sC;
                    __syncwarp();
                    for (int ly = 0; ly < L; ly++) {
                        double s = 0.0;
                        for (int lx = 0; lx < L - ly; lx++) s += c[lx] * xt[lx * nx];
                        c += L - ly;
                        sT[ly * 33 + lane] = s;
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int ly = 0; ly < kAcc; ly++) {
                    if (ly >= L) break;
                    T[ly] = sT[ly * 33 + off + (lane & ((1 << lw) - 1))];
                }
            } else {
#pragma unroll
                for (int ly = 0; ly < kAcc; ly++) T[ly] = 0.0;
            }
            constexpr int kU = kAdj ? 4 : 2;  // rows in flight per lane
            for (int r0 = grp + sub * kU * ng; r0 - grp < nrow; r0 += (kU * ng) << lsub) {
                bool act[kU];
                int jy[kU];
                int64_t at[kU];
                bool any = false;
#pragma unroll
                for (int u = 0; u < kU; u++) {
                    const int r = r0 + u * ng, jg = jgmin + min(r, nrow - 1);
                    jy[u] = jg - lb1;
                    act[u] = in && r < nrow && igf >= rows[fold(jg)];
                    const int yi = yidx[jy[u]];
                    if (act[u] && (xi < 0 || yi < 0)) {
                        atomicOr(status, kStatOutOfWindow);
                        act[u] = false;
                    }
                    at[u] = ((int64_t)k * gn1 + yi) * gn0 + xi;
                    any = any || act[u];
                }
                if (!__any_sync(0xffffffffu, any)) continue;
                double v[kU];
#pragma unroll
                for (int u = 0; u < kU; u++) v[u] = kAdj && act[u] ? grid[at[u]] : 0.0;
#pragma unroll
                for (int ly = 0; ly < kAcc; ly++) {
                    if (ly >= L) break;
#pragma unroll
                    for (int u = 0; u < kU; u++) {
                        const double y = Yt[ly * ny + jy[u]];
                        if (kAdj) T[ly] = fma(v[u], y, T[ly]);
                        else v[u] = fma(T[ly], y, v[u]);
                    }
                }
                if (!kAdj) {
#pragma unroll
                    for (int u = 0; u < kU; u++)
                        if (act[u]) atomicAdd(grid + at[u], v[u]);
                }
            }
            if (kAdj) {  // the row groups' sums, then cxy over the columns of (up to) two blocks
                const int off = (c0 - xbeg) & 31;
#pragma unroll
                for (int ly = 0; ly < kAcc; ly++) {
                    if (ly >= L) break;
                    double v = T[ly];
                    for (int o = 1 << lw; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (grp == 0) sT[ly * 33 + off + lane] = v;
                }
                if (off + (1 << lw) == 32 || left <= 1 << lw) {
                    __syncwarp();
                    const int n = off + min(left, 1 << lw);
                    const double *xw = Xt0 + (c0 - off);
#pragma unroll
                    for (int m = 0; m < kM2; m++) {
                        if (oly[m] < 0) continue;
                        const double *t = sT + oly[m] * 33, *x = xw + olx[m] * nx;
                        double s = cxy[m];
                        for (int i = lane & ((1 << lg) - 1); i < n; i += 1 << lg) s = fma(t[i], x[i], s);
                        cxy[m] = s;
                    }
                    __syncwarp();
                }
            }
            c0 += 1 << lw;
        }
        if (kAdj) {
            for (int o = 1; o < (1 << lg); o <<= 1) cxy[0] += __shfl_xor_sync(0xffffffffu, cxy[0], o);
#pragma unroll
            for (int m = 0; m < kM2; m++)
                if (oly[m] >= 0) sC[(lane >> lg) + 32 * m] = cxy[m];
            __syncwarp();
#pragma unroll
            for (int m = 0; m < kMC; m++) {
                const int t = lane + 32 * m;
                if (t < nc) W[m] = fma(sC[dec[t] >> 8], Zk[(dec[t] & 255) * np], W[m]);
            }
        }
    }
    if (kAdj) {
        for (int w = 0; w < kOrthoWarps; w++) {
            if (warp == w) {
#pragma unroll
                for (int m = 0; m < kMC; m++)
                    if (lane + 32 * m < nc) C[lane + 32 * m] += W[m];
            }
            __syncthreads();
        }
        put_moments(items[blockIdx.x], nc, ps, mom + (extra ? g.mom_ext_off : g.coef_off), [&](int t) { return C[t]; });
    }
}

// ---------------------------------------------------------------------------
// general cell, one CTA per item (every nparts-th plane of a pair's index box; row
// bounds: general_row, gpw_common.cuh)
// (one row of margin: a geometry update moves a box's extent by at most one)
int smem_general_fp64(const PairGeom &g, int extra) {
    const int L = g.lp + 1 + extra;
    const int ny = g.hi[1] - g.cc[1] + 2;
    return 8 * (L * L * L + L * L + ny * L) + 12 * ny;
}

template <bool kAdj>
__global__ void __launch_bounds__(256)
k_general_fp64(const PairGeom *__restrict__ geoms, const Fp64Item *__restrict__ items, int uparts,
             const LevelDev *__restrict__ levels,
               const double *__restrict__ coef, double *__restrict__ mom, PartSums ps, GridPtrs grids,
               int *status, int extra) {
    extern __shared__ double sm[];
    const Fp64Item it = items ? items[blockIdx.x] : Fp64Item{(int)blockIdx.x / uparts, (int)blockIdx.x % uparts, uparts, 1, -1};
    const PairGeom g = geoms[it.pair];
    const LevelDev &lv = levels[g.level];
    double *__restrict__ grid = grids.p[g.level];
    const int lp = g.lp + extra, L = lp + 1;
    const int64_t mom_off = extra ? g.mom_ext_off : g.coef_off;
    const int ny = g.hi[1] - g.cc[1] + 1;
    double *Q = sm;              // [k][j][i] dense
    double *Qjk = Q + L * L * L; // [j][i]
    double *Qj = Qjk + L * L;    // [row][i]
    int *rows = (int *)(Qj + ny * L);  // ismin, ismax, jidx
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarp = nthr >> 5;
    for (int t = tid; t < L * L * L; t += nthr) {
        const int i = t % L, j = (t / L) % L, k = t / (L * L);
        Q[t] = (!kAdj && i + j + k <= lp) ? coef[g.coef_off + pidx(lp, k, j, i)] : 0.0;
    }
    __syncthreads();
    int off[3];
    for (int d = 0; d < 3; d++) off[d] = imod(g.cc[d] + lv.lb_grid[d], lv.npts[d]);
    for (int kk = g.cc[2] + it.part; kk <= g.hi[2]; kk += it.nparts) {
        const double dk = rsub((double)kk, g.off[2]);
        const int kidx = lv.periodic[2] ? imod(kk, lv.npts[2]) : kk - g.cc[2] + off[2];
        if (kidx < 0 || kidx >= lv.ngrid[2]) {
            if (tid == 0) atomicOr(status, kStatOutOfWindow);
            continue;
        }
        if (!kAdj) {
            for (int t = tid; t < L * L; t += nthr) {
                const int i = t % L, j = t / L;
                double s = 0.0, p = 1.0;
                for (int k = 0; k <= lp - i - j; k++) {
                    s += Q[(k * L + j) * L + i] * p;
                    p *= dk;
                }
                Qjk[t] = s;
            }
            __syncthreads();
        }
        for (int t = tid; t < ny * L; t += nthr) {
            const int row = t / L, i = t % L;
            const int jj = g.cc[1] + row;
            const double dj = rsub((double)jj, g.off[1]);
            if (!kAdj) {
                double s = 0.0, p = 1.0;
                for (int j = 0; j <= lp - i; j++) {
                    s += Qjk[j * L + i] * p;
                    p *= dj;
                }
                Qj[t] = s;
            }
            if (i == 0) {
                int ismin = 0, ismax = -1;
                if (!general_row(lv.dh, g.off, dj, dk, g.radius, ismin, ismax)) { ismin = 0; ismax = -1; }
                rows[3 * row] = ismin;
                rows[3 * row + 1] = ismax;
                rows[3 * row + 2] = lv.periodic[1] ? imod(jj, lv.npts[1]) : jj - g.cc[1] + off[1];
            }
        }
        __syncthreads();
        for (int row = warp; row < ny; row += nwarp) {
            const int ismin = rows[3 * row], ismax = rows[3 * row + 1], jidx = rows[3 * row + 2];
            if (ismax < ismin) continue;
            if (jidx < 0 || jidx >= lv.ngrid[1]) {
                if (lane == 0) atomicOr(status, kStatOutOfWindow);
                continue;
            }
            const double dj = (double)(g.cc[1] + row) - g.off[1];
            const int64_t rowbase = ((int64_t)kidx * lv.ngrid[1] + jidx) * lv.ngrid[0];
            double acc[kNPow];
#pragma unroll
            for (int n = 0; n < kNPow; n++) acc[n] = 0.0;
            for (int ii = ismin + lane; ii <= ismax; ii += 32) {
                const int iidx = lv.periodic[0] ? imod(ii, lv.npts[0]) : ii - g.cc[0] + off[0];
                if (iidx < 0 || iidx >= lv.ngrid[0]) {
                    atomicOr(status, kStatOutOfWindow);
                    continue;
                }
                const double di = (double)ii - g.off[0];
                double r2 = 0.0;
                for (int c = 0; c < 3; c++) {
                    const double rc = di * lv.dh[0][c] + dj * lv.dh[1][c] + dk * lv.dh[2][c];
                    r2 += rc * rc;
                }
                const double e = exp(-g.zetp * r2);
                if (!kAdj) {
                    double s = 0.0, p = 1.0;
                    for (int n = 0; n < L; n++) {
                        s += Qj[row * L + n] * p;
                        p *= di;
                    }
                    atomicAdd(grid + rowbase + iidx, s * e);
                } else {
                    const double ve = grid[rowbase + iidx] * e;
                    double p = 1.0;
#pragma unroll
                    for (int n = 0; n < kNPow; n++) {
                        if (n < L) acc[n] += ve * p;
                        p *= di;
                    }
                }
            }
            if (kAdj) {
#pragma unroll
                for (int n = 0; n < kNPow; n++) {
                    double v = acc[n];
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    acc[n] = v;
                }
                if (lane == 0)
                    for (int n = 0; n < L; n++) Qj[row * L + n] = acc[n];
            }
        }
        __syncthreads();
        if (kAdj) {
            // Qjk[j][i] = sum_rows Qj[row][i] dj^j;  Q[k][j][i] += Qjk[j][i] dk^k
            for (int t = tid; t < L * L; t += nthr) {
                const int i = t % L, j = t / L;
                if (i + j > lp) continue;
                double s = 0.0;
                for (int row = 0; row < ny; row++) {
                    if (rows[3 * row + 1] < rows[3 * row]) continue;
                    const double dj = (double)(g.cc[1] + row) - g.off[1];
                    double p = 1.0;
                    for (int e = 0; e < j; e++) p *= dj;
                    s += Qj[row * L + i] * p;
                }
                double p = 1.0;
                for (int k = 0; k <= lp - i - j; k++) {
                    Q[(k * L + j) * L + i] += s * p;
                    p *= dk;
                }
            }
            __syncthreads();
        }
    }
    if (kAdj) {
        const uint32_t *dec = d_decode.e + d_decode_at(lp);
        put_moments(it, ncoef(lp), ps, mom + mom_off, [&](int t) {
            const uint32_t de = __ldg(dec + t);  // (k, j, i)
            return Q[((de & 15) * L + (de >> 4 & 15)) * L + (de >> 8 & 15)];
        });
    }
}


// ---------------------------------------------------------------------------
// General cell in float-float (the mixed path).  The value at a point of the index
// box is P(di, dj, dk) exp(-zetp r^2), r^2 = G00 di^2 + A1 di + A0 along a row (metric
// G = dh dh^T; A1, A0 per row in FP64, split to float-float); the row's i-range is the
// reference's quadratic (general_row_fast32, general_row_unsure), so the point set is the reference's.
//
// As k_ortho_fp64: a CTA (4 warps) takes an item, a warp a plane, 64 rows at a time, a
// lane a column i (blocks of 32, 16 or 8 columns):
//   collocate  T[j] = sum_i Qjk[j][i] di^i once per column, then Horner in dj per point;
//   integrate  T[j] += V E dj^j per point, lane-local; then over the columns and dk once
//              per 64 rows and plane (T through shared memory).
// Two rows share each instruction (packed float-float), and what meets FP64 (the grid's
// values) is converted on the integer pipe: the FP64 pipe takes 17 cycles per
// instruction, conversions included.  (One warp per row, points one at a time, shuffle
// reductions per row and conversions on the FP64 pipe: 6.84 ms to integrate and 3.86 ms
// to collocate 1500 pairs, l <= 4, 128^3; this form 3.98 and 3.21 ms.)  128 registers
// for four CTAs per SM: with 232 (two CTAs) 5.52 and 4.53 against 4.42 and 3.68 ms, the chains being long.
constexpr int kGenRows = 64;  // rows of a plane in hand

// a warp's working set (floats): row data, Qjk; integrate: T of the block's columns
__host__ __device__ constexpr int general_ff_warp_bytes(int L) {
    return kGenRows * (4 * 4 + 3 * 4) + 8 * nshell(L - 1) + 8 * 33 * L;
}
// its static part in front (per CTA): coefficients or moments, per-row powers base and
// grid row, the decode table
static int general_ff_cta_bytes(const PairGeom &g) {
    const int ny = g.hi[1] - g.cc[1] + 2;  // one row of margin: a geometry update moves a box's extent by at most one
    return 8 * ncoef(g.lp) + 4 * ncoef(g.lp) + 16 * (ny + 2) + 16 + 256;
}

__device__ __forceinline__ float2 ld2(const float *p) { return *reinterpret_cast<const float2 *>(p); }

__device__ __forceinline__ ff ff_shfl_xor(ff v, int o) {
    return {__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
}

template <bool kAdj>
__global__ void __launch_bounds__(32 * kOrthoWarps, 4)
k_general_ff(const PairGeom *__restrict__ geoms, const Fp64Item *__restrict__ items, int uparts,
             const LevelDev *__restrict__ levels, const double *__restrict__ coef, double *__restrict__ mom,
             PartSums ps, GridPtrs grids, int *status) {
    extern __shared__ double smd[];
    constexpr int kM2 = (kNPow * (kNPow + 1) / 2 + 31) / 32, kMC = ((kMaxLp + 1) * (kMaxLp + 2) * (kMaxLp + 3) / 6 + 31) / 32;
    const Fp64Item it = items ? items[blockIdx.x] : Fp64Item{(int)blockIdx.x / uparts, (int)blockIdx.x % uparts, uparts, 1, -1};
    const PairGeom &g = geoms[it.pair];
    const LevelDev &lv = levels[g.level];
    double *__restrict__ grid = grids.p[g.level];
    const int lp = g.lp, L = lp + 1, nc = ncoef(lp), n2 = nshell(lp);
    const int cc0 = g.cc[0], cc1 = g.cc[1], cc2 = g.cc[2];
    const int ny = g.hi[1] - cc1 + 1, ny2 = (ny + 1) & ~1;  // rows come in pairs
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // shared memory: per CTA, then per warp
    ff *Q = reinterpret_cast<ff *>(smd);              // packed (k, j, i): coefficients, or the CTA's moments
    float2 *exptab = reinterpret_cast<float2 *>(Q + nc);
    float *djh = reinterpret_cast<float *>(exptab + 32), *djn = djh + ny2, *djl = djn + ny2;  // dj, -dj.hi, -dj.lo
    int *jrow = reinterpret_cast<int *>(djl + ny2);   // grid row of the box row, -1 outside the window
    int *dec = jrow + ny2;                            // packed (k, j, i) -> k | (j, i) << 8
    float *wbase = reinterpret_cast<float *>(dec + ((nc + 1) & ~1));
    float *ws = wbase + warp * (general_ff_warp_bytes(L) / 4);
    float *a1h = ws, *a1l = a1h + kGenRows, *a0h = a1l + kGenRows, *a0l = a0h + kGenRows;
    int *i0 = reinterpret_cast<int *>(a0l + kGenRows), *i1 = i0 + kGenRows;
    ff *sC = reinterpret_cast<ff *>(i1 + 2 * kGenRows);  // Qjk, packed (j, i)
    ff *sT = sC + n2;                                    // [j][lane], rows of 33
    if (tid < 32) exptab[tid] = c_exp2_32[tid];
    int off[3];
    for (int d = 0; d < 3; d++) off[d] = imod(g.cc[d] + lv.lb_grid[d], lv.npts[d]);
    for (int r = tid; r < ny2; r += 32 * kOrthoWarps) {
        const ff dj = ff_from_double(rsub((double)(cc1 + r), g.off[1]));
        djh[r] = dj.hi;
        djn[r] = -dj.hi;
        djl[r] = -dj.lo;
        const int j = lv.periodic[1] ? imod(cc1 + r, lv.npts[1]) : r + off[1];
        jrow[r] = j < lv.ngrid[1] ? j : -1;
    }
    for (int t = tid; t < nc; t += 32 * kOrthoWarps) {
        Q[t] = kAdj ? ff{0.0f, 0.0f} : ff_from_double(coef[g.coef_off + t]);
        int k = 0, j = 0, r = t;
        while (r >= nshell(lp - k)) r -= nshell(lp - k++);
        while (r > lp - k - j) r -= lp - k - j++ + 1;
        dec[t] = k | ((j * L - (j * (j - 1)) / 2 + r) << 8);
    }
    // this lane's (j, i) entries of Qjk; with n2 <= 16 of them, 2^lg lanes share one
    int lg = 0;
    if (kAdj)
        while ((n2 << (lg + 1)) <= 32) lg++;
    int oj[kM2], oi[kM2];
#pragma unroll
    for (int m = 0; m < kM2; m++) {
        const int o = (lane >> lg) + 32 * m;
        int j = 0, r = o;
        while (j < L && r > lp - j) r -= lp - j++ + 1;
        oj[m] = o < n2 ? j : -1;
        oi[m] = r;
    }
    ff W[kAdj ? kMC : 1];
#pragma unroll
    for (int m = 0; m < (kAdj ? kMC : 1); m++) W[m] = ff{0.0f, 0.0f};
    // metric of the lattice steps
    auto met = [&](int a, int b) { return lv.dh[a][0] * lv.dh[b][0] + lv.dh[a][1] * lv.dh[b][1] + lv.dh[a][2] * lv.dh[b][2]; };
    const double G01 = met(0, 1), G02 = met(0, 2), G11 = met(1, 1), G12 = met(1, 2), G22 = met(2, 2);
    const ff g00 = ff_from_double(met(0, 0));
    __shared__ GeneralRow32 R32;
    __shared__ GeneralRowFF Rff;
    if (tid == 0) general_row_constants(lv.dh, R32, Rff);
    const float gi = (float)(g.off[0] - (double)cc0), gj = (float)(g.off[1] - (double)cc1), gk = (float)(g.off[2] - (double)cc2);
    const float r2f = (float)(g.radius * g.radius);
    const ff2n mz = ff2n_dup(ff_from_double(-g.zetp));
    const int gn0 = lv.ngrid[0], gn1 = lv.ngrid[1], np0 = lv.npts[0], per0 = lv.periodic[0];
    __syncthreads();
    const int np = (g.hi[2] - cc2 + it.nparts - it.part) / it.nparts;  // this item's planes
    for (int turn = warp; turn - warp < np; turn += kOrthoWarps) {
        const int pl = plane_of_turn(turn, np);
        if (pl < 0) continue;
        const int kk = cc2 + it.part + pl * it.nparts;
        const double dk = rsub((double)kk, g.off[2]);
        const int kidx = lv.periodic[2] ? imod(kk, lv.npts[2]) : kk - cc2 + off[2];
        if (kidx < 0 || kidx >= lv.ngrid[2]) {
            if (lane == 0) atomicOr(status, kStatOutOfWindow);
            continue;
        }
        const ff dkf = ff_from_double(dk);
        const float dkc = (float)(kk - cc2) - gk;
        __syncwarp();
        if (!kAdj) {  // Qjk[j][i] = sum_k Q[k][j][i] dk^k (Horner)
#pragma unroll
            for (int m = 0; m < kM2; m++) {
                if (oj[m] < 0) continue;
                const int j = oj[m], i = oi[m], top = lp - i - j;
                int base = nc;  // packed index of (k + 1, 0, 0)
                for (int k = lp; k > top; k--) base -= nshell(lp - k);
                ff s = {0.0f, 0.0f};
                for (int k = top; k >= 0; k--) {
                    const int q = lp - k;
                    base -= nshell(q);
                    s = ff_fma(s, dkf, Q[base + j * (q + 1) - (j * (j - 1)) / 2 + i]);
                }
                sC[lane + 32 * m] = s;
            }
        }
        ff cji[kAdj ? kM2 : 1];
#pragma unroll
        for (int m = 0; m < (kAdj ? kM2 : 1); m++) cji[m] = ff{0.0f, 0.0f};
        for (int r0 = 0; r0 < ny; r0 += kGenRows) {
            const int nr = min(kGenRows, ny - r0);
            __syncwarp();
            int imin = INT32_MAX, imax = INT32_MIN;
            for (int r = lane; r < ((nr + 1) & ~1); r += 32) {
                int ismin = 1, ismax = 0;
                if (r < nr) {
                    const int jj = cc1 + r0 + r;
                    bool unsure;
                    bool some = general_row_fast32(R32, gi, gj, gk, (float)(r0 + r) - gj, dkc, r2f, cc0, ismin, ismax,
                                                   unsure);
                    if (unsure)
                        some = general_row_unsure(&Rff, lv.dh, g.off, cc0, jj, kk, g.radius, ismin, ismax);
                    if (!some || ismin > ismax) {
                        ismin = 1;
                        ismax = 0;
                    } else if (jrow[r0 + r] < 0) {
                        atomicOr(status, kStatOutOfWindow);
                        ismin = 1;
                        ismax = 0;
                    } else {  // (rows without points need no constants)
                        const double dj = rsub((double)jj, g.off[1]);
                        imin = min(imin, ismin);
                        imax = max(imax, ismax);
                        const ff a1 = ff_from_double_bits(2.0 * (G01 * dj + G02 * dk));
                        const ff a0 = ff_from_double_bits(G11 * dj * dj + 2.0 * G12 * dj * dk + G22 * dk * dk);
                        a1h[r] = a1.hi;
                        a1l[r] = a1.lo;
                        a0h[r] = a0.hi;
                        a0l[r] = a0.lo;
                    }
                }
                i0[r] = ismin;
                i1[r] = ismax;
            }
            imin = __reduce_min_sync(0xffffffffu, imin);
            imax = __reduce_max_sync(0xffffffffu, imax);
            __syncwarp();
            for (int c0 = imin; c0 <= imax;) {
                const int left = imax - c0 + 1, lw = left > 16 ? 5 : (left > 8 ? 4 : 3);
                const int grp = lane >> lw, ng = 32 >> lw;
                const int ii = c0 + (lane & ((1 << lw) - 1));
                const int iidx = per0 ? imod(ii, np0) : ii - cc0 + off[0];
                const bool iok = iidx >= 0 && iidx < gn0;
                const ff di = ff_from_double(rsub((double)ii, g.off[0]));
                const ff2n din = ff2n_dup(di);
                const ff2 gd = ff2_dup(ff_mul(g00, di));
                ff2 T[kNPow];  // collocate: the column's value twice; integrate: sums over even and odd rows
#pragma unroll
                for (int j = 0; j < kNPow; j++) T[j] = ff2{f2(0.0f), f2(0.0f)};
                if (!kAdj) {
                    const ff *c = sC;
#pragma unroll
                    for (int j = 0; j < kNPow; j++) {
                        if (j >= L) break;
                        ff s = c[lp - j];
                        for (int i = lp - j - 1; i >= 0; i--) s = ff_fma(s, di, c[i]);
                        c += L - j;
                        T[j] = ff2_dup(s);
                    }
                }
                for (int rp = grp; 2 * (rp - grp) < nr; rp += ng) {  // row pairs
                    const int r = min(2 * rp, (nr - 1) & ~1);
                    const int2 lo2 = *reinterpret_cast<const int2 *>(i0 + r), hi2 = *reinterpret_cast<const int2 *>(i1 + r);
                    const bool mine = 2 * rp < nr;
                    bool act0 = mine && ii >= lo2.x && ii <= hi2.x, act1 = mine && ii >= lo2.y && ii <= hi2.y;
                    if ((act0 || act1) && !iok) {
                        atomicOr(status, kStatOutOfWindow);
                        act0 = act1 = false;
                    }
                    if (!__any_sync(0xffffffffu, act0 || act1)) continue;
                    const int2 jr = *reinterpret_cast<const int2 *>(jrow + r0 + r);
                    double *const p0 = grid + ((int64_t)kidx * gn1 + jr.x) * gn0 + iidx;
                    double *const p1 = grid + ((int64_t)kidx * gn1 + jr.y) * gn0 + iidx;
                    double v0 = 1.0, v1 = 1.0;  // (zero would take the split's slow path)
                    if (kAdj) {
                        if (act0) v0 = __ldg(p0);
                        if (act1) v1 = __ldg(p1);
                    }
                    const ff2 t = ff2_add(gd, ff2{ld2(a1h + r), ld2(a1l + r)});
                    const ff2 r2 = ff2_fma(t, din, ff2{ld2(a0h + r), ld2(a0l + r)});
                    const ff2 e = ff2_exp(ff2_mul(r2, mz), exptab);
                    const ff2n dj = {ld2(djh + r0 + r), ld2(djn + r0 + r), ld2(djl + r0 + r)};
                    if (!kAdj) {
                        ff2 s = {f2(0.0f), f2(0.0f)};
#pragma unroll
                        for (int j = kNPow - 1; j >= 0; j--) {
                            if (j >= L) continue;
                            s = j == L - 1 ? T[j] : ff2_fma(s, dj, T[j]);
                        }
                        const ff2 v = ff2_mul(s, ff2n_of(e));
                        if (act0) atomicAdd(p0, ff_to_double_bits(ff{v.hi.x, v.lo.x}));
                        if (act1) atomicAdd(p1, ff_to_double_bits(ff{v.hi.y, v.lo.y}));
                    } else {
                        ff2 w = ff2_mul(ff2_pair(ff_from_double_bits(v0), ff_from_double_bits(v1)), ff2n_of(e));
                        if (!act0) w.hi.x = w.lo.x = 0.0f;
                        if (!act1) w.hi.y = w.lo.y = 0.0f;
#pragma unroll
                        for (int j = 0; j < kNPow; j++) {
                            if (j >= L) break;
                            T[j] = ff2_add(T[j], w);
                            w = ff2_mul(w, dj);
                        }
                    }
                }
                if (kAdj) {  // cji[j][i] += sum over the block's lanes of T[j] di^i
                    for (int i = 0; i < L; i++) {  // one power of di at a time (T di^i for j <= lp - i)
                        __syncwarp();
#pragma unroll
                        for (int j = 0; j < kNPow; j++) {
                            if (j > lp - i) break;
                            const ff v = i == 0 ? ff_add(ff{T[j].hi.x, T[j].lo.x}, ff{T[j].hi.y, T[j].lo.y})
                                                : ff_mul(ff{T[j].hi.x, T[j].lo.x}, di);
                            T[j].hi.x = v.hi;
                            T[j].lo.x = v.lo;
                            sT[j * 33 + lane] = v;
                        }
                        __syncwarp();
#pragma unroll
                        for (int m = 0; m < kM2; m++) {
                            if (oj[m] < 0 || oi[m] != i) continue;
                            ff s = cji[m];
                            for (int l = lane & ((1 << lg) - 1); l < 32; l += 1 << lg) s = ff_add(s, sT[oj[m] * 33 + l]);
                            cji[m] = s;
                        }
                    }
                    __syncwarp();
                }
                c0 += 1 << lw;
            }
        }
        if (kAdj) {  // W[k][j][i] += Qjk[j][i] dk^k
            for (int o = 1; o < (1 << lg); o <<= 1) cji[0] = ff_add(cji[0], ff_shfl_xor(cji[0], o));
            __syncwarp();
#pragma unroll
            for (int m = 0; m < kM2; m++)
                if (oj[m] >= 0) sC[(lane >> lg) + 32 * m] = cji[m];
            __syncwarp();
#pragma unroll
            for (int m = 0; m < kMC; m++) {
                const int t = lane + 32 * m;
                if (t >= nc) continue;
                const int k = dec[t] & 255;
                ff dp = {1.0f, 0.0f};
                for (int e = 0; e < k; e++) dp = ff_mul(dp, dkf);
                W[m] = ff_fma(sC[dec[t] >> 8], dp, W[m]);
            }
        }
    }
    if (kAdj) {
        for (int w = 0; w < kOrthoWarps; w++) {
            if (warp == w) {
#pragma unroll
                for (int m = 0; m < kMC; m++)
                    if (lane + 32 * m < nc) Q[lane + 32 * m] = ff_add(Q[lane + 32 * m], W[m]);
            }
            __syncthreads();
        }
        put_moments(it, nc, ps, mom + g.coef_off, [&](int t) { return (double)Q[t].hi + (double)Q[t].lo; });
    }
}

// ---------------------------------------------------------------------------
// bytes: the CTA's whole shared memory; a kernel's static shared arrays come out of it
static cudaError_t set_smem(const void *fn, int bytes) {
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, fn);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes - (int)a.sharedSizeBytes);
}

// Opt every dynamic-shared-memory kernel of this file into the device maximum once,
// so that launches (and CUDA graph capture) need no attribute calls.
cudaError_t fp64_kernel_attributes(int smem_max) {
    const void *fns[] = {(const void *)k_prep, (const void *)k_backtransform,
                         (const void *)k_ortho_fp64<false, kNPow>, (const void *)k_ortho_fp64<true, kNPow>,
                         (const void *)k_ortho_fp64<true, kNPowB>,
                         (const void *)k_general_fp64<false>, (const void *)k_general_fp64<true>,
                         (const void *)k_general_ff<false>, (const void *)k_general_ff<true>};
    for (const void *fn : fns) {
        cudaError_t e = set_smem(fn, smem_max);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_prep(const TaskSet &ts, const double *d_pab, cudaStream_t s) {
    if (ts.ntasks == 0) return cudaSuccess;
    const int smem = smem_prep(ts.max_A, ts.max_B);
    ts.n_kernels++;
    k_prep<<<(unsigned)ts.ntasks, 128, smem, s>>>(ts.d_geom, ts.plan->d_levels, ts.plan->d_tmat,
                                                  ts.tau, d_pab, ts.d_coef);
    return cudaGetLastError();
}

// The items of the FP64 launches and of the float-float general-cell kernel (1500
// pairs of a general cell, 128^3, collocate + integrate: one CTA per pair 38.1 ms, most
// of it the tail of the largest boxes; with items and the same kernel 10.7 ms).  A pair
// is divided into parts (interleaved planes, so that parts cost alike) where it holds
// more than a given part of an even per-CTA share of all cube points, down to one plane
// per warp.  The number of planes is not needed exactly: a geometry update may move a
// general box's extent by one.
//
// Parts of at most 1/kWaves of a CTA's share.  Orthorhombic: a part costs a CTA's tables and
// (integrate) the sum over its warps, and the largest parts run first (integrate and
// collocate of 1000 pairs, 64^3: 443 and 418 us; 8 waves in the pairs' order 450 and 423;
// two more powers 569 and 543 against 571 and 549; 16 waves 462 and 421).  General cells,
// whose CTAs set little up: 4.04 and 3.28 ms for 1500 pairs on 128^3, mixed, with 16 waves in
// the pairs' order, 4.15 and 3.32 sorted, 4.15 and 3.49 with 8 waves.
constexpr int kWavesOrtho = 7, kWavesGeneral = 16, kCtas = 4;
constexpr double kLeast = 16384.0;  // points x powers: below this a part is mostly tables and set-up

Fp64Planner::Fp64Planner(TaskSet &t, double total, int sms, int smem_limit_)
    : ts(t), smem_limit(smem_limit_),
      target{std::max(kLeast, total / ((double)sms * kCtas) / kWavesGeneral),
             std::max(kLeast, total / ((double)sms * kCtas) / kWavesOrtho)},
      first(kClasses + 1, 0) {
    pairs.reserve((size_t)ts.ntasks);
}

void Fp64Planner::add(const PairGeom &g) {
    const int planes = g.ortho ? 2 - 2 * g.kgmin : g.ext0[2];
    const int most = std::max(1, (planes + kOrthoWarps - 1) / kOrthoWarps);
    const double cost = (double)g.cost * (g.lp + 1);
    int parts = std::max(1, (int)std::min<double>(most, std::ceil(cost / target[g.ortho ? 1 : 0])));
    int xp = 1;
    if (g.ortho) {
        int zp = parts;
        if (fit_ortho_item(g, 2, smem_limit, zp, xp)) {
            parts = zp;
        } else {  // thousands of rows: no gradients
            xp = 1;
            fit_ortho_item(g, 0, smem_limit, parts, xp);
            ts.fp64_ext_fits = false;
        }
        ts.fp64_smem = std::max(ts.fp64_smem, smem_ortho_item(g, 0, parts, xp) - kOrthoStatic);
        ts.fp64_smem_ext = std::max(ts.fp64_smem_ext, smem_ortho_item(g, 2, parts, xp) - kOrthoStatic);
        parts *= xp;
        ts.fp64_ortho += parts;
    } else {
        ts.fp64_smem_gen = std::max(ts.fp64_smem_gen, smem_general_fp64(g));
        // (fits: the test of smem_general_ff_limit, 16 L + 36 bytes a row, is the narrower one)
        ts.fp64_smem_gen_ext = std::max(ts.fp64_smem_gen_ext, smem_general_fp64(g, 2));
        ts.fp64_general += parts;
    }
    if (parts > 1) ts.fp64_slots += parts;
    // class of the items' cost: a factor 2^(1/4) or so, from the float's leading bits
    const float c = (float)(cost / parts);
    unsigned bits;
    memcpy(&bits, &c, sizeof bits);
    const int cls = kClasses - 1 - (int)std::min(bits >> 21, (unsigned)kClasses - 1);
    if (g.ortho) first[cls + 1] += parts;
    pairs.push_back(Pair{parts, xp, g.ortho ? cls : -1});
}

void Fp64Planner::write(Fp64Item *items) {
    for (int c = 0; c < kClasses; c++) first[c + 1] += first[c];
    int64_t at_gen = ts.fp64_ortho;
    int slot = 0;
    for (size_t k = 0; k < pairs.size(); k++) {
        const Pair &p = pairs[k];
        int64_t &at = p.cls >= 0 ? first[p.cls] : at_gen;
        for (int i = 0; i < p.parts; i++)
            items[at++] = Fp64Item{(int)k, i, p.parts, p.xparts, p.parts > 1 ? slot++ : -1};
    }
}

static cudaError_t launch_fp64_impl(const TaskSet &ts, const GridPtrs &g, bool adj, int extra, double *mom,
                                    cudaStream_t s) {
    const Plan &P = *ts.plan;
    const PartSums ps = {extra ? ts.d_parts_ext : static_cast<double *>(ts.d_scratch), ts.d_ticket,
                         ncoef(ts.max_lp + extra)};
    if (ts.fp64_ortho > 0) {
        ProfScope prof(ts, s);
        const unsigned n = (unsigned)ts.fp64_ortho;
        if (adj && extra)
            k_ortho_fp64<true, kNPowB><<<n, 32 * kOrthoWarps, ts.fp64_smem_ext, s>>>(
                ts.d_geom, ts.d_fp64_items, 1, 1, P.d_levels, ts.d_table, ts.d_coef, mom, ps, g, ts.d_status, extra);
        else if (adj)
            k_ortho_fp64<true, kNPow><<<n, 32 * kOrthoWarps, ts.fp64_smem, s>>>(
                ts.d_geom, ts.d_fp64_items, 1, 1, P.d_levels, ts.d_table, ts.d_coef, mom, ps, g, ts.d_status, 0);
        else
            k_ortho_fp64<false, kNPow><<<n, 32 * kOrthoWarps, ts.fp64_smem, s>>>(
                ts.d_geom, ts.d_fp64_items, 1, 1, P.d_levels, ts.d_table, ts.d_coef, mom, ps, g, ts.d_status, 0);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (ts.fp64_general > 0) {
        ProfScope prof(ts, s);
        const unsigned n = (unsigned)ts.fp64_general;
        const Fp64Item *items = ts.d_fp64_items + ts.fp64_ortho;
        if (adj)
            k_general_fp64<true><<<n, 256, extra ? ts.fp64_smem_gen_ext : ts.fp64_smem_gen, s>>>(
                ts.d_geom, items, 1, P.d_levels, ts.d_coef, mom, ps, g, ts.d_status, extra);
        else
            k_general_fp64<false><<<n, 256, ts.fp64_smem_gen, s>>>(ts.d_geom, items, 1, P.d_levels, ts.d_coef, mom, ps, g,
                                                                  ts.d_status, 0);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// general-cell pairs of a mixed call: the float-float kernel
int smem_general_ff(const PairGeom &g) {
    return general_ff_cta_bytes(g) + kOrthoWarps * general_ff_warp_bytes(g.lp + 1);
}
// the boxes that the float-float path accepts: what one CTA held when it kept all rows
// of a plane in shared memory
int smem_general_ff_limit(const PairGeom &g) {
    const int L = g.lp + 1;
    const int ny = g.hi[1] - g.cc[1] + 2;
    return 8 * (L * L * L + L * L + 2 * ny * L + 3 * ny) + 12 * ny;
}

// one launch over the items of all general-cell pairs
cudaError_t launch_general_ff(const TaskSet &ts, const GridPtrs &g, bool adj, cudaStream_t s) {
    if (ts.gen_count == 0) return cudaSuccess;
    const PartSums ps = {static_cast<double *>(ts.d_scratch), ts.d_ticket, ncoef(ts.max_lp)};
    ProfScope prof(ts, s);
    const unsigned n = (unsigned)ts.fp64_general;
    const Fp64Item *items = ts.d_fp64_items + ts.fp64_ortho;
    if (adj)
        k_general_ff<true><<<n, 32 * kOrthoWarps, ts.gen_smem, s>>>(ts.d_geom, items, 1, ts.plan->d_levels, ts.d_coef, ts.d_mom, ps, g,
                                                      ts.d_status);
    else
        k_general_ff<false><<<n, 32 * kOrthoWarps, ts.gen_smem, s>>>(ts.d_geom, items, 1, ts.plan->d_levels, ts.d_coef, ts.d_mom, ps, g,
                                                       ts.d_status);
    return cudaGetLastError();
}

cudaError_t launch_moments_fp64(const TaskSet &ts, const GridPtrs &g, int extra, double *out, cudaStream_t s) {
    return launch_fp64_impl(ts, g, true, extra, out, s);
}

// n pairs without a task set: every pair in zparts xparts parts
cudaError_t launch_pairs_fp64(const PairGeom *d_geoms, const LevelDev *d_levels, const double *d_tmat,
                              double *d_coef, int *d_status, int n, int zparts, int xparts, int tau, int max_A, int max_B,
                              int smem_coll, const double *d_pab, double *d_grid, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_prep<<<(unsigned)n, 128, smem_prep(max_A, max_B), s>>>(d_geoms, d_levels, d_tmat, tau, d_pab, d_coef);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    GridPtrs g;
    for (int l = 0; l < GPW_MAX_LEVELS; l++) g.p[l] = d_grid;
    const int parts = zparts * xparts;
    k_ortho_fp64<false, kNPow><<<(unsigned)(n * parts), 32 * kOrthoWarps, smem_coll - kOrthoStatic, s>>>(
        d_geoms, nullptr, parts, xparts, d_levels, nullptr, d_coef, nullptr, PartSums{}, g, d_status, 0);
    return cudaGetLastError();
}

// one plane per CTA (orthorhombic), four planes per CTA (general cell)
int fp64_single_parts(const PairGeom &g) {
    return std::max(1, g.ortho ? 2 - 2 * g.kgmin : (g.ext0[2] + kOrthoWarps - 1) / kOrthoWarps);
}

// One pair from raw device pointers, orthorhombic (with its cube list in d_table
// when the pair has one) or general cell: set-up, then the FP64 collocation.
cudaError_t launch_one_fp64(const PairGeom &g, const PairGeom *d_geom, const LevelDev *d_levels, const double *d_tmat,
                            const int *d_table, double *d_coef, int *d_status, int func, const double *d_pab,
                            double *d_grid, int smem_limit, cudaStream_t s) {
    k_prep<<<1, 128, smem_prep(g.la_max, g.lb_max), s>>>(d_geom, d_levels, d_tmat, func, d_pab, d_coef);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    GridPtrs gp;
    for (int l = 0; l < GPW_MAX_LEVELS; l++) gp.p[l] = d_grid;
    int parts = fp64_single_parts(g), xparts = 1;
    if (g.ortho) fit_ortho_item(g, 0, smem_limit, parts, xparts);
    if (g.ortho)
        k_ortho_fp64<false, kNPow><<<(unsigned)(parts * xparts), 32 * kOrthoWarps,
                                     smem_ortho_item(g, 0, parts, xparts) - kOrthoStatic, s>>>(
            d_geom, nullptr, parts * xparts, xparts, d_levels, d_table, d_coef, nullptr, PartSums{}, gp, d_status, 0);
    else
        k_general_fp64<false><<<(unsigned)parts, 256, smem_general_fp64(g), s>>>(d_geom, nullptr, parts, d_levels,
                                                                               d_coef, nullptr, PartSums{}, gp, d_status, 0);
    return cudaGetLastError();
}

cudaError_t launch_collocate_fp64(const TaskSet &ts, const GridPtrs &g, cudaStream_t s) {
    return launch_fp64_impl(ts, g, false, 0, ts.d_mom, s);
}

cudaError_t launch_integrate_fp64(const TaskSet &ts, const GridPtrs &g, cudaStream_t s) {
    return launch_fp64_impl(ts, g, true, 0, ts.d_mom, s);
}

cudaError_t launch_backtransform(const TaskSet &ts, const double *d_mom, int extra, double *d_hab,
                                 cudaStream_t s) {
    if (ts.ntasks == 0) return cudaSuccess;
    const int smem = smem_prep(ts.max_A, ts.max_B);
    ts.n_kernels++;
    k_backtransform<<<(unsigned)ts.ntasks, 128, smem, s>>>(ts.d_geom, ts.plan->d_levels,
                                                           ts.plan->d_tmat, ts.tau, d_mom, extra, d_hab);
    return cudaGetLastError();
}

}  // namespace gpw
