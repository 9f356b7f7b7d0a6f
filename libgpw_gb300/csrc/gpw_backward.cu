// Backward pass of E = sum over levels of <V, rho>: gradients with respect to
// the density blocks (the integrate path), the two centres and the two
// exponents of every pair, FP64.
//
// With phi_a = (x-ax)^lx (y-ay)^ly (z-az)^lz exp(-za |r-a|^2):
//   d phi_a / d ax  = -lx phi_{a-ex} + 2 za phi_{a+ex}
//   d phi_a / d za  = -(phi_{a+2ex} + phi_{a+2ey} + phi_{a+2ez})
// (the derivative rule the reference applies for tau, grid_base_ref_c.cc:77-140),
// so every gradient is a combination of pair integrals I(a', b) = <V, phi_a' phi_b>
// with |a'| <= la_max + 2.  Those come from the moments of V against the product
// Gaussian up to degree lp + 2 (one more integrate pass, the 1-D tables are
// recomputed), re-centred on a and b with the binomials of grid_base_ref_c.cc:195-231.
// The derivative functions (tau and phi_a d phi_b - d phi_a phi_b) are sums over
// their local block P'(a', b') of P' phi_a' phi_b' (shells l +- 1, coefficients
// that depend on the exponents): the same rule applies per local element, plus
// dP'/dzeta I(a', b') for the exponent gradients.
#include <cuda_runtime.h>

#include "gpw_coef.cuh"
#include "gpw_internal.h"

namespace gpw {

constexpr int kBI = kMaxL + 4;          // components up to l_max + 1 (local block) + 2
constexpr int kBK = 2 * kBI - 1;

constexpr int kBWarps = 12;  // 3 axes x (centre a, centre b) x 2 halves of the local block

struct BwdSmem {
    double al[3][kBI][kBI][kBK];
    double W[(kNPowB * (kNPowB + 1) * (kNPowB + 2)) / 6];  // moments up to degree lp + 2
    short row[kNPowB][kNPowB];                             // packed index of (lz, ly, 0)
    double red[8][kBWarps];
};

__device__ __forceinline__ double pair_integral(const BwdSmem &s, const int a[3], const int b[3]) {
    const double *ax = s.al[0][a[0]][b[0]];
    double acc = 0.0;
    for (int lz = 0; lz <= a[2] + b[2]; lz++) {
        double accz = 0.0;
        for (int ly = 0; ly <= a[1] + b[1]; ly++) {
            const double *W = s.W + s.row[lz][ly];
            double accy = 0.0;
            for (int lx = 0; lx <= a[0] + b[0]; lx++) accy += ax[lx] * W[lx];
            accz += s.al[1][a[1]][b[1]][ly] * accy;
        }
        acc += s.al[2][a[2]][b[2]][lz] * accz;
    }
    return acc;
}

// One CTA per pair.  The pair integrals are dependent FP64 chains, so they are spread
// over 12 warps: a warp takes one axis d, one centre and every second element of the
// local block, up to three integrals per element (a +- e_d, a + 2 e_d).  (Four warps
// with an element's 18 integrals to a thread and the packed index searched in the inner
// loop: 459 us for 2000 pairs, l <= 2.)
__global__ void __launch_bounds__(32 * kBWarps)
k_backward_epilogue(const PairGeom *__restrict__ geoms, const LevelDev *__restrict__ levels,
                    const double *__restrict__ tmat, const double *__restrict__ mom_ext, int func,
                    const double *__restrict__ pab, double *dra, double *drb, double *dza, double *dzb) {
    __shared__ BwdSmem s;
    const PairGeom &g = geoms[blockIdx.x];
    const int tid = threadIdx.x;
    const int lpe = g.lp + 2;
    const int ia = g.la_max + 2, jb = g.lb_max + 2;  // local shells (after the function's shift)
    // re-centring binomials (x-a)^i (x-b)^j = sum_k al[i][j][k] (x-p)^k
    for (int t = tid; t < 3 * (ia + 1) * (jb + 1); t += blockDim.x) {
        const int j = t % (jb + 1), i = (t / (jb + 1)) % (ia + 1), ax = t / ((jb + 1) * (ia + 1));
        const double pa = g.rp[ax] - g.ra[ax], pb = g.rp[ax] - g.rb[ax];
        double *out = s.al[ax][i][j];
        // one multiplication by (u + pa) or (u + pb) at a time, as fill_alpha
        out[0] = 1.0;
        for (int k = 1; k < kBK; k++) out[k] = 0.0;
        for (int m = 0; m < i + j; m++) {
            const double c = m < i ? pa : pb;
            out[m + 1] = out[m];
            for (int k = m; k >= 1; k--) out[k] = fma(c, out[k], out[k - 1]);
            out[0] *= c;
        }
    }
    // Cartesian moments (general cells: transpose of the lattice transform)
    const int nc = ncoef(lpe);
    for (int t = tid; t < kNPowB * kNPowB; t += blockDim.x) {
        const int lz = t / kNPowB, ly = t - lz * kNPowB;
        s.row[lz][ly] = (short)(lz + ly <= lpe ? pidx(lpe, lz, ly, 0) : 0);
    }
    const double *Wsrc = mom_ext + g.mom_ext_off;
    for (int t = tid; t < nc; t += blockDim.x) {
        if (g.ortho) {
            s.W[t] = Wsrc[t];
            continue;
        }
        int lz = 0, ly = 0, lx = 0, r = t;
        for (lz = 0; lz <= lpe; lz++) {
            const int cnt = ((lpe - lz + 1) * (lpe - lz + 2)) / 2;
            if (r < cnt) break;
            r -= cnt;
        }
        const int q = lpe - lz;
        for (ly = 0; ly <= q; ly++) {
            if (r <= q - ly) break;
            r -= q - ly + 1;
        }
        lx = r;
        const int n = lx + ly + lz;
        const int NT = ncoef(kMaxLp);
        const double *Tm = tmat + levels[g.level].tmat_off;
        const int col = pidx(kMaxLp, lz, ly, lx);
        double acc = 0.0;
        for (int k = 0; k <= n; k++)
            for (int j = 0; j <= n - k; j++) acc += Tm[(int64_t)pidx(kMaxLp, k, j, n - k - j) * NT + col] * Wsrc[pidx(lpe, k, j, n - k - j)];
        s.W[t] = acc;
    }
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5;
    const int d = warp % 3, side = (warp / 3) % 2, half = warp / 6;
    double gc = 0.0, gz[2] = {0.0, 0.0};  // this centre's derivative along d; dza, dzb
    const int a0 = ncoset(g.la_min - 1), b0 = ncoset(g.lb_min - 1);  // the local block's shells
    const int na = ncoset(g.la_max) - a0, nb = ncoset(g.lb_max) - b0;
    for (int t = 2 * lane + half; t < na * nb; t += 64) {
        const int jco = b0 + t / na, ico = a0 + t % na;
        int c[2][3];
        coset_decode(ico, c[0][0], c[0][1], c[0][2]);
        coset_decode(jco, c[1][0], c[1][1], c[1][2]);
        double dP[2];  // dP'/dzeta, dP'/dzetb of the local element
        const double P = local_entry(g, func, pab, c[0], c[1], &dP[0], &dP[1]);
        if (d == 0 && side == 0 && (dP[0] != 0.0 || dP[1] != 0.0)) {
            const double I0 = pair_integral(s, c[0], c[1]);
            gz[0] += dP[0] * I0;
            gz[1] += dP[1] * I0;
        }
        if (P == 0.0) continue;
        const int l = c[side][d];
        const double zeta = side == 0 ? g.zeta : g.zetb;
        c[side][d] = l + 1;
        double v = 2.0 * zeta * pair_integral(s, c[0], c[1]);
        if (l > 0) {
            c[side][d] = l - 1;
            v -= l * pair_integral(s, c[0], c[1]);
        }
        gc += P * v;
        c[side][d] = l + 2;
        const double q = P * pair_integral(s, c[0], c[1]);
        gz[0] -= side == 0 ? q : 0.0;
        gz[1] -= side == 0 ? 0.0 : q;
    }
    // block reduction: the warps' three sums, then the eight gradients
    double r3[3] = {gc, gz[0], gz[1]};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        for (int o = 16; o > 0; o >>= 1) r3[k] += __shfl_xor_sync(0xffffffffu, r3[k], o);
        if (lane == 0) s.red[k][warp] = r3[k];
    }
    __syncthreads();
    if (tid < 8) {
        double v = 0.0;
        if (tid < 6) {  // dRa, dRb: the two halves of (axis, centre)
            v = s.red[0][tid] + s.red[0][tid + 6];
        } else {
            for (int w = 0; w < kBWarps; w++) v += s.red[tid - 5][w];
        }
        v *= g.prefactor;
        const int64_t t = g.task;
        if (tid < 3) {
            if (dra) dra[3 * t + tid] = v;
        } else if (tid < 6) {
            if (drb) drb[3 * t + tid - 3] = v;
        } else if (tid == 6) {
            if (dza) dza[t] = v;
        } else {
            if (dzb) dzb[t] = v;
        }
    }
}

// orthorhombic moments go to degree lp + 2 <= kMaxLpB; general cells map them through
// the lattice transform, which is built to degree kMaxLp; their tables must fit a CTA
bool backward_supported(const TaskSet &ts) {
    for (int64_t k = ts.gen_first; k < ts.gen_first + ts.gen_count; k++)
        if (ts.h_geom[k].lp + 2 > kMaxLp) return false;
    return ts.fp64_ext_fits && ts.max_lp + 2 <= kMaxLpB;
}

cudaError_t launch_backward(const TaskSet &ts, const double *d_pab, const GridPtrs &g, double *d_hab,
                            double *d_dra, double *d_drb, double *d_dza, double *d_dzb, cudaStream_t s) {
    if (ts.ntasks == 0) return cudaSuccess;
    if (!backward_supported(ts)) return cudaErrorNotSupported;
    TaskSet &mts = const_cast<TaskSet &>(ts);
    if (!mts.d_mom_ext) {  // the moments, and the divided pairs' slots where the scratch memory is too small
        const size_t parts = sizeof(double) * (size_t)ts.fp64_slots * ncoef(ts.max_lp + 2), own = parts > ts.scratch_bytes ? parts : 0;
        cudaError_t e = cudaMalloc(&mts.d_mom_ext, std::max<size_t>(sizeof(double) * (size_t)ts.mom_ext_len + own, 8));
        if (e != cudaSuccess) return e;
        mts.d_parts_ext = own ? mts.d_mom_ext + ts.mom_ext_len : static_cast<double *>(ts.d_scratch);
    }
    cudaError_t e = launch_moments_fp64(ts, g, 2, mts.d_mom_ext, s);
    if (e != cudaSuccess) return e;
    // the matrix elements come from the same moments (those to degree lp)
    if (d_hab && (e = launch_backtransform(ts, mts.d_mom_ext, 2, d_hab, s)) != cudaSuccess) return e;
    ts.n_kernels++;
    k_backward_epilogue<<<(unsigned)ts.ntasks, 32 * kBWarps, 0, s>>>(ts.d_geom, ts.plan->d_levels, ts.plan->d_tmat,
                                                           mts.d_mom_ext, ts.tau, d_pab, d_dra, d_drb, d_dza,
                                                           d_dzb);
    return cudaGetLastError();
}

}  // namespace gpw
