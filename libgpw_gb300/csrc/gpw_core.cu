// Dense cube contractions of the factorised prototype (collocate.cc:438-623),
// FP64 on the device.  Used as known-answer kernels with the shapes of the
// reference's own tests (collocate_test.cc:35-140, called from collocate.cc:1185-1212).
//
// At those sizes (0.3 MFLOP each way) the time is latency: launch, dependent FP64
// chains, the last partial wave.  Both kernels therefore spread one call over as many
// CTAs as its planes give and keep the chains short.
#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include "gpw_internal.h"

namespace gpw {

// out[z][y][x] = sum_{a,g,b} co[a][g][b] P0[g][z] P1[b][y] P2[a][x]; one CTA per z and
// kCoreRows rows y, a warp per row (13 x 45 x 29 points, L = 7: one CTA per z, 8.0 us;
// 78 CTAs of 8 rows, 4.5 us)
constexpr int kCoreRows = 8;
__global__ void __launch_bounds__(32 * kCoreRows)
k_collocate_core(int nz, int ny, int nx, int L, const double *__restrict__ co, const double *__restrict__ pol, int ld,
                 double *__restrict__ out) {
    __shared__ double C1[16 * 16];         // [a][b]
    __shared__ double C2[kCoreRows][16];   // [y][a]
    const int z = blockIdx.x, y0 = blockIdx.y * kCoreRows;
    const double *P0 = pol, *P1 = pol + (size_t)L * ld, *P2 = pol + (size_t)2 * L * ld;
    for (int t = threadIdx.x; t < L * L; t += blockDim.x) {
        const int a = t / L, b = t - a * L;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
        for (int g = 0; g < L; g++) {
            const double v = co[(a * L + g) * L + b] * P0[g * ld + z];
            if (g & 1) s1 += v;
            else s0 += v;
        }
        C1[t] = s0 + s1;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < kCoreRows * L; t += blockDim.x) {
        const int r = t / L, a = t - r * L;
        if (y0 + r >= ny) break;
        double s = 0.0;
#pragma unroll 4
        for (int b = 0; b < L; b++) s += C1[a * L + b] * P1[b * ld + y0 + r];
        C2[r][a] = s;
    }
    __syncthreads();
    const int r = threadIdx.x >> 5, y = y0 + r;
    if (y >= ny) return;
    for (int x = threadIdx.x & 31; x < nx; x += 32) {
        double s = 0.0;
#pragma unroll 4
        for (int a = 0; a < L; a++) s += C2[r][a] * P2[a * ld + x];
        out[((size_t)z * ny + y) * nx + x] = s;
    }
}

// co[g][b][a] = sum_{z,y,x} V[z][y][x] P0[g][z] P1[b][y] P2[a][x], contracted axis by
// axis: a cluster of kCoreCluster CTAs per a, each CTA every kCoreCluster-th plane z:
//   R[y] = sum_x V[z][y][x] P2[a][x] (a thread per row), Q[b] = sum_y R[y] P1[b][y],
//   W[g][b] += P0[g][z] Q[b], then the CTAs' W are summed through distributed shared
// memory in rank order (deterministic).  (One CTA per output, each reading all of V with
// an index division per value: 45.4 us at 13 x 45 x 29, L = 7; this form 9.4 us, and 8.0 us
// with the latencies shortened: 16 loads of a row in flight, up to 16 lanes per Q entry, the
// ranks' W read before they are added.)
constexpr int kCoreCluster = 8, kCoreThreads = 256;
constexpr int kCoreChunk = 1024;  // rows of one plane handled together
__host__ __device__ constexpr int core_planes(int ny, int L) {  // planes handled together
    const int a = kCoreThreads / (ny > 1 ? ny : 1), b = kCoreThreads / L, n = a < b ? a : b;
    return n > 1 ? n : 1;
}
__global__ void __launch_bounds__(kCoreThreads) __cluster_dims__(kCoreCluster, 1, 1)
k_integrate_core(int nz, int ny, int nx, int L, const double *__restrict__ pol, int ld, const double *__restrict__ V,
                 double *__restrict__ co) {
    namespace cg = cooperative_groups;
    __shared__ double R[kCoreChunk];      // [plane][y] of the rows in hand
    __shared__ double W[16 * 16];         // [g][b]
    __shared__ double Q[kCoreThreads];    // [plane][b], or partial sums
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), a = blockIdx.x / kCoreCluster, tid = threadIdx.x;
    const double *P0 = pol, *P1 = pol + (size_t)L * ld, *P2 = pol + (size_t)(2 * L + a) * ld;
    for (int t = tid; t < L * L; t += kCoreThreads) W[t] = 0.0;
    // np planes at a time (np > 1 only where all their rows fit the threads)
    const int np = core_planes(ny, L);
    int lq = 0;  // 2^lq lanes share a Q entry
    while (lq < 4 && (np * L) << (lq + 1) <= kCoreThreads) lq++;
    for (int z0 = rank; z0 < nz; z0 += np * kCoreCluster) {
        double q[2] = {0.0, 0.0};
        const int qe = tid >> lq, qpl = qe / L, qb = qe - qpl * L, qs = tid & ((1 << lq) - 1);  // this thread's Q entry
        for (int y0 = 0; y0 < ny; y0 += kCoreChunk) {
            const int ry = min(kCoreChunk, ny - y0);
            __syncthreads();
            for (int t = tid; t < np * ry; t += kCoreThreads) {
                const int pl = t / ry, y = t - pl * ry, z = z0 + pl * kCoreCluster;
                double s0 = 0.0, s1 = 0.0;
                if (z < nz) {
                    const double *v = V + ((size_t)z * ny + y0 + y) * nx;
                    for (int x0 = 0; x0 < nx; x0 += 16) {  // 16 loads in flight
                        double w[16];
#pragma unroll
                        for (int i = 0; i < 16; i++) w[i] = x0 + i < nx ? v[x0 + i] : 0.0;
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            if (x0 + i < nx) s0 += w[i] * P2[x0 + i];
                            if (x0 + i + 1 < nx) s1 += w[i + 1] * P2[x0 + i + 1];
                        }
                    }
                }
                R[t] = s0 + s1;
            }
            __syncthreads();
            if (qe < np * L)
                for (int y = qs; y < ry; y += 2 << lq)
#pragma unroll
                    for (int u = 0; u < 2; u++)
                        if (y + (u << lq) < ry) q[u] += R[qpl * ry + y + (u << lq)] * P1[qb * ld + y0 + y + (u << lq)];
        }
        double qt = q[0] + q[1];
        for (int o = 1; o < (1 << lq); o <<= 1) qt += __shfl_xor_sync(0xffffffffu, qt, o);
        if (qs == 0 && qe < np * L) Q[qe] = qt;
        __syncthreads();
        for (int t = tid; t < L * L; t += kCoreThreads) {
            const int g = t / L, b = t - g * L;
            double s = W[t];
            for (int pl = 0; pl < np && z0 + pl * kCoreCluster < nz; pl++)
                s += P0[g * ld + z0 + pl * kCoreCluster] * Q[pl * L + b];
            W[t] = s;
        }
    }
    cl.sync();
    for (int t = rank * kCoreThreads + tid; t < L * L; t += kCoreCluster * kCoreThreads) {
        double w[kCoreCluster], s = 0.0;
#pragma unroll
        for (int r = 0; r < kCoreCluster; r++) w[r] = *cl.map_shared_rank(W + t, r);
#pragma unroll
        for (int r = 0; r < kCoreCluster; r++) s += w[r];
        co[(size_t)t * L + a] = s;
    }
    cl.sync();  // no CTA leaves while another may read its W
}

cudaError_t launch_collocate_core(const int length[3], int L, const double *co, const double *pol, int ld,
                                  double *out, cudaStream_t s) {
    // The sizes accepted are those of the form that kept a plane's rows in shared memory.
    const int64_t rows = 8 * ((int64_t)L * L + (int64_t)length[1] * L);
    if (rows < 0 || rows > 227 * 1024) return cudaErrorInvalidValue;
    if (length[0] > 0 && length[1] <= 0) return cudaSuccess;  // no points
    const dim3 grid((unsigned)length[0], (unsigned)((length[1] + kCoreRows - 1) / kCoreRows));
    k_collocate_core<<<grid, 32 * kCoreRows, 0, s>>>(length[0], length[1], length[2], L, co, pol, ld, out);
    return cudaGetLastError();
}

cudaError_t launch_integrate_core(const int length[3], int L, const double *pol, int ld, const double *V,
                                  double *co, cudaStream_t s) {
    k_integrate_core<<<(unsigned)(kCoreCluster * L), kCoreThreads, 0, s>>>(length[0], length[1], length[2], L, pol,
                                                                            ld, V, co);
    return cudaGetLastError();
}

}  // namespace gpw
