// tdse_ground.cu -- the ground state of a grid spread over a thread-block cluster.
//
// build_grids_kernel iterates one grid per CTA with its vectors in L2: 8.1 ms for 8001 sites, where a
// pass waits for L2 at every site and one SM does the arithmetic.  Few grids (a single call builds
// one) take a cluster each instead: vectors and tables in shared memory, the scans of tdse_cluster.cuh in
// real arithmetic, four cluster barriers an iteration.  The energy quotient does not depend on the
// scale, so it is taken from the unnormalised solution and the norm enters the next right-hand side.
// Same iteration and stopping rule as ground_state() (tridiag.c:86-159).  8001 sites (41 iterations):
// 8.1 -> 0.42 ms; 601 sites 1.1 -> 0.30 ms.
#include <cuda_runtime.h>

#include "tdse_cluster.cuh"
#include "tdse_host.cuh"

namespace mma {
namespace clk {

__host__ __device__ inline size_t gs_bytes(int nc, int m)
{
    const size_t nw = (size_t)nc * kW;
    return 8 * (6 * (size_t)m * kT + 2 * nw + 2 * kW * nw + 3 * nw);
}

__global__ void __launch_bounds__(kT, 1) ground_state_cluster_kernel(const mma_tdse_grid* grids, int m_cap)
{
    typedef Real64 N;
    cg::cluster_group cluster = cg::this_cluster();
    const int NC = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), NW = NC * kW;
    const int t = threadIdx.x, lane = t & 31, g = rank * kW + (t >> 5);
    extern __shared__ __align__(16) unsigned char smem[];
    const int ML = m_cap * kT;
    double* const u = reinterpret_cast<double*>(smem);
    double *const yv = u + ML, *const ib = yv + ML, *const hh = ib + ML, *const gg = hh + ML, *const vq = gg + ML;
    double *const totF = vq + ML, *const totB = totF + NW, *const wtF = totB + NW, *const wtB = wtF + kW * NW,
                 *const red = wtB + kW * NW;
    Scan<N> scan(cluster, totF, totB, wtF, wtB);
    __shared__ double edge[2];

    const mma_tdse_grid G = grids[blockIdx.x / NC];
    const int n = (int)G.n, m256 = (int)G.m, m = (n + NC * kT - 1) / (NC * kT);
    const int64_t L = G.m * kThreads;
    const int c0 = rank * kT + t, s0 = c0 * m;
    const double* tab = G.gs_tab;
    auto pot = [&](int j) { return j >= 0 && j < n ? G.gv[j] : 0.0; };  // V, left there by the table build
    double cF = 1.0, cB = 1.0;
    for (int i = 0; i < m; i++) {
        const int j = s0 + i, q = i * kT + t;
        const int64_t e = (int64_t)(j % m256) * kThreads + j / m256;
        const bool in = j < n;
        ib[q] = in ? tab[GS_IB12 * L + e] : 0.0;
        hh[q] = in ? tab[GS_H * L + e] : 0.0;
        gg[q] = in ? tab[GS_G * L + e] : 0.0;
        vq[q] = pot(j);
        u[q] = in ? 1.0 : 0.0;  // tools.c:39-42
        cF *= -hh[q];
        cB *= -gg[q];
    }
    const double vl = pot(s0 - 1), vr = pot(s0 + m);
    if (t == 0) {
        if (rank == 0) edge[0] = 0.0;
        if (rank == NC - 1) edge[1] = 0.0;
    }
    cluster.sync();  // every CTA has started: its shared memory may be written
    auto send_edges = [&] {
        if (t == 0 && rank > 0) *cluster.map_shared_rank(&edge[1], rank - 1) = u[0];
        if (t == kT - 1 && rank + 1 < NC) *cluster.map_shared_rank(&edge[0], rank + 1) = u[(m - 1) * kT + t];
    };
    send_edges();
    scan.setup(cluster, cF, cB);
    const double inv_dx2 = 1.0 / (G.dx * G.dx), k12 = 1.0 / 12.0, k10 = 10.0 / 12.0;
    double e_old = G.Eguess, energy = G.Eguess, test = 0.0, s2 = 1.0, inv = 1.0;
    int64_t it = 0;
    int status = MMA_OK;
    for (;;) {
        // ---- solve (K - Eg M2) u' = M2 u / |u|
        double pm = t == 0 ? edge[0] : u[(m - 1) * kT + t - 1];
        const double nx = t == kT - 1 ? edge[1] : u[t + 1];
        double pc = u[t], b = 0.0;
        for (int i = 0; i < m; i++) {
            const int q = i * kT + t;
            const double pn = i + 1 < m ? u[q + kT] : nx;
            const double r = ib[q] * (inv * fma(10.0, pc, pm + pn));
            yv[q] = r;
            b = fma(-hh[q], b, r);
            pm = pc;
            pc = pn;
        }
        b = scan.forward_out(cluster, b);
        cluster.sync();
        double y = scan.forward_in(shfl_up(b, 1));
        for (int i = 0; i < m; i++) {
            const int q = i * kT + t;
            y = fma(-hh[q], y, yv[q]);
            yv[q] = y;
        }
        b = y;
        for (int i = m - 2; i >= 0; i--) b = fma(-gg[i * kT + t], b, yv[i * kT + t]);
        b = scan.backward_out(cluster, b);
        cluster.sync();
        double v = scan.backward_in(shfl_down(b, 1));
        for (int i = m - 1; i >= 0; i--) {
            const int q = i * kT + t;
            v = fma(-gg[q], v, yv[q]);
            u[q] = v;
        }
        send_edges();
        cluster.sync();
        // ---- norm (tools.c:137-145) and energy quotient (tridiag.c:172-238)
        double acc[3] = {0.0, 0.0, 0.0};
        pm = t == 0 ? edge[0] : u[(m - 1) * kT + t - 1];
        const double nu = t == kT - 1 ? edge[1] : u[t + 1];
        pc = u[t];
        double vm = vl, vc = vq[t];
#pragma unroll 1  // unrolled, the compiled loop summed two of three sites at m = 3 (tested at m = 1 .. 7)
        for (int i = 0; i < m; i++) {
            const int q = i * kT + t;
            const double pn = i + 1 < m ? u[q + kT] : nu, vn = i + 1 < m ? vq[q + kT] : vr;
            const double sum = pm + pn;
            const double kpsi = fma(inv_dx2, fma(-0.5, sum, pc), fma(k10 * vc, pc, k12 * fma(pm, vm, pn * vn)));
            const double mpsi = fma(k10, pc, k12 * sum);
            if (s0 + i < n) {
                acc[0] = fma(pc, pc, acc[0]);
                acc[1] = fma(kpsi, mpsi, acc[1]);
                acc[2] = fma(mpsi, mpsi, acc[2]);
            }
            pm = pc;
            pc = pn;
            vm = vc;
            vc = vn;
        }
#pragma unroll
        for (int k = 0; k < 3; k++) {
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) acc[k] += shfl_xor(acc[k], d);
            if (lane < NC) cluster.map_shared_rank(red, lane)[k * NW + g] = acc[k];
        }
        cluster.sync();
#pragma unroll
        for (int k = 0; k < 3; k++) {  // the same order in every warp: the decision below is uniform
            double s = 0.0;
            for (int q = lane; q < NW; q += 32) s += red[k * NW + q];
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) s += shfl_xor(s, d);
            acc[k] = s;
        }
        s2 = acc[0];
        inv = 1.0 / sqrt(s2);
        energy = acc[1] / acc[2];
        test = fabs(energy - e_old);
        e_old = energy;
        ++it;
        if (it >= G.max_iter) {
            status = MMA_ERR_GS_NOCONV;
            break;
        }
        if (!(test > G.CV)) break;
    }
    const double nrm = sqrt(s2);
    for (int i = 0; i < m; i++) {
        const int j = s0 + i;
        if (j < n) st2(G.psi0 + 2 * j, cd{u[i * kT + t] / nrm, 0.0});
    }
    if (rank == 0 && t == 0) {
        G.result[0] = energy;
        G.result[1] = (double)it;
        G.result[2] = (double)status;
        G.result[3] = test;
    }
    cluster.sync();  // no CTA leaves while another may still write to it
}

}  // namespace clk

bool ground_state_cluster(const mma_tdse_grid* grids_dev, int n_grids, int64_t max_n, int sms, cudaStream_t st)
{
    // clusters of at least four CTAs that are all resident at once; more grids fill the SMs by themselves
    int nc = sms / n_grids < clk::kMaxNC ? sms / n_grids : clk::kMaxNC;
    while (nc > 4 && (max_n + (nc - 1) * clk::kT - 1) / ((nc - 1) * clk::kT) == (max_n + nc * clk::kT - 1) / (nc * clk::kT))
        nc--;  // fewer CTAs with the same sites per thread
    auto kern = clk::ground_state_cluster_kernel;
    for (; nc >= 4; nc -= nc > 8 ? nc - 8 : 1) {
        const int m = (int)((max_n + nc * clk::kT - 1) / (nc * clk::kT));
        const size_t smem = clk::gs_bytes(nc, m);
        if (smem > 220 * 1024) return false;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            return false;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(n_grids * nc));
        cfg.blockDim = dim3(clk::kT);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)nc;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int active = 0;
        if (cudaOccupancyMaxActiveClusters(&active, kern, &cfg) != cudaSuccess || active < n_grids) {
            cudaGetLastError();
            continue;
        }
        return cudaLaunchKernelEx(&cfg, kern, grids_dev, m) == cudaSuccess;
    }
    return false;
}

}  // namespace mma
